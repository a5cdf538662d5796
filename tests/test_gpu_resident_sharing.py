"""Resident solves that share the device: threads, device memory, launches."""
import threading
import time

import numpy as np
import pytest

from plantfem_gb300 import FEMSolver, FEMSolverBatch, problems
from plantfem_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _solver(p):
    s = FEMSolver()
    s.setDomain(p["domain"])
    s.setCRS(3)
    s.assembleStiffness(p["E"], p["nu"])
    s.setRHS(p["rhs"])
    s.fix(1, p["fix_ids"], FixValue=0.0)
    return s


def _poisson(n=6000):
    """1-D Poisson matrix: CG takes about n iterations."""
    rows = [[j for j in (i - 1, i, i + 1) if 0 <= j < n] for i in range(n)]
    rp = np.concatenate([[1], 1 + np.cumsum([len(r) for r in rows])]).astype(np.int64)
    ci = np.concatenate(rows).astype(np.int32) + 1
    v = np.concatenate([[2.0 if j == i else -1.0 for j in r] for i, r in enumerate(rows)])
    s = FEMSolver()
    s.setCRS(CRS=(rp, ci, v))
    s.setRHS(np.random.default_rng(8).normal(size=n))
    return s


def test_a_short_solve_does_not_wait_for_a_long_one(cuda):
    """While one thread runs 100,000 iterations (25 launches, about a second), another's
    solve of a few milliseconds comes in between two launches; neither's bits change."""
    kw = dict(algorithm="CG", stop_rule="true_relative")
    long = _poisson()
    long.relative_er, long.itrmax = 1e-30, 100000
    ref = long.solve(**kw)
    short = _solver(problems.cube(8))
    alone = short.solve(**kw)
    got = []
    t = threading.Thread(target=lambda: got.append(long.solve(**kw)))
    t.start()
    time.sleep(0.1)
    x = short.solve(**kw)
    between = t.is_alive()
    t.join()
    assert between and np.array_equal(x, alone) and np.array_equal(got[0], ref)


def test_threads_get_their_own_answers(cuda):
    """Four threads, each with its own systems and forms, over and over: the bits of
    the solves made one after another."""
    forms = [dict(algorithm=a, precision=p, stop_rule="true_relative") for a in ("CG", "BiCGSTAB")
             for p in ("fp64", "mixed")]
    meshes = [problems.lognormal(n, seed=n) for n in (3, 6, 9, 12)]
    ref = [[_solver(m).solve(**kw) for m in meshes] for kw in forms]
    wrong = []

    def work(k):
        solvers = [_solver(m) for m in meshes]
        for rep in range(6):
            for i, s in enumerate(solvers):
                kw = forms[(k + rep) % 4]
                s.setRHS(meshes[i]["rhs"])
                if not np.array_equal(s.solve(**kw), ref[(k + rep) % 4][i]):
                    wrong.append((k, rep, i))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not wrong, wrong


@pytest.mark.parametrize("kw", [dict(algorithm="CG", precision="mixed"), dict(algorithm="BiCGSTAB")])
def test_small_handles_stay_small(cuda, kw):
    """What resident solves exchange sums through is the device's, and a resident solve
    holds no vectors of the other form: 64 solved handles of a 64-node mesh take less
    than 1 MB each (kernel by kernel 0.5 to 0.8 MB; with 3.3 MB of slots each, 4.5)."""
    import torch
    p = problems.cube(3)
    keep = []

    def more(n):
        for _ in range(n):
            s = _solver(p)
            s.solve(**kw)
            keep.append(s)
        return torch.cuda.mem_get_info()[0]

    before = more(4)
    assert (before - more(64)) / 64 < 1.0e6


def _resident(s, launch_iterations=0, ctas=0):
    N.check(N.load().pfg_set_resident(s.handle, launch_iterations, ctas))


@pytest.mark.parametrize("algorithm", ["CG", "BiCGSTAB"])
@pytest.mark.parametrize("precision,storage", [("fp64", "full"), ("mixed", "full"), ("mixed", "symmetric")])
def test_a_grid_the_device_does_not_hold(cuda, algorithm, precision, storage):
    """More CTAs than the device has SMs: the launch is refused and the solve runs kernel
    by kernel, to the same bits as when that form is asked for (all but the symmetric
    CG's, whose sums go by atomics).  Fewer CTAs: resident, with its own order of sums
    (tolerance as in the resident tests)."""
    s = _solver(problems.lognormal(17, seed=4))  # 183 slices
    s.relative_er = 1e-12
    kw = dict(algorithm=algorithm, precision=precision, storage=storage, stop_rule="true_relative",
              preconditioning="BlockJacobi")
    sep = s.solve(update_mode="separate", **kw)
    _resident(s, ctas=160)
    x = s.solve(**kw)
    info = dict(s.last_info)
    assert info["status"] == 0 and info["kernel_launches"] > 10, info
    if (algorithm, storage) == ("CG", "symmetric"):
        assert np.linalg.norm(x - sep) <= 1e-8 * np.linalg.norm(sep)
    else:
        assert np.array_equal(x, sep)
    _resident(s, ctas=40)
    y = s.solve(**kw)
    assert s.last_info["status"] == 0 and s.last_info["kernel_launches"] < 10, s.last_info
    assert np.linalg.norm(y - sep) <= 1e-8 * np.linalg.norm(sep)
    _resident(s)
    z = s.solve(**kw)
    t = _solver(problems.lognormal(17, seed=4))
    t.relative_er = 1e-12
    assert np.array_equal(z, t.solve(**kw))


def test_beside_a_batch_and_kernel_by_kernel_solves(cuda):
    """A batch's persistent kernel, resident solves and kernel-by-kernel ones from three
    threads: each waits for its SMs and ends with the bits it has alone (the batch: its
    teams follow the solve before, so the answers to 1e-8 relative residuals)."""
    ps = [problems.lognormal(n, seed=n) for n in (4, 5, 6, 7, 8)]
    batch = FEMSolverBatch([_solver(p) for p in ps])
    batch.config = {"threads": 512, "cluster": 2, "team_fraction": 0.4}
    ref_b = batch.solve(precision="fp64", relative_er=1e-8)
    p = problems.lognormal(14, seed=3)
    kw = dict(algorithm="BiCGSTAB", stop_rule="true_relative", preconditioning="BlockJacobi")
    res, sep = _solver(p), _solver(p)
    ref_r, ref_s = res.solve(**kw), sep.solve(update_mode="separate", **kw)
    wrong = []

    def again(what, f, good):
        for k in range(12):
            if not good(f()):
                wrong.append((what, k))

    ts = [threading.Thread(target=again, args=a) for a in (
        ("batch", lambda: batch.solve(precision="fp64", relative_er=1e-8),
         lambda xs: all(np.linalg.norm(x - r) <= 1e-4 * np.linalg.norm(r) for x, r in zip(xs, ref_b))),
        ("resident", lambda: res.solve(**kw), lambda x: np.array_equal(x, ref_r)),
        ("separate", lambda: sep.solve(update_mode="separate", **kw), lambda x: np.array_equal(x, ref_s)))]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not wrong, wrong
