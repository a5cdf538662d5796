"""Batched persistent solves of uneven thin slabs (the batching form).

Every system of a batch is compared with an FP64 direct solve of the oracle's
eliminated system (SuperLU) at <= 1e-8 relative displacement error and with
the plain one-system GPU path.  Thin slabs clamped on one short edge are
ill-conditioned: even the direct solve leaves a relative residual of up to
~3e-11, so the solves here stop at 1e-9 (the displacement is then already
accurate to ~1e-11).  Every launch configuration (single CTAs,
clusters of 2 / 4 / 8 CTAs, all systems as cluster jobs) must give those
answers.  The abort flag and the error returns are exercised on the host side
of the persistent kernel: no case faults or hangs the GPU.
"""
import ctypes as C

import numpy as np
import pytest

import oracle as O
from plantfem_gb300 import FEMDomain, FEMSolver, FEMSolverBatch, problems
from plantfem_gb300 import _native as N

pytestmark = pytest.mark.gpu

_CACHE = {}
TOL = 1e-9  # true relative residual the batched solves stop at


def _slabs(count=16, seed=7, lo=4, hi=20):
    rng = np.random.default_rng(seed)
    out = []
    for _ in range(count):
        nx, ny = rng.integers(lo, hi + 1, size=2)
        nz = rng.integers(1, 4)
        E = float(np.exp(rng.normal(np.log(1e4), 0.5)))
        out.append(problems.slab(int(nx), int(ny), int(nz), E))
    return out


def _solver(p):
    s = FEMSolver()
    s.setDomain(p["domain"])
    s.setCRS(3)
    s.assembleStiffness(p["E"], p["nu"])
    s.setRHS(p["rhs"])
    s.fix(1, p["fix_ids"], FixValue=0.0)
    return s


def _oracle(p):
    dom = p["domain"]
    rp, ci = O.zero_matrix(dom.nn(), dom.elemnod, 3)
    val = O.assemble(dom.nodcoord, dom.elemnod, rp, ci, "stiffness", E=p["E"], nu=p["nu"])
    b = p["rhs"].copy()
    fixed = np.zeros(3 * dom.nn(), np.uint8)
    fixed[p["fix_ids"] - 1] = 1
    O.apply_fix(rp, ci, val, b, fixed, np.zeros(3 * dom.nn()))
    import scipy.sparse.linalg as sla
    return sla.spsolve(O.crs_to_scipy(rp, ci, val).tocsc(), b)


def _data():
    if "slabs" not in _CACHE:
        ps = _slabs()
        _CACHE["slabs"] = (ps, [_oracle(p) for p in ps])
    return _CACHE["slabs"]


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cfg", [(256, 1, 0.0), (512, 2, 0.5), (512, 4, 0.25), (1024, 8, 1.0)])
def test_batch_matches_oracle(cuda, precision, cfg):
    ps, refs = _data()
    solvers = [_solver(p) for p in ps]
    b = FEMSolverBatch(solvers)
    b.config = {"threads": cfg[0], "cluster": cfg[1], "team_fraction": cfg[2]}
    xs = b.solve(precision=precision, relative_er=TOL)
    assert b.last_info["launches"] == 1
    assert b.last_info["config"]["cluster"] == cfg[1]
    for k, (x, ref) in enumerate(zip(xs, refs)):
        inf = b.last_infos[k]
        assert inf["status"] == 0, (k, inf)
        assert inf["rel_residual"] <= TOL, (k, inf)
        assert _rel(x, ref) <= 1e-8, (k, _rel(x, ref))
        # fixed DOFs carry their prescribed values exactly
        assert np.all(x[ps[k]["fix_ids"] - 1] == 0.0)
    # a second solve reorders the jobs by the measured iteration counts
    xs2 = b.solve(precision=precision, relative_er=TOL)
    for x, ref in zip(xs2, refs):
        assert _rel(x, ref) <= 1e-8


def test_batch_matches_plain_path_and_get_x(cuda):
    ps, refs = _data()
    solvers = [_solver(p) for p in ps[:6]]
    b = FEMSolverBatch(solvers)
    b.solve(precision="fp64", relative_er=TOL, return_x=False)
    for k, s in enumerate(solvers):
        s.relative_er = TOL
        xp = s.solve(algorithm="CG", preconditioning="BlockJacobi", precision="fp64", stop_rule="true_relative")
        xb = b.get_x(k)
        assert _rel(xb, xp) <= 1e-9
        assert _rel(xb, refs[k]) <= 1e-8


def test_batch_zero_load_and_point_jacobi(cuda):
    ps, refs = _data()
    q = problems.slab(5, 9, 1, 2.0e4)
    q["rhs"] = np.zeros_like(q["rhs"])
    solvers = [_solver(ps[0]), _solver(q), _solver(ps[1])]
    b = FEMSolverBatch(solvers)
    for pc in ("Jacobi", None):
        xs = b.solve(precision="mixed", preconditioning=pc, relative_er=TOL)
        assert np.all(xs[1] == 0.0) and b.last_infos[1]["status"] == 0
        assert _rel(xs[0], refs[0]) <= 1e-8 and _rel(xs[2], refs[1]) <= 1e-8


def test_batch_tune_picks_a_valid_config(cuda):
    ps, refs = _data()
    b = FEMSolverBatch([_solver(p) for p in ps])
    cfg, ms = b.tune(precision="mixed", relative_er=TOL)
    assert cfg["threads"] in (256, 512, 1024) and cfg["cluster"] in (1, 2, 4, 8)
    assert 0.0 <= cfg["team_fraction"] <= 1.0 and ms > 0.0
    c = b.config
    assert c["tuned"] and c["cluster"] == cfg["cluster"] and c["threads"] == cfg["threads"]
    xs = b.solve(precision="mixed", relative_er=TOL)
    for x, ref in zip(xs, refs):
        assert _rel(x, ref) <= 1e-8


def test_batch_abort_flag(cuda):
    ps, refs = _data()
    b = FEMSolverBatch([_solver(p) for p in ps[:4]])
    flag = b.abort_flag()
    flag[0] = 1
    for precision in ("fp64", "mixed"):
        with pytest.raises(N.NativeError) as e:
            b.solve(precision=precision, relative_er=TOL)
        assert e.value.code == -11  # PFG_E_ABORTED
    flag[0] = 0
    xs = b.solve(precision="mixed", relative_er=TOL)
    assert all(i["status"] == 0 for i in b.last_infos)
    for x, ref in zip(xs, refs[:4]):
        assert _rel(x, ref) <= 1e-8


def test_batch_error_returns(cuda):
    lib = N.load()
    b = FEMSolverBatch()
    with pytest.raises(N.NativeError) as e:  # solve before set
        b.solve()
    assert e.value.code == -2
    empty = FEMSolver()  # no CRS matrix
    with pytest.raises(N.NativeError) as e:
        b.set([empty])
    assert e.value.code == -2
    ps, _ = _data()
    b.set([_solver(ps[0])])
    o = N.default_opts(algorithm=N.ALG_BICGSTAB)
    rc = lib.pfg_batch_solve(b._h, C.byref(o), None, None, None)
    assert rc == -9  # PFG_E_UNSUPPORTED: the batch runs CG
    bad = N.BatchConfig(300, 3, 2.0)
    assert lib.pfg_batch_set_config(b._h, C.byref(bad)) == -1
    # a scalar (1x1-block) system is refused
    dom = FEMDomain().create("Cube3D", 2, 2, 2)
    s1 = FEMSolver()
    n = 10
    rp = np.arange(1, n + 2, dtype=np.int64)
    ci = np.arange(1, n + 1, dtype=np.int32)
    s1.setCRS(CRS=(rp, ci, np.full(n, 2.0)))
    with pytest.raises(N.NativeError) as e:
        b.set([s1])
    assert e.value.code == -9
    del dom


# Team sizes: one or two long systems among short ones get teams of four or of both
# halves of a cluster, down to sizes whose slices are fewer than the team's warps (and
# than its CTAs, where the whole batch is solved in clusters); the second solve
# knows the iteration counts.
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cfg", [(256, 2, 0.1), (512, 2, 0.1), (512, 4, 0.1), (512, 8, 0.1), (1024, 8, 1.0)])
def test_batch_long_systems_in_larger_teams(cuda, precision, cfg):
    if "teams" not in _CACHE:
        dims = [(24, 20, 3), (20, 7, 2), (14, 14, 2), (9, 9, 3), (7, 6, 1), (4, 4, 1)] + [(5, 3, 1), (2, 2, 1)] * 4
        ps = [problems.slab(*d, 1.0e4 * (1.0 + 0.1 * k)) for k, d in enumerate(dims)]
        _CACHE["teams"] = (ps, [_oracle(p) for p in ps])
    ps, refs = _CACHE["teams"]
    b = FEMSolverBatch([_solver(p) for p in ps])
    b.config = {"threads": cfg[0], "cluster": cfg[1], "team_fraction": cfg[2]}
    for _ in range(3):
        xs = b.solve(precision=precision, relative_er=TOL)
        assert b.last_info["launches"] == 1
        for k, (x, ref) in enumerate(zip(xs, refs)):
            inf = b.last_infos[k]
            assert inf["status"] == 0 and inf["rel_residual"] <= TOL, (k, inf)
            assert _rel(x, ref) <= 1e-8, (k, _rel(x, ref))  # conditioning times TOL, as above
