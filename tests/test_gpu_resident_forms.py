"""Resident solves beyond one launch and beyond shared memory.

A solve that is continued by further launches has the bits of one that is not: every
vector and scalar comes back from memory as it was.  And above some 40 to 80 thousand
block rows a CTA's own vectors and inverse blocks no longer all lie in shared memory, and
it owns more slices than it has warps: 85,184 rows are 2,662 slices, 17 or 18 to a CTA.
"""
import numpy as np
import pytest

from plantfem_gb300 import FEMSolver, problems
from plantfem_gb300 import _native as N

pytestmark = pytest.mark.gpu

FORMS = [(a, p, pc) for a in ("CG", "BiCGSTAB") for p in ("fp64", "mixed") for pc in (None, "BlockJacobi")]
_CACHE = {}


def _solver(n):
    if n not in _CACHE:
        _CACHE[n] = problems.lognormal(n, seed=n)
    p = _CACHE[n]
    s = FEMSolver()
    s.setDomain(p["domain"])
    s.setCRS(3)
    s.assembleStiffness(p["E"], p["nu"])
    s.setRHS(p["rhs"])
    s.fix(1, p["fix_ids"], FixValue=0.0)
    return s


def _limits(s, launch_iterations):
    N.check(N.load().pfg_set_resident(s.handle, launch_iterations, 0))


@pytest.mark.parametrize("algorithm,precision,pc", FORMS)
@pytest.mark.parametrize("n,step", [(2, 1), (9, 7), (20, 40)])
def test_continued_solves_keep_their_bits(cuda, algorithm, precision, pc, n, step):
    s = _solver(n)
    s.relative_er = 1e-11
    kw = dict(algorithm=algorithm, precision=precision, preconditioning=pc, stop_rule="true_relative")
    x = s.solve(**kw)
    whole = dict(s.last_info)
    _limits(s, step)
    y = s.solve(**kw)
    assert s.last_info["kernel_launches"] > whole["kernel_launches"]
    assert np.array_equal(x, y) and s.last_info["iterations"] == whole["iterations"]
    assert s.last_info["rel_residual"] == whole["rel_residual"]


@pytest.mark.parametrize("algorithm,precision,pc", FORMS)
def test_vectors_outside_shared_memory(cuda, algorithm, precision, pc):
    """Against the kernel-by-kernel form: solutions of relative residual 1e-11 differ by
    less than 2 kappa 1e-11, with kappa of about 6 h^-2 times ten for the spread of E, 1.2e5
    here: 2.4e-6."""
    s = _solver(43)
    s.relative_er = 1e-11
    kw = dict(algorithm=algorithm, precision=precision, preconditioning=pc, stop_rule="true_relative")
    x = s.solve(**kw)
    info = dict(s.last_info)
    assert info["status"] == 0 and info["rel_residual"] <= 1e-11 and info["kernel_launches"] < 10, info
    _limits(s, 100)
    assert np.array_equal(x, s.solve(**kw)) and s.last_info["kernel_launches"] > info["kernel_launches"]
    y = s.solve(update_mode="separate", **kw)
    assert s.last_info["status"] == 0
    assert np.linalg.norm(x - y) <= 2.4e-6 * np.linalg.norm(y)


def _band(rows, half, bs, spread=1):
    """Diagonally dominant band matrix of 2 half + 1 blocks a row as 1-based CRS (fewer at
    the ends), each block off the diagonal -1 on its diagonal."""
    off = spread * np.arange(-half, half + 1)
    j = np.arange(rows)[:, None] + off[None, :]
    keep = (j >= 0) & (j < rows)
    cnt = keep.sum(axis=1)
    cols = j[keep].astype(np.int32)
    row = np.repeat(np.arange(rows, dtype=np.int32), cnt)
    val = np.where(cols == row, 2.0 * half + 1.0, -1.0)
    if bs == 1:
        return np.concatenate([[1], 1 + np.cumsum(cnt)]).astype(np.int64), cols + 1, val
    first = np.concatenate([[0], np.cumsum(cnt)])[:-1]
    pos = np.arange(cols.size) - first[row]
    rp = np.concatenate([[1], 1 + np.cumsum(np.repeat(bs * cnt, bs))]).astype(np.int64)
    ci, v = np.empty(bs * bs * cols.size, np.int32), np.zeros(bs * bs * cols.size)
    for r in range(bs):
        for c in range(bs):
            at = bs * bs * first[row] + r * bs * cnt[row] + bs * pos + c
            ci[at] = bs * cols + c + 1
            if r == c:
                v[at] = val
    return rp, ci, v


# (rows, blocks on each side, block size, form, runs resident): both sides of the rules that
# count entries and bytes.  The 3x3 copy of 30,000 rows with 121 blocks is 145 MB, of 20,000
# rows 97 MB; 70,000 rows with 31 entries are 2.2 million.
@pytest.mark.parametrize("rows,half,bs,kw,resident", [
    (70000, 15, 1, dict(precision="fp64"), False),
    (60000, 20, 1, dict(precision="fp64"), True),
    (70000, 10, 1, dict(precision="fp64"), True),
    (70000, 15, 1, dict(precision="fp64", algorithm="BiCGSTAB"), False),
    (70000, 15, 1, dict(precision="mixed"), True),
    (30000, 60, 3, dict(precision="mixed", storage="symmetric"), False),
    (30000, 60, 3, dict(precision="mixed"), True),
    (20000, 60, 3, dict(precision="mixed", storage="symmetric"), True)])
def test_which_solves_run_resident(cuda, rows, half, bs, kw, resident):
    rp, ci, v = _band(rows, half, bs, spread=3)
    s = FEMSolver()
    s.setCRS(CRS=(rp, ci, v))
    b = np.random.default_rng(1).normal(size=bs * rows)
    s.setRHS(b)
    s.relative_er = 1e-8
    x = s.solve(**{"algorithm": "CG", "stop_rule": "true_relative", "preconditioning": "BlockJacobi", **kw})
    assert s.last_info["status"] == 0
    assert (s.last_info["kernel_launches"] < 10) == resident, s.last_info
    row = np.repeat(np.arange(bs * rows), np.diff(rp))
    r = b - np.bincount(row, weights=v * x[ci - 1], minlength=bs * rows)
    assert np.linalg.norm(r) <= 1.01e-8 * np.linalg.norm(b)
