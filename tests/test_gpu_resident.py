"""The resident solves (one cooperative launch) against the kernel-by-kernel ones.

``update_mode`` left open lets a system that fits the SMs run resident;
``update_mode="separate"`` names the kernel-by-kernel form of the same iteration.
Both stop at the same tolerance, so with kappa the condition number of the
eliminated matrix (below 1e4 on these meshes, E within a factor of ten) two
solutions at a relative residual of 1e-12 differ by less than 2 kappa 1e-12 = 2e-8
of the solution's norm; 1e-8 was met by every form against the oracle before.

Sizes: fewer slices than SMs and a single one; CTAs with fewer slots than warps
(one-element-thick slabs); one slice per CTA and a ragged second; more rows than
one slice per warp.
"""
import numpy as np
import pytest

import oracle as O
from plantfem_gb300 import FEMSolver, problems
from plantfem_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


def _solver(p):
    s = FEMSolver()
    s.setDomain(p["domain"])
    s.setCRS(3)
    s.assembleStiffness(p["E"], p["nu"])
    s.setRHS(p["rhs"])
    s.fix(1, p["fix_ids"], FixValue=0.0)
    s.relative_er = 1e-12
    return s


MESHES = {"cube1": lambda: problems.cube(1), "cube3": lambda: problems.lognormal(3, seed=2),
          "slab12x3x1": lambda: problems.slab(12, 3, 1, 1e4), "cube17": lambda: problems.lognormal(17, seed=4),
          "cube26": lambda: problems.lognormal(26, seed=6)}


@pytest.mark.parametrize("mesh", list(MESHES))
@pytest.mark.parametrize("alg", ["CG", "BiCGSTAB"])
@pytest.mark.parametrize("prec,storage", [("fp64", "full"), ("mixed", "full"), ("mixed", "symmetric")])
@pytest.mark.parametrize("pc", [None, "BlockJacobi"])
def test_resident_equals_kernel_by_kernel(cuda, mesh, alg, prec, storage, pc):
    s = _solver(MESHES[mesh]())
    kw = dict(algorithm=alg, preconditioning=pc, precision=prec, storage=storage, stop_rule="true_relative")
    x = s.solve(**kw)
    info = dict(s.last_info)
    again = s.solve(**kw)
    xs = s.solve(update_mode="separate", **kw)
    sep = dict(s.last_info)
    assert info["status"] == 0 and info["rel_residual"] <= 1e-12, info
    assert sep["status"] == 0, sep
    assert info["kernel_launches"] < 10 < sep["kernel_launches"], (info, sep)
    assert np.array_equal(x, again)  # every sum has a fixed order
    assert _rel(x, xs) <= 1e-8, _rel(x, xs)
    assert info["iterations"] <= 1.25 * sep["iterations"] + 20, (info, sep)


def test_resident_reference_rule_and_limits(cuda):
    """The reference stop rule, itrmax and a warm start follow the other form."""
    s = _solver(problems.cube(8))
    x = s.solve()  # FP64 BiCGSTAB, reference rule
    it = s.last_info["iterations"]
    xs = s.solve(update_mode="separate")
    assert abs(it - s.last_info["iterations"]) <= 5 and _rel(x, xs) <= 1e-8
    s.itrmax = 7
    for um in (0, "separate"):
        for prec in ("fp64", "mixed"):
            s.solve(algorithm="CG", precision=prec, stop_rule="true_relative", update_mode=um)
            assert s.last_info["status"] == N.PFG_W_NOT_CONVERGED and s.last_info["iterations"] == 7, s.last_info
    s.itrmax = 100000
    for prec in ("fp64", "mixed"):
        s.solve(algorithm="CG", precision=prec, stop_rule="true_relative", x0=x)
        assert s.last_info["iterations"] <= 40 and s.last_info["status"] == 0, s.last_info


def test_resident_goes_on_after_a_full_launch(cuda):
    """A solve of more iterations than one launch makes (4096): CG on the 1-D
    Poisson matrix of 6,000 unknowns takes about one iteration per unknown; its
    true residual is recomputed on the host."""
    n = 6000
    rows = [[j for j in (i - 1, i, i + 1) if 0 <= j < n] for i in range(n)]
    rp = np.concatenate([[1], 1 + np.cumsum([len(r) for r in rows])]).astype(np.int64)
    ci = np.concatenate(rows).astype(np.int32) + 1
    v = np.concatenate([[2.0 if j == i else -1.0 for j in r] for i, r in enumerate(rows)])
    s = FEMSolver()
    s.setCRS(CRS=(rp, ci, v))
    b = np.random.default_rng(8).normal(size=n)
    s.setRHS(b)
    s.relative_er = 1e-8
    x = s.solve(algorithm="CG", stop_rule="true_relative")
    assert s.last_info["iterations"] > 4096 and s.last_info["status"] == 0, s.last_info
    assert 2 <= s.last_info["kernel_launches"] < 10
    assert np.linalg.norm(b - O.spmv(rp, ci, v, x)) <= 1.01e-8 * np.linalg.norm(b)


def test_resident_scalar_rows_with_empty_slices(cuda):
    """1x1 blocks: rows of 0 to 40 entries, whole slices without any off-diagonal, and
    an unsymmetric matrix for BiCGSTAB; solved to 1e-12, checked with a dense solve
    (condition number below 10 by diagonal dominance: 2e-11)."""
    n = 1000
    rng = np.random.default_rng(3)
    A = np.zeros((n, n))
    for i in range(n):
        k = 0 if 320 <= i < 448 else int(rng.integers(0, 40))
        cols = rng.choice(n, size=k, replace=False)
        A[i, cols] = rng.normal(size=k)
    np.fill_diagonal(A, 0.0)
    np.fill_diagonal(A, 1.0 + 1.5 * np.abs(A).sum(axis=1))
    b = rng.normal(size=n)
    for M, alg in ((0.5 * (A + A.T) + np.diag(np.abs(A).sum(axis=0)), "CG"), (A, "BiCGSTAB")):
        rp = np.concatenate([[1], 1 + np.cumsum((M != 0).sum(axis=1))]).astype(np.int64)
        ci = (np.concatenate([np.nonzero(M[i])[0] for i in range(n)]) + 1).astype(np.int32)
        v = np.concatenate([M[i][M[i] != 0] for i in range(n)])
        s = FEMSolver()
        s.setCRS(CRS=(rp, ci, v))
        s.setRHS(b)
        s.relative_er = 1e-12
        for prec in ("fp64", "mixed"):
            x = s.solve(algorithm=alg, precision=prec, stop_rule="true_relative", preconditioning="Jacobi")
            assert s.last_info["status"] == 0 and s.last_info["kernel_launches"] < 10, s.last_info
            assert _rel(x, np.linalg.solve(M, b)) <= 2e-11


def test_resident_refuses_and_breaks_down_as_before(cuda):
    """Unsymmetric matrix with symmetric storage: PFG_E_ARG; an indefinite one: CG
    breakdown; a right-hand side of zeros: x = 0 in no iteration."""
    s = _solver(problems.cube(2))
    s.eliminate()
    rp, ci, v = s.getCRS()
    bad = v.copy()
    off = np.where(np.repeat(np.arange(1, rp.shape[0]), np.diff(rp)) == ci, 0.0, np.abs(v))
    bad[np.argmax(off)] *= 1.5
    t = FEMSolver()
    t.setCRS(CRS=(rp, ci, bad))
    t.setRHS(s.CRS_RHS)
    with pytest.raises(N.NativeError) as e:
        t.solve(algorithm="CG", precision="mixed", storage="symmetric", stop_rule="true_relative")
    assert e.value.code == -1
    t.setCRS(CRS=(rp, ci, -v))
    for prec in ("fp64", "mixed"):
        with pytest.raises(N.NativeError) as e:
            t.solve(algorithm="CG", precision=prec, stop_rule="true_relative")
        assert e.value.code == -4
    t.setCRS(CRS=(rp, ci, v))
    t.setRHS(np.zeros(rp.shape[0] - 1))
    x = t.solve(algorithm="CG", precision="mixed", stop_rule="true_relative")
    assert not x.any() and t.last_info["iterations"] == 0
