"""Solves at the edges of what the entry points take: what is refused, which status a
solve ends with, extreme scales and limits, and the settings that leave the answer as
it is.  The kernel-by-kernel form (update_mode "separate") is the measure of the
resident one.
"""
import numpy as np
import pytest

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
    return s


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("update_mode", [0, "separate"])
def test_symmetric_storage_refuses_non_finite_pairs(cuda, bad, update_mode):
    """The same NaN or infinity at (i, j) and (j, i) is no symmetric pair: PFG_E_ARG."""
    s = _solver(problems.cube(2))
    s.eliminate()
    rp, ci, v = s.getCRS()
    row = np.repeat(np.arange(1, rp.shape[0]), np.diff(rp))
    off = np.nonzero((row - 1) // 3 != (ci - 1) // 3)[0]
    k = off[np.argmax(np.abs(v[off]))]
    v[k] = bad
    v[np.nonzero((row == ci[k]) & (ci == row[k]))[0][0]] = bad
    t = FEMSolver()
    t.setCRS(CRS=(rp, ci, v))
    t.setRHS(s.CRS_RHS)
    with pytest.raises(N.NativeError) as e:
        t.solve(algorithm="CG", precision="mixed", storage="symmetric", stop_rule="true_relative",
                update_mode=update_mode)
    assert e.value.code == -1, e.value


@pytest.mark.parametrize("update_mode", ["separate", "fused"])
def test_symmetric_storage_with_unsymmetric_diagonal_blocks(cuda, update_mode):
    """The check is of the off-diagonal blocks, so a diagonal block may be unsymmetric.
    Its inverse, unsymmetric too, is the preconditioner from either copy: both take
    about the same iterations (an FP64 model 20; the mirrored upper triangles of the
    inverses have not converged after 300)."""
    nb = 100
    rng = np.random.default_rng(5)
    G, K = rng.normal(size=(nb, 3, 3)), rng.normal(size=(nb, 3, 3))
    D = 4.0 * np.eye(3) + 0.25 * (G + G.transpose(0, 2, 1)) + 0.25 * (K - K.transpose(0, 2, 1))
    rp, ci, v = [1], [], []
    for i in range(nb):
        for r in range(3):
            for j in range(max(0, i - 1), min(nb, i + 2)):
                for c in range(3):
                    ci.append(3 * j + c + 1)
                    v.append(D[i, r, c] if j == i else (-0.8 if r == c else 0.0))
            rp.append(len(ci) + 1)
    s = FEMSolver()
    s.setCRS(CRS=(np.array(rp, np.int64), np.array(ci, np.int32), np.array(v)))
    s.setRHS(rng.normal(size=3 * nb))
    got = {}
    for storage in ("full", "symmetric"):
        s.solve(algorithm="CG", precision="mixed", storage=storage, stop_rule="true_relative",
                preconditioning="BlockJacobi", update_mode=update_mode)
        got[storage] = (s.last_info["iterations"], s.last_info["fallback"])
    assert got["symmetric"][1] == got["full"][1] == 0, got
    assert abs(got["symmetric"][0] - got["full"][0]) <= 5, got


@pytest.mark.parametrize("algorithm,precision", [("CG", "fp64"), ("CG", "mixed"), ("BiCGSTAB", "mixed")])
def test_unreachable_tolerance_is_reported(cuda, algorithm, precision):
    """Below FP64's reach (1e-18): CG and the mixed solves end with the warning whatever
    the stop rule, which is FP64 BiCGSTAB's alone."""
    s = _solver(problems.cube(4))
    s.relative_er = 1e-18
    s.itrmax = 3000
    for stop_rule in ("reference", "true_relative"):
        for update_mode in (0, "separate"):
            s.solve(algorithm=algorithm, precision=precision, stop_rule=stop_rule, preconditioning="BlockJacobi",
                    update_mode=update_mode)
            assert s.last_info["status"] == N.PFG_W_NOT_CONVERGED, (stop_rule, update_mode, s.last_info)


@pytest.mark.parametrize("er0,relative_er", [(-1.0, 1e-8), (-1e300, 1e-8), (0.0, 1e-8), (1e-200, 1e-8),
                                             (1e-9, -1.0), (1e-9, 1e-200), (1e-9, 0.0), (1e200, 1e-8)])
def test_limits_that_no_square_stands_for(cuda, er0, relative_er):
    """The reference stop rule compares sqrt(rr / rr1) and sqrt(rr) with its limits: a
    negative one never holds (er0 = -1 leaves the relative test alone), a tiny one does
    once the residual is as small."""
    s = _solver(problems.cube(4))
    s.er0, s.relative_er = er0, relative_er
    s.solve()
    res = dict(s.last_info)
    s.solve(update_mode="separate")
    sep = s.last_info
    assert res["status"] == sep["status"] == 0
    assert abs(res["iterations"] - sep["iterations"]) <= 3, (res, sep)


@pytest.mark.parametrize("scale", [1e-140, 1e-152, 1e-154, 1e-155, 1e150])
@pytest.mark.parametrize("algorithm", ["CG", "BiCGSTAB"])
def test_right_hand_sides_of_extreme_scale(cuda, algorithm, scale):
    """FP64 solves of K x = scale b to 1e-4: <r, z> down to 1e-312, whose reciprocal is
    out of range, and up to 1e302.  Scaling by a power of two changes no bit until
    numbers become subnormal; those still hold more digits than the tolerance."""
    p = problems.cube(4)
    p["E"] = np.ones_like(p["E"])
    p["rhs"] = p["rhs"] * scale
    s = _solver(p)
    s.relative_er = 1e-4
    kw = dict(algorithm=algorithm, stop_rule="true_relative", preconditioning="BlockJacobi")
    s.solve(**kw)
    res = dict(s.last_info)
    s.solve(update_mode="separate", **kw)
    sep = s.last_info
    assert res["status"] == sep["status"] == 0 and res["rel_residual"] <= 1e-4, (res, sep)
    assert abs(res["iterations"] - sep["iterations"]) <= 2, (res, sep)


@pytest.mark.parametrize("algorithm", ["CG", "BiCGSTAB"])
@pytest.mark.parametrize("precision,storage", [("fp64", "full"), ("mixed", "full"), ("mixed", "symmetric")])
def test_debug_prints_and_changes_nothing(cuda, capfd, algorithm, precision, storage):
    """debug shows the solve that runs without it: same bits, same count, a line every 32
    iterations (graph_chunk)."""
    s = _solver(problems.lognormal(12, seed=2))
    kw = dict(algorithm=algorithm, precision=precision, storage=storage, stop_rule="true_relative")
    x = s.solve(**kw)
    it = s.last_info["iterations"]
    assert "[pfg]" not in capfd.readouterr().err
    s.debug = True
    y = s.solve(**kw)
    lines = [t for t in capfd.readouterr().err.splitlines() if t.startswith("[pfg]")]
    assert np.array_equal(x, y) and s.last_info["iterations"] == it
    assert len(lines) >= it // 32 >= 2, lines
