"""Set-up of a solve on matrices with rows of 1 to 70 blocks (the mesh's have at most
27): elimination, sliced copies, symmetry check, inverse diagonal blocks.

The elimination is bit-exact with the oracle's.  A product sums at most 210 terms per
scalar row: within 210 eps sum |a||x| <= 1e-12 of the result's norm for these values.
"""
import numpy as np
import pytest
import torch

import oracle as O
from plantfem_gb300 import FEMSolver, problems
from plantfem_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _block_matrix(nb, widest, seed):
    """A symmetric positive definite scalar CRS of 3x3 blocks with uneven rows
    (columns unsorted, as a first-appearance pattern's)."""
    rng = np.random.default_rng(seed)
    nbr = [set() for _ in range(nb)]
    for i in range(nb):
        for j in rng.choice(nb, size=int(rng.integers(0, max(1, widest // 2))), replace=False):
            if len(nbr[i]) < widest - 1 and len(nbr[j]) < widest - 1 and i != j:
                nbr[i].add(int(j))
                nbr[int(j)].add(i)
    B = {}
    for i in range(nb):
        for j in nbr[i]:
            if i < j:
                B[i, j] = rng.normal(size=(3, 3))
                B[j, i] = B[i, j].T.copy()
    for i in range(nb):
        s = sum((np.abs(B[i, j]).sum(axis=1) for j in nbr[i]), np.zeros(3))
        B[i, i] = np.diag(1.0 + 1.5 * s)
    rp, ci, v = [1], [], []
    for i in range(nb):
        cols = list(rng.permutation(sorted(nbr[i] | {i})))
        for r in range(3):
            for j in cols:
                ci += [3 * int(j) + 1, 3 * int(j) + 2, 3 * int(j) + 3]
                v += list(B[i, int(j)][r])
            rp.append(1 + len(ci))
    return np.array(rp, np.int64), np.array(ci, np.int32), np.array(v)


@pytest.mark.parametrize("nb,widest", [(1, 1), (31, 4), (33, 33), (90, 70)])
def test_copies_elimination_and_check(cuda, nb, widest):
    rp, ci, v = _block_matrix(nb, widest, nb)
    n = 3 * nb
    rng = np.random.default_rng(7)
    b = rng.normal(size=n)
    fixed = np.zeros(n, np.uint8)
    ids = rng.choice(n, size=max(1, n // 7), replace=False)
    vals = rng.normal(size=ids.shape[0])
    fixed[ids] = 1
    fv = np.zeros(n)
    fv[ids] = vals
    vo, bo = v.copy(), b.copy()
    O.apply_fix(rp, ci, vo, bo, fixed, fv)
    s = FEMSolver()
    s.setCRS(CRS=(rp, ci, v))
    s.setRHS(b)
    s.fix(1, (ids + 1).astype(np.int32), FixValues=vals)
    s.eliminate()
    assert np.array_equal(s.getCRS()[2], vo) and np.array_equal(s.CRS_RHS, bo)
    x = rng.normal(size=n)
    y = torch.empty(n, dtype=torch.float64, device=cuda)
    s.matvec_device(torch.as_tensor(x, device=cuda), y)
    want = O.spmv(rp, ci, vo, x)
    assert np.linalg.norm(y.cpu().numpy() - want) <= 1e-12 * np.linalg.norm(want)
    s.relative_er = 1e-12
    for um in (0, "separate"):
        for alg in ("CG", "BiCGSTAB"):
            if nb == 1 and alg == "BiCGSTAB":
                # the preconditioner is the inverse: e is rounding noise after half a step,
                # and whether <v, v> is exactly zero (a breakdown) follows the last bit
                continue
            xs = s.solve(algorithm=alg, preconditioning="BlockJacobi", precision="mixed", storage="symmetric",
                         stop_rule="true_relative", update_mode=um)
            # diagonally dominant: condition number below 10
            assert s.last_info["status"] == 0
            assert np.linalg.norm(bo - O.spmv(rp, ci, vo, xs)) <= 1e-11 * np.linalg.norm(bo)


@pytest.mark.parametrize("nb,widest", [(33, 33), (90, 70)])
@pytest.mark.parametrize("factor,ok", [(1.0 + 1e-12, True), (1.0 + 1e-6, False)])
def test_symmetry_check_far_slots(cuda, nb, widest, factor, ok):
    """One entry off by a factor, in the row's last block: rounding noise passes, a
    difference does not."""
    rp, ci, v = _block_matrix(nb, widest, nb + 1)
    rows = np.repeat(np.arange(rp.shape[0] - 1), np.diff(rp))
    off = (rows // 3) != (ci - 1) // 3
    k = int(np.nonzero(off)[0][-1])
    bad = v.copy()
    bad[k] *= factor
    s = FEMSolver()
    s.setCRS(CRS=(rp, ci, bad))
    s.setRHS(np.ones(rp.shape[0] - 1))
    kw = dict(algorithm="CG", precision="mixed", storage="symmetric", stop_rule="true_relative")
    if ok:
        s.solve(**kw)
        assert s.last_info["status"] == 0
    else:
        with pytest.raises(N.NativeError) as e:
            s.solve(**kw)
        assert e.value.code == -1


def test_further_loads_and_new_values(cuda):
    """A second load on an eliminated matrix, new fixed values and a new stiffness
    give what a fresh solver gives (same operations: same bits)."""
    p = problems.lognormal(6, seed=5)
    kw = dict(algorithm="CG", preconditioning="BlockJacobi", stop_rule="true_relative")

    def fresh(E, rhs, value):
        t = FEMSolver()
        t.setDomain(p["domain"])
        t.setCRS(3)
        t.assembleStiffness(E, p["nu"])
        t.setRHS(rhs)
        t.fix(1, p["fix_ids"], FixValue=value)
        return t.solve(**kw)

    s = FEMSolver()
    s.setDomain(p["domain"])
    s.setCRS(3)
    s.assembleStiffness(p["E"], p["nu"])
    s.setRHS(p["rhs"])
    s.fix(1, p["fix_ids"], FixValue=0.0)
    assert np.array_equal(s.solve(**kw), fresh(p["E"], p["rhs"], 0.0))
    s.setRHS(2.5 * p["rhs"])
    assert np.array_equal(s.solve(**kw), fresh(p["E"], 2.5 * p["rhs"], 0.0))
    E2 = p["E"] * np.linspace(0.5, 2.0, p["E"].shape[0])
    s.zeros()
    s.assembleStiffness(E2, p["nu"])
    s.setRHS(p["rhs"])
    s.fix(1, p["fix_ids"], FixValue=1e-3)
    assert np.array_equal(s.solve(**kw), fresh(E2, p["rhs"], 1e-3))
