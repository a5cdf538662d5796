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
