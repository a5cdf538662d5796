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
