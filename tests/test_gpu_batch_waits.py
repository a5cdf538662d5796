"""Batched solves whose CTAs wait for one another too long.

The systems of half a cluster meet at barriers with a limited wait.  One that runs
out must leave no system with a good status and another answer: each ends with its own
solution or with PFG_E_INTERNAL, the systems of whole clusters and of single CTAs are
not touched, and the next solve is as good as the first.  The limit is a setting, so a
wait runs out without anything being late; every wait stays bounded.

Batch: one system for a whole cluster of four, seven for halves (768 to 1,535 unknowns
in FP64, 3,072 to 6,143 in mixed precision), four for single CTAs.
"""
import ctypes as C

import numpy as np
import pytest

from plantfem_gb300 import FEMSolver, FEMSolverBatch, problems
from plantfem_gb300 import _native as N

pytestmark = pytest.mark.gpu

PFG_E_INTERNAL = -8


def _solver(p):
    s = FEMSolver()
    s.setDomain(p["domain"])
    s.setCRS(3)
    s.assembleStiffness(p["E"], p["nu"])
    s.setRHS(p["rhs"])
    s.fix(1, p["fix_ids"], FixValue=0.0)
    return s


def _batch(precision):
    n = 6 if precision == "fp64" else 10
    ps = [problems.lognormal(n + 3, seed=1)] + [problems.lognormal(n, seed=2 + k) for k in range(7)]
    ps += [problems.cube(2)] * 4
    b = FEMSolverBatch([_solver(p) for p in ps])
    b.config = {"threads": 256, "cluster": 4, "team_fraction": 1.0 / 12.0}
    return b


def _limited(b, cycles):
    N.check(N.load().pfg_batch_set_wait_limit(b._h, cycles))


def _solve(b, precision):
    """Status of the call, and of each system."""
    o = b._opts(precision, "BlockJacobi", 1e-9, 100000, None)
    infos = (N.Info * len(b.solvers))()
    rc = N.load().pfg_batch_solve(b._h, C.byref(o), None, infos, None)
    return rc, [i.status for i in infos]


def _same(b, ref):
    """Every system as in ref: a condition number below 1e4 times both tolerances."""
    return all(np.linalg.norm(b.get_x(k) - r) <= 2e-5 * np.linalg.norm(r) for k, r in enumerate(ref))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_waits_that_run_out_end_with_an_error(cuda, precision):
    b = _batch(precision)
    _limited(b, -1)
    rc, first = _solve(b, precision)  # no record of an earlier solve
    assert rc == PFG_E_INTERNAL
    assert first[0] == 0 and first[8:] == [0] * 4 and PFG_E_INTERNAL in first, first
    assert set(first[1:8]) <= {0, PFG_E_INTERNAL}, first
    _limited(b, 1 << 32)
    for _ in range(2):
        assert _solve(b, precision) == (0, [0] * 12)
    ref = [b.get_x(k) for k in range(12)]
    _limited(b, -1)  # good records from the solve before
    rc, again = _solve(b, precision)
    assert rc == PFG_E_INTERNAL and set(again) == {0, PFG_E_INTERNAL}, again
    _limited(b, 1 << 32)
    assert _solve(b, precision) == (0, [0] * 12) and _same(b, ref)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("cycles", [0, 30, 100, 300, 1000, 3000])
def test_short_limits_give_an_answer_or_an_error(cuda, precision, cycles):
    b = _batch(precision)
    assert _solve(b, precision)[0] == 0
    ref = [b.get_x(k) for k in range(12)]
    _limited(b, cycles)
    for _ in range(3):
        rc, st = _solve(b, precision)
        assert rc in (0, PFG_E_INTERNAL) and set(st) <= {0, PFG_E_INTERNAL}
        for k, r in enumerate(ref):
            if st[k] == 0:  # conditioning below 1e4 times both tolerances
                assert np.linalg.norm(b.get_x(k) - r) <= 2e-5 * np.linalg.norm(r), k
