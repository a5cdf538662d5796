"""Assembly of hexahedra that name a node twice (collapsed to wedges and pyramids).

Several of such an element's 64 blocks fall on one entry of the matrix; each has to be
added.  Against the oracle's serial loop: an entry is a sum of at most some 60 terms of
eight-point quadratures, 1e-12 of the largest entry covers their rounding.
"""
import numpy as np
import pytest

import oracle as O
from plantfem_gb300 import FEMSolver, problems

pytestmark = pytest.mark.gpu

# local nodes 0-3 below, 4-7 above: (kept, replaced by it)
SHAPES = {"wedge, a vertical edge": [(0, 4)], "wedge, two vertical edges": [(1, 5), (2, 6)],
          "wedge, a bottom edge": [(2, 3)], "pyramid": [(4, 5), (4, 6), (4, 7)],
          "two edges": [(0, 4), (2, 3)]}


@pytest.mark.parametrize("shape", list(SHAPES))
@pytest.mark.parametrize("n", [1, 2, 5])
def test_repeated_nodes(cuda, shape, n):
    p = problems.lognormal(n, seed=3)
    d = p["domain"]
    en = d.elemnod.copy()
    some = np.random.default_rng(n).random(en.shape[0]) < 0.6
    some[0] = True
    for kept, gone in SHAPES[shape]:
        en[some, gone] = en[some, kept]
    d.elemnod = en
    rp, ci = O.zero_matrix(d.nn(), en, 3)
    s = FEMSolver()
    s.setDomain(d)
    s.setCRS(3)
    grp, gci, _ = s.getCRS()
    assert np.array_equal(grp, rp) and np.array_equal(gci, ci)

    def same(ref):
        got = s.getCRS()[2]
        s.zeros()
        assert np.abs(got - ref).max() <= 1e-12 * np.abs(ref).max()

    s.assembleStiffness(p["E"], p["nu"])
    same(O.assemble(d.nodcoord, en, rp, ci, "stiffness", E=p["E"], nu=p["nu"]))
    rho = np.linspace(900.0, 1100.0, d.ne())
    mass = O.assemble(d.nodcoord, en, rp, ci, "mass", rho=rho)
    s.assembleMass(rho)
    same(mass)
    s.assembleMass(rho, True)
    row = np.repeat(np.arange(rp.shape[0] - 1), np.diff(rp))
    lumped = np.where(row + 1 == ci, np.bincount(row, weights=mass, minlength=rp.shape[0] - 1)[row], 0.0)
    same(lumped)
