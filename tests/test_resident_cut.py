"""CPU replay of the resident solves' cut (Cut in resident.cu): the CTA's slots fall into
one run per warp, and the segments where runs and slices meet have places of their own."""
import random

import pytest


def _widths(rng, ns):
    return [rng.choice([0, 0, 1, 5, 8, 12, 14, 18, 27, rng.randint(0, 70)]) for _ in range(ns)]


def _sptr(w):
    sp = [0]
    for x in w:
        sp.append(sp[-1] + x)
    return sp


NW = 16


def _cut_start(n, w):
    return n // NW * w + min(w, n % NW)


def _cut_warp(n, t):
    q, rem = n // NW, n % NW
    big = rem * (q + 1)
    return t // (q + 1) if t < big else rem + (t - big) // q


@pytest.mark.parametrize("seed", range(40))
def test_resident_cut_segments(seed):
    rng = random.Random(1000 + seed)
    nsl = rng.randint(1, 40)
    sp = _sptr(_widths(rng, nsl))
    n = sp[-1]
    assert _cut_start(n, 0) == 0 and _cut_start(n, NW) == n
    places = {}
    for w in range(NW):
        t, t1, sl = _cut_start(n, w), _cut_start(n, w + 1), 0
        while t < t1:
            while sp[sl + 1] <= t:
                sl += 1
            e = min(t1, sp[sl + 1])
            assert sl + w not in places
            places[sl + w] = sl
            assert all(_cut_warp(n, q) == w for q in range(t, e))
            t = e
    taken = set(places)
    for sl in range(nsl):
        t0, t1 = sp[sl], sp[sl + 1]
        lo = _cut_warp(n, min(t0, n - 1)) if n else 0
        if t1 > t0:
            hi = _cut_warp(n, t1 - 1)
            assert sorted(k for k, s in places.items() if s == sl) == list(range(sl + lo, sl + hi + 1))
        else:
            assert sl + lo not in taken  # an empty slice's own place
            taken.add(sl + lo)
    assert all(k < nsl + NW for k in taken)
