"""The walk by cells against the oracle where its 32-bit candidate test or its splitting of cells
could lose or repeat a pair: the inputs of the half-stencil tiles, grids of two and of exactly three
cells an axis, more than 32 atoms a cell, and system sizes on each side of the splitting rule.

Lists are compared exactly, twice per context: the first build counts and emits in two walks, the
next ones in one.
"""
import numpy as np
import pytest

import ipg
import oracle
from test_gpu_half_tiles import CASES as TILE_CASES

pytestmark = pytest.mark.gpu


def uniform(n, L, rc, periodic=(True, True, True)):
    def make():
        pos = np.random.default_rng(n).uniform(0, 1, (n, 3)) * np.asarray(L)
        return ipg.System(pos, ["Ar"] * n, list(L), periodic), rc
    return make


CASES = dict(TILE_CASES)
CASES.update({
    "two_cells": uniform(249, (7.5, 7.5, 7.5), 3.2),
    "three_cells": uniform(400, (9.1, 9.1, 9.1), 3.03),
    "two_and_many": uniform(3000, (7.0, 12.5, 40.0), 3.1),
    "dense": uniform(2500, (9.5, 10.0, 13.0), 3.1),
    "open_axis": uniform(900, (9.5, 14.0, 30.0), 3.1, (True, True, False)),
    "n8192": uniform(8192, (41.0, 43.0, 45.0), 4.0),
    "n40000": uniform(40000, (70.0, 72.0, 75.0), 4.0),
})


@pytest.mark.parametrize("case", sorted(CASES))
def test_walk_matches_oracle(case):
    s, rc = CASES[case]()
    off, j, r = oracle.nlist_half(s.positions, s.L, rc)
    for _ in range(2):
        nl = ipg.neighborlist(s, rc)
        assert np.array_equal(nl.offsets, off)
        assert np.array_equal(nl._j, j)
        assert np.array_equal(nl._r, r)
