"""Lengths in any unit: the neighbor search proposes its candidates in 32 bits, whose range is far narrower
than that of the 64-bit results.  Boxes, cutoffs and positions from 1e-24 to 1e+24 of the usual ones, pairs close to
the cutoff among them, against the oracle; lists exactly, forces at the repository's parity bound.
"""
import numpy as np
import pytest

import ipg
import oracle
from conftest import TOL, rel_err
from test_gpu_pair import oracle_eval

pytestmark = pytest.mark.gpu

UNITS = [1e-24, 3e-22, 1e-21, 1e-10, 1e10, 1e16, 1e24]


def system(unit, periodic=True, n=900):
    """Random positions, and shells just inside and outside the cutoff 3 (in the unit) of the first atoms."""
    rng = np.random.default_rng(11)
    pos = rng.uniform(0, 12.5, (n, 3))
    d = rng.normal(size=(200, 3))
    d *= (3.0 * (1 + np.linspace(-1e-4, 1e-4, 200)) / np.linalg.norm(d, axis=1))[:, None]
    pos[100:300] = pos[:200] % 12.5 + d
    return ipg.System(pos * unit, ["Ar"] * n, [12.5 * unit] * 3, (periodic,) * 3)


@pytest.mark.parametrize("unit", UNITS)
@pytest.mark.parametrize("periodic", [True, False])
def test_neighbor_list(unit, periodic):
    s = system(unit, periodic)
    off, j, r = oracle.nlist_half(s.positions, s.L, 3.0 * unit)
    nl = ipg.neighborlist(s, 3.0 * unit, ctx=ipg.Context(0))
    assert len(j) > 0 and np.array_equal(nl.offsets, off) and np.array_equal(nl._j, j) and np.array_equal(nl._r, r)


@pytest.mark.parametrize("unit", UNITS)
def test_pair_potential(unit):
    s = system(unit)
    p = ipg.Morse(0.1, 0.5 / unit, 1.5 * unit, 3.0 * unit, ["Ar"])
    e, f, w = ipg.empirical.pair_eval(s, ipg.empirical.empirical_terms(p), ctx=ipg.Context(0))
    eo, fo, wo = oracle_eval(s, p)
    assert eo != 0.0 and abs(e - eo) <= TOL * abs(eo) and rel_err(f, fo) <= TOL and rel_err(w, wo) <= TOL


@pytest.mark.parametrize("unit", UNITS)
def test_snap(unit):
    s = system(unit, n=400)
    snap = ipg.SNAP(len(s), 2, ["Ar"], 3.0 * unit, 0.0, 0.99363, [0.5], [1.0], switch_flag=True, ctx=ipg.Context(0))
    orc = oracle.Snap(2, [0.5], [1.0], 3.0 * unit, switch=True)
    beta = np.random.default_rng(1).normal(size=(1, snap.K))
    e, f, w = snap.energy_forces(s, beta)
    eo, fo, wo = orc.energy_forces(s.positions, np.zeros(len(s), np.int32), s.L, beta)
    assert abs(e - eo) <= TOL * abs(eo) and rel_err(f, fo) <= TOL and rel_err(w, wo) <= TOL
