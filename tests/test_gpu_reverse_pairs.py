"""Forces and descriptors gathered through each pair's reverse, where a shell lies exactly at the cutoff (the
rounding of the minimum image can then put a pair on one atom's list only), against the oracle at the
repository's parity bound.
"""
import numpy as np
import pytest

import ipg
import oracle
from conftest import TOL, rel_err

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a", [1.55, 1.1, 0.7])
@pytest.mark.parametrize("shift", [0.0, 0.3])
def test_shell_at_cutoff(a, shift):
    m = 6
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    s = ipg.System(g * a + shift, ["A"] * m**3, [m * a] * 3)
    rc = 2 * a  # the cutoff is (0.5 + 0.5) rc
    snap = ipg.SNAP(len(s), 4, ["A"], rc, 0.0, 0.99363, [0.5], [1.0], switch_flag=True, ctx=ipg.Context(0))
    orc = oracle.Snap(4, [0.5], [1.0], rc, switch=True)
    sp = np.zeros(len(s), np.int32)
    beta = np.random.default_rng(3).normal(0.0, 0.1, (1, snap.K))
    eo, fo, _ = orc.energy_forces(s.positions, sp, s.L, beta)
    e, f, _ = snap.energy_forces(s, beta)
    assert abs(e - eo) <= TOL * max(1.0, abs(eo))
    assert np.max(np.abs(f - fo)) <= TOL * max(1.0, np.max(np.abs(fo)))
    Bo, dBo, _ = orc.descriptors(s.positions, sp, s.L)
    dB = np.asarray(ipg.compute_force_descriptors(s, snap))
    assert np.max(np.abs(dB - dBo.transpose(0, 2, 1))) <= TOL * np.max(np.abs(Bo))
    assert rel_err(ipg.compute_local_descriptors(s, snap), Bo) <= TOL
