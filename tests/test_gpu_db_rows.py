"""dB/dr of the register-chain path against the oracle where a pass of 32 pairs, an output tile of
16 pairs or the three groups of components end: owners of 0, 1, 15 to 17, 31 to 33 and 65
neighbors, every twojmax of the kernel.  Bound: the repository's parity bound."""
import numpy as np
import pytest

import ipg
import oracle
from conftest import TOL

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("twojmax", range(1, 9))
def test_db_neighbor_counts(twojmax):
    rng = np.random.default_rng(twojmax)
    pos, sp = [], []
    for k, m in enumerate([1, 2, 16, 17, 18, 32, 33, 34, 66]):  # clusters of m atoms, all within the cutoff
        c = rng.normal(size=(m, 3))
        c = c / np.linalg.norm(c, axis=1)[:, None] * rng.uniform(0.6, 2.0, (m, 1))
        pos.append(c + np.array([20.0 * k, 0.0, 0.0]))
        sp.append(rng.integers(0, 2, m))
    pos, sp = np.concatenate(pos), np.concatenate(sp).astype(np.int32)
    s = ipg.System(pos, [["A", "B"][q] for q in sp], [500.0] * 3, (False, False, False))
    radii, weight = [0.5, 0.48], [1.0, 0.7]
    snap = ipg.SNAP(len(s), twojmax, ["A", "B"], 4.5, 0.0, 0.99363, radii, weight, switch_flag=True,
                    ctx=ipg.Context(0))
    orc = oracle.Snap(twojmax, radii, weight, 4.5, switch=True)
    beta = rng.normal(size=(2, snap.K))
    Bo, dBo, Wo = orc.descriptors(pos, sp, s.L)
    B, dB, W = ipg.compute_all_descriptors(s, snap)
    close = lambda a, b: np.max(np.abs(a - b)) <= TOL * np.max(np.abs(b))  # noqa: E731
    assert close(B, Bo) and close(dB, dBo.transpose(0, 2, 1)) and close(W, Wo.T)
    e, f, w = snap.energy_forces(s, beta, mode="plain")
    eo, fo, wo = orc.energy_forces(pos, sp, s.L, beta)
    assert abs(e - eo) <= TOL * abs(eo) and close(f, fo) and close(w, wo)
