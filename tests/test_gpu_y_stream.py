"""The streamed Clebsch-Gordan contraction (Y, Z, and both) against the oracle at the sizes where
its tiles and streams end: one atom, a tile of 32 atoms and one more, every twojmax of the kernel,
and eight species (the largest coefficient table).  Bound: the repository's parity bound."""
import numpy as np
import pytest

import ipg
import oracle
from conftest import TOL, rel_err

pytestmark = pytest.mark.gpu


def system(n, nsp, seed):
    rng = np.random.default_rng(seed)
    L = max(9.0, 3.0 * n ** (1.0 / 3.0))
    k = int(np.ceil(n ** (1.0 / 3.0)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
    pos = (g + 0.5) * (L / k) + rng.normal(0.0, 0.2, (n, 3))
    sp = rng.integers(0, nsp, n).astype(np.int32)
    return ipg.System(pos, [f"S{q}" for q in sp], [L] * 3), sp


@pytest.mark.parametrize("twojmax", range(1, 9))
@pytest.mark.parametrize("n,nsp", [(1, 1), (32, 2), (33, 8)])
def test_contraction_tiles(twojmax, n, nsp):
    s, sp = system(n, nsp, 10 * twojmax + n)
    radii, weight = list(np.linspace(0.5, 0.45, nsp)), list(np.linspace(1.0, 0.6, nsp))
    snap = ipg.SNAP(n, twojmax, [f"S{q}" for q in range(nsp)], 4.4, 0.0, 0.99363, radii, weight, switch_flag=True,
                    ctx=ipg.Context(0))
    orc = oracle.Snap(twojmax, radii, weight, 4.4, switch=True)
    rng = np.random.default_rng(n)
    beta = rng.normal(0.0, 1e-1, (nsp, snap.K))
    gF = rng.normal(0.0, 1.0, (n, 3))
    e, f, w = snap.energy_forces(s, beta)  # Y
    eo, fo, wo = orc.energy_forces(s.positions, sp, s.L, beta)
    assert abs(e - eo) <= TOL * max(1.0, abs(eo))
    assert np.max(np.abs(f - fo)) <= TOL * max(1.0, np.max(np.abs(fo)))
    B = ipg.compute_local_descriptors(s, snap)  # Z
    assert rel_err(B, orc.descriptors(s.positions, sp, s.L)[0]) <= TOL
    gb, _, _ = snap.vjp(s, beta, 0.3, gF)  # Y and Z
    gbo = orc.vjp_beta(s.positions, sp, s.L, 0.3, gF)[0]
    assert np.max(np.abs(gb - gbo)) <= TOL * max(1.0, np.max(np.abs(gbo)))


@pytest.mark.parametrize("copies", [97, 256, 385])
@pytest.mark.parametrize("twojmax", [3, 8])
def test_contraction_many_tiles(twojmax, copies):
    # copies of one cluster beyond each other's cutoff: every copy gives the cluster's values, whether its tile
    # is split over blocks, has one of its own, or is one of several of a block
    m, rc = 37, 3.0
    rng = np.random.default_rng(twojmax)
    c = np.round(rng.uniform(0, 6.0, (m, 3)) * 2**20) / 2**20
    k = int(np.ceil(copies ** (1 / 3)))
    g = np.stack(np.meshgrid(*[np.arange(k)] * 3, indexing="ij"), -1).reshape(-1, 3)[:copies]
    pos = (10.0 * g[:, None, :] + c[None]).reshape(-1, 3)
    n = len(pos)
    one, s = ipg.System(c, ["A"] * m, [10.0 * k] * 3), ipg.System(pos, ["A"] * n, [10.0 * k] * 3)
    snap = ipg.SNAP(n, twojmax, ["A"], rc, 0.0, 0.99363, [0.5], [1.0], switch_flag=True, ctx=ipg.Context(0))
    orc = oracle.Snap(twojmax, [0.5], [1.0], rc, switch=True)
    sp = np.zeros(m, np.int32)
    beta = rng.normal(0.0, 1e-1, (1, snap.K))
    g1 = rng.normal(0.0, 1.0, (m, 3))
    eo, fo, _ = orc.energy_forces(one.positions, sp, one.L, beta)
    e, f, _ = snap.energy_forces(s, beta)
    assert abs(e - copies * eo) <= TOL * max(1.0, abs(copies * eo))
    assert np.max(np.abs(f.reshape(copies, m, 3) - fo)) <= TOL * max(1.0, np.max(np.abs(fo)))
    B = np.asarray(ipg.compute_local_descriptors(s, snap)).reshape(copies, m, -1)
    Bo = orc.descriptors(one.positions, sp, one.L)[0].reshape(m, -1)
    assert np.max(np.abs(B - Bo)) <= TOL * np.max(np.abs(Bo))
    gb, _, _ = snap.vjp(s, beta, 0.3, np.tile(g1, (copies, 1)))
    gbo = orc.vjp_beta(one.positions, sp, one.L, 0.3, g1)[0]
    assert np.max(np.abs(gb - copies * gbo)) <= TOL * max(1.0, copies * np.max(np.abs(gbo)))
