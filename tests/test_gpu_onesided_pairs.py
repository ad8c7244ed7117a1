"""Pairs on one atom's list only: a shell exactly at the cutoff, where the rounding of the minimum image
differs by direction.  Such a pair still acts on both its atoms.  Without the switching function its share
is finite, so a lost reaction shows in F and dB; with it, it vanishes.

Against the oracle, which scatters every pair to both atoms, at the repository's parity bound.  The bound is of the
largest force (descriptor derivative): a shell has at most 30 pairs an atom, each of the order of the largest one.
"""
import numpy as np
import pytest

import ipg
import oracle
from conftest import TOL

pytestmark = pytest.mark.gpu

LATTICES = [(3.2, 7, 0.0), (3.2, 7, 0.3), (0.7, 8, 0.0), (0.7, 8, 0.3), (2.9, 5, 0.3)]  # edge, cells, shift


def lattice(a, m, shift, nsp=1):
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    sp = np.random.default_rng(m).integers(0, nsp, m**3).astype(np.int32)
    return ipg.System(g * a + shift, [f"S{q}" for q in sp], [m * a] * 3), sp


def one_sided(s, sp, nsp, rc):
    off, j, _ = oracle.nlist_snap(s.positions, s.L, sp, [0.5] * nsp, rc)
    i = np.repeat(np.arange(len(s)), np.diff(off))
    pairs = set(zip(i.tolist(), j.tolist()))
    return sum((k, i) not in pairs for i, k in pairs)


def close(x, ref, scale=1.0):
    return np.max(np.abs(np.asarray(x) - ref)) <= TOL * max(scale, np.max(np.abs(ref)))


@pytest.mark.parametrize("lat", LATTICES)
@pytest.mark.parametrize("switch", [False, True])
@pytest.mark.parametrize("nsp", [1, 3])
def test_reaction_reaches_the_other_atom(lat, switch, nsp):
    s, sp = lattice(*lat, nsp)
    rc = 2 * lat[0]  # the cutoff is (0.5 + 0.5) rc
    assert one_sided(s, sp, nsp, rc) > 0
    names, radii, weight = [f"S{q}" for q in range(nsp)], [0.5] * nsp, list(np.linspace(1.0, 0.6, nsp))
    snap = ipg.SNAP(len(s), 4, names, rc, 0.0, 0.99363, radii, weight, switch_flag=switch, ctx=ipg.Context(0))
    orc = oracle.Snap(4, radii, weight, rc, switch=switch)
    beta = np.random.default_rng(3).normal(0.0, 0.1, (nsp, snap.K))
    eo, fo, wo = orc.energy_forces(s.positions, sp, s.L, beta)
    results = [snap.energy_forces(s, beta, mode=m) for m in ("adjoint", "plain")]
    snap.set_skin(0.05 * lat[0])  # the list filtered from a larger one
    results.append(snap.energy_forces(s, beta))
    for e, f, w in results:
        assert close([e], [eo]) and close(f, fo)
        assert close(w, wo, abs(eo))  # a perfect lattice's virial cancels
    snap.set_skin(0.0)
    _, dBo, _ = orc.descriptors(s.positions, sp, s.L)
    assert close(ipg.compute_force_descriptors(s, snap), dBo.transpose(0, 2, 1))
    # -gE F of the position pullback, and the fitting rows of a batch
    assert close(snap.vjp(s, beta, gE=1.0, gF=np.zeros((len(s), 3)))[2], -fo)
    Af = snap.fitting_matrices([s, s])[1]
    assert close(Af.reshape(2, len(s), 3, -1), dBo.transpose(0, 2, 1)[None])


def test_replayed_and_repeated():
    s, sp = lattice(3.2, 7, 0.0)
    snap = ipg.SNAP(len(s), 4, ["S0"], 6.4, 0.0, 0.99363, [0.5], [1.0], switch_flag=False, ctx=ipg.Context(0))
    beta = np.random.default_rng(3).normal(0.0, 0.1, (1, snap.K))
    _, fo, _ = oracle.Snap(4, [0.5], [1.0], 6.4, switch=False).energy_forces(s.positions, sp, s.L, beta)
    batch = ipg.DeviceBatch(snap, [s])
    runs = [batch.evaluate(beta, graph=True)[1].cpu().numpy().copy() for _ in range(3)]
    snap.ctx.set_stream(None)
    assert close(runs[0], fo)
    assert all(np.array_equal(r, runs[0]) for r in runs[1:])  # sums in a fixed order
