"""A replayed graph whose pair count still fits, but one of whose atoms has more neighbors than the padded
walk has slots for: the call runs again eagerly.  The list of the replay that is thrown away has to hold valid
atoms in the slots that were not written, also where the buffer still has the atoms of a larger system.
"""
import numpy as np
import pytest

import ipg
from ipg import workloads as W

pytestmark = pytest.mark.gpu


def test_more_neighbors_than_slots():
    import torch
    big, prm, beta = W.snap_j8(cells=14)
    snap = ipg.SNAP(1, prm["twojmax"], prm["species"], prm["rcutfac"], prm["rmin0"], prm["rfac0"], prm["radii"],
                    prm["weight"], switch_flag=True, ctx=ipg.Context(0))
    snap.energy_forces(big, beta)
    snap.energy_forces(big, beta)
    small, _, _ = W.snap_j8(cells=5)
    db = ipg.DeviceBatch(snap, [small])
    for _ in range(2):
        db.evaluate(beta, graph=True)
    rng = np.random.default_rng(0)
    pos = small.positions.copy()
    pos[1:40] = pos[0] + rng.uniform(-1.5, 1.5, (39, 3))  # about 39 neighbors more for a few atoms
    moved = ipg.System(pos, small.symbols, small.box, small.periodic)
    db.set_positions(pos)
    E, F, V = db.evaluate(beta, graph=True)
    torch.cuda.synchronize()
    snap.ctx.set_stream(None)
    E1, F1, V1 = snap.batch_energy_forces([moved], beta)
    assert np.array_equal(E.cpu().numpy(), E1) and np.array_equal(F.cpu().numpy(), F1)
    assert np.array_equal(V.cpu().numpy(), V1)


def test_collapse():
    """Every atom a neighbor of every other: lists cut at the capacity and at the slots."""
    import torch
    n, L = 1000, 42.0
    rng = np.random.default_rng(1)
    pos = rng.uniform(0, L, (n, 3))
    s = ipg.System(pos, ["A"] * n, [L] * 3)
    snap = ipg.SNAP(n, 2, ["A"], 5.0, 0.0, 0.99363, [0.5], [1.0], switch_flag=True, ctx=ipg.Context(0))
    beta = rng.normal(size=(1, snap.K))
    db = ipg.DeviceBatch(snap, [s])
    for _ in range(2):
        db.evaluate(beta, graph=True)
    small = 21.0 + rng.uniform(-1.2, 1.2, (n, 3))
    db.set_positions(small)
    E, F, _ = db.evaluate(beta, graph=True)
    torch.cuda.synchronize()
    snap.ctx.set_stream(None)
    E1, F1, _ = snap.batch_energy_forces([ipg.System(small, s.symbols, s.box)], beta)
    assert np.array_equal(E.cpu().numpy(), E1) and np.array_equal(F.cpu().numpy(), F1)
