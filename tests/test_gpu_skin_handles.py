"""Verlet skins of several SNAP handles on one context: each handle reuses the list that it built, whatever the
others build in between, and gives its buffers back when it is closed.
"""
import numpy as np
import pytest

import ipg
from conftest import TOL, rel_err

pytestmark = pytest.mark.gpu


def test_each_handle_reuses_its_own_list():
    rng = np.random.default_rng(6)
    ctx = ipg.Context(0)
    # the same system for a short and a long cutoff, and a larger one
    pos = {"small": rng.uniform(0, 14, (300, 3)), "large": rng.uniform(0, 30, (2500, 3))}
    box = {"small": 14.0, "large": 30.0}
    kinds = [("small", 3.0), ("small", 4.5), ("large", 3.5)]
    snaps, fresh, beta = [], [], []
    for k, (name, rc) in enumerate(kinds):
        args = (1, 3, ["A"], rc, 0.0, 0.99363, [0.5], [1.0])
        snaps.append(ipg.SNAP(*args, switch_flag=True, ctx=ctx))
        snaps[-1].set_skin(0.5)
        fresh.append(ipg.SNAP(*args, switch_flag=True, ctx=ipg.Context(0)))
        beta.append(rng.normal(size=(1, snaps[-1].K)))
    for step in range(4):
        for k in (0, 1, 2, 1, 0):
            name, _ = kinds[k]
            s = ipg.System(pos[name] + 0.02 * step, ["A"] * len(pos[name]), [box[name]] * 3)
            e, f, w = snaps[k].energy_forces(s, beta[k])
            e0, f0, w0 = fresh[k].energy_forces(s, beta[k])
            assert abs(e - e0) <= TOL * abs(e0) and rel_err(f, f0) <= TOL and rel_err(w, w0) <= TOL
    assert [s.skin_stats()[0] for s in snaps] == [1, 1, 1]


def test_buffers_are_given_back():
    import torch
    rng = np.random.default_rng(7)
    ctx = ipg.Context(0)
    s = ipg.System(rng.uniform(0, 60, (20000, 3)), ["A"] * 20000, [60.0] * 3)
    free = []
    for _ in range(4):
        snap = ipg.SNAP(1, 1, ["A"], 4.0, 0.0, 0.99363, [0.5], [1.0], switch_flag=True, ctx=ctx)
        snap.set_skin(0.5)
        snap.energy_forces(s, rng.normal(size=(1, snap.K)))
        snap.close()
        free.append(torch.cuda.mem_get_info()[0])
    assert free[-1] >= free[1] - (1 << 20)
