"""Fitting rows of more configurations than one dimension of a launch's grid holds (65,535), empty ones among them, and
of more than one group of the sums' buffer holds (wide quadratic columns): the set repeats a few distinct
configurations, whose rows the oracle gives, so every repeat has to match the first bit for bit.
"""
import numpy as np
import pytest

import ipg
import oracle
from conftest import TOL

pytestmark = pytest.mark.gpu


def distinct(empty):
    rng = np.random.default_rng(2)
    sizes = [1, 2, 3, 5, 4, 2] + ([0] if empty else [])
    return [ipg.System(rng.uniform(0, 4, (m, 3)), ["A"] * m, [6.0, 6.5, 7.0]) for m in sizes]


@pytest.mark.parametrize("twojmax,quadratic,nconf", [(1, False, 70001), (6, True, 5003)])
def test_fitting_rows(twojmax, quadratic, nconf):
    S = distinct(empty=not quadratic)
    snap = ipg.SNAP(1, twojmax, ["A"], 3.9, 0.0, 0.99363, [0.5], [1.0], switch_flag=True, quadratic_flag=quadratic,
                    ctx=ipg.Context(0))
    orc = oracle.Snap(twojmax, [0.5], [1.0], 3.9, switch=True, quadratic=quadratic)
    pick = np.arange(nconf) % len(S)
    Ae, Af, Aw = snap.fitting_matrices([S[q] for q in pick])
    start = np.concatenate([[0], np.cumsum([len(S[q]) for q in pick])])
    for q, s in enumerate(S):
        B, dB, W = orc.descriptors(s.positions, np.zeros(len(s), np.int32), s.L) if len(s) else (
            np.zeros((0, snap.K)), np.zeros((0, snap.K, 3)), np.zeros((snap.K, 6)))
        same = pick == q
        assert (Ae[same] == Ae[q]).all() and (Aw[same] == Aw[q]).all()
        rows = Af.reshape(-1, 3, snap.K)[start[:-1][same][:, None] + np.arange(len(s))]
        assert (rows == rows[:1]).all()
        close = lambda a, b: np.max(np.abs(a - b), initial=0.0) <= TOL * max(1.0, np.max(np.abs(b), initial=0.0))  # noqa: E731
        assert close(Ae[q], B.sum(0)) and close(rows[0], dB.transpose(0, 2, 1)) and close(Aw[q], W.T)


def test_no_launch_without_a_reader():
    """Force descriptors come out of the pass that forms the virial ones: no launch more."""
    from ipg._lib import DESC_DB, DESC_W
    rng = np.random.default_rng(4)
    s = ipg.System(rng.uniform(0, 9, (60, 3)), ["A"] * 60, [9.0] * 3)
    snap = ipg.SNAP(60, 4, ["A"], 3.0, 0.0, 0.99363, [0.5], [1.0], switch_flag=True, ctx=ipg.Context(0))

    def launches(what):
        snap._descriptors(s, what)
        k = snap.ctx.launch_count()
        snap._descriptors(s, what)
        return snap.ctx.launch_count() - k

    assert launches(DESC_DB | DESC_W) == launches(DESC_W)
