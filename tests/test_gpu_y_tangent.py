"""The one-pass tangent of Y in the position pullback against the per-atom forward-mode kernel
(IPG_GENERIC_HVP=1) at the sizes where its tiles end: one atom, one tile of 32 and one atom more,
every twojmax, eight species.  Both are exact, so they agree to rounding (1e-12 of the largest
component, the bound of the kernels' comparison at ordinary sizes)."""
import numpy as np
import pytest

import ipg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("twojmax", range(0, 9))
@pytest.mark.parametrize("n", [1, 32, 33])
def test_tangent_tiles(twojmax, n, monkeypatch):
    rng = np.random.default_rng(100 * twojmax + n)
    names = [f"S{q}" for q in range(8)]
    L = 4.0 + 1.2 * n ** (1 / 3)
    s = ipg.System(rng.uniform(0, L, (n, 3)), [names[q] for q in rng.integers(0, 8, n)], [L] * 3)
    args = (n, twojmax, names, 3.6, 0.0, 0.97, list(np.linspace(0.5, 0.45, 8)), list(np.linspace(1.0, 0.6, 8)))
    fast = ipg.SNAP(*args, switch_flag=True)
    monkeypatch.setenv("IPG_GENERIC_HVP", "1")
    slow = ipg.SNAP(*args, switch_flag=True)
    beta = rng.normal(0, 1e-1, (8, len(fast)))
    gF = rng.normal(size=(n, 3))
    g1, g2 = fast.vjp(s, beta, 0.25, gF)[2], slow.vjp(s, beta, 0.25, gF)[2]
    assert np.max(np.abs(g1 - g2)) <= 1e-12 * max(1.0, np.max(np.abs(g2)))
