"""The adjoint route of chem_flag and quadratic SNAP against the oracle (and the dB/dr route of the
plain mode): one atom, a tile of 32 atoms and one more, three elements (a second pass over Z per
three elements is reached with four), bzero and wselfall; and a batch of two equal configurations
whose atoms straddle a chunk of Z.  Bound: the repository's parity bound; equal configurations
agree to rounding."""
import numpy as np
import pytest

import ipg
import oracle
from conftest import TOL
from test_gpu_y_stream import system

pytestmark = pytest.mark.gpu


def close(a, b):
    return np.max(np.abs(np.asarray(a) - b)) <= TOL * max(1.0, np.max(np.abs(b)))


@pytest.mark.parametrize("twojmax,nsp,opts", [
    (1, 2, {}), (2, 4, {}), (3, 3, {"wselfall": True}), (4, 2, {"bzero": True}), (6, 2, {}), (8, 2, {"bzero": True}),
    (2, 1, {"quadratic": True}), (5, 2, {"quadratic": True}), (8, 1, {"quadratic": True, "bzero": True})])
@pytest.mark.parametrize("n", [1, 33])
def test_adjoint_route(twojmax, nsp, opts, n):
    quad, bzero, wself = opts.get("quadratic", False), opts.get("bzero", False), opts.get("wselfall", False)
    s, sp = system(n, nsp, 7 * twojmax + n)
    radii, weight = list(np.linspace(0.5, 0.45, nsp)), list(np.linspace(1.0, 0.6, nsp))
    snap = ipg.SNAP(n, twojmax, [f"S{q}" for q in range(nsp)], 4.4, 0.0, 0.99363, radii, weight, chem_flag=not quad,
                    bnorm_flag=not quad, bzero_flag=bzero, switch_flag=True, wselfall_flag=wself,
                    quadratic_flag=quad, ctx=ipg.Context(0))
    orc = oracle.Snap(twojmax, radii, weight, 4.4, bzero=bzero, bnorm=not quad, switch=True, chem=not quad,
                      wselfall=wself, quadratic=quad)
    beta = np.random.default_rng(n).normal(0.0, 1e-2, (nsp, snap.K))
    e, f, w = snap.energy_forces(s, beta, mode="adjoint")
    eo, fo, wo = orc.energy_forces(s.positions, sp, s.L, beta)
    assert close([e], [eo]) and close(f, fo) and close(w, wo)
    ep, fp, _ = snap.energy_forces(s, beta, mode="plain")
    assert close([e], [ep]) and close(f, fp)


def test_chunks_of_z():
    n = 14200  # 2 n atoms: one more than a chunk of Z holds (4 GiB, two elements, twojmax 8)
    s, _ = system(n, 2, 3)
    snap = ipg.SNAP(n, 8, ["S0", "S1"], 4.4, 0.0, 0.99363, [0.5, 0.47], [1.0, 0.6], chem_flag=True, bnorm_flag=True,
                    switch_flag=True, ctx=ipg.Context(0))
    beta = np.random.default_rng(1).normal(0.0, 1e-2, (2, snap.K))
    E, F, W = snap.batch_energy_forces([s, s], beta)
    scale = np.max(np.abs(F[:n]))
    assert abs(E[1] - E[0]) <= 1e-12 * abs(E[0]) and np.max(np.abs(F[n:] - F[:n])) <= 1e-12 * scale
