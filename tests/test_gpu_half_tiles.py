"""The half-stencil pair walk's 32-bit candidate test against the oracle where it could lose or
double a pair: neighbors exactly at the cutoff, atoms on cell boundaries and whole box lengths
outside the box, cell populations around the 32-row tile, and sparse open axes with huge cells.

Bounds: the pair sums are a few hundred products of 64-bit values, so 1e-10 relative (the
repository's parity bound) is far above rounding and far below one lost pair.
"""
import numpy as np
import pytest

import ipg
from conftest import TOL, rel_err
from test_gpu_pair import oracle_eval

pytestmark = pytest.mark.gpu


def grid(nx, ny, nz, a):
    g = np.stack(np.meshgrid(np.arange(nx), np.arange(ny), np.arange(nz), indexing="ij"), -1).reshape(-1, 3)
    return g * a


def at_cutoff():
    # simple cubic: the second shell lies exactly at rcut, every atom on a cell boundary
    return ipg.System(grid(8, 7, 9, 1.5), ["Ar"] * 504, [12.0, 10.5, 13.5]), 3.0


def outside_box():
    rng = np.random.default_rng(1)
    pos = rng.uniform(0, 14, (777, 3)) + 14.0 * rng.integers(-3, 4, (777, 3))
    pos[:8] = 14.0 * np.array([[0, 0, 0], [1, 0.5, 0.5], [0.5, 1, 0], [-1, 0.5, 0.25], [2, 0.25, 0], [0, 0.75, 1],
                               [1e-17, 0.6, 0.1], [-1e-17, 0.4, 0.9]])
    return ipg.System(pos, ["Ar"] * 777, [14.0] * 3), 3.1


def cell_population(m):
    # m atoms in one cell of a 4 x 4 x 4 grid, a few in the others
    rng = np.random.default_rng(m)
    pos = np.concatenate([rng.uniform(0.01, 3.99, (m, 3)) + 4.0, rng.uniform(0, 16, (97, 3))])
    return ipg.System(pos, ["Ar"] * len(pos), [16.0] * 3), 4.0


def open_sparse():
    rng = np.random.default_rng(5)
    pos = rng.normal(0, 2.0, (64, 3)) + 1e5 * rng.integers(0, 3, (64, 1)) * np.array([[1.0, 0.0, 0.0]])
    return ipg.System(pos, ["Ar"] * 64, [9.0, 9.0, 9.0], (False, True, False)), 2.9


CASES = {"at_cutoff": at_cutoff, "outside_box": outside_box, "open_sparse": open_sparse}
CASES.update({f"cell_{m}": (lambda m=m: cell_population(m)) for m in (1, 31, 32, 33, 64, 65)})


@pytest.mark.parametrize("case", sorted(CASES))
def test_half_tiles_edges(case):
    s, rc = CASES[case]()
    # terms that stay of order one at any distance, so that no close pair hides a lost one
    p = ipg.Morse(0.1, 0.5, 1.5, rc, ["Ar"]) + 0.5 * ipg.BornMayer(0.3, 0.7, 1.0, 0.0, 0.0, 0.8 * rc, ["Ar"])
    e, f, w = ipg.empirical.pair_eval(s, ipg.empirical.empirical_terms(p), ctx=ipg.Context(0))
    eo, fo, wo = oracle_eval(s, p)
    assert abs(e - eo) <= TOL * abs(eo)
    scale = np.max(np.abs(fo)) if case != "at_cutoff" else 1e-2  # a perfect lattice's forces cancel
    assert np.max(np.abs(f - fo)) <= TOL * scale
    assert rel_err(w, wo) <= TOL


# terms of one cutoff with species filters, and of several cutoffs: a warp's lanes then differ in the terms they need
TERMS = {
    "one_cutoff": [("Ar", "Ne"), ("Ar",), ("Ne",), ("Kr", "Ar")],
    "cutoffs": [("Ar", "Ne", "Kr"), ("Ar",), ("Ne", "Kr"), ("Kr",)],
}


@pytest.mark.parametrize("case", sorted(TERMS))
@pytest.mark.parametrize("n", [1, 2, 33, 700])
def test_half_tiles_mixed_terms(case, n):
    rng = np.random.default_rng(n)
    L = max(6.5, (n / 0.25) ** (1 / 3))
    s = ipg.System(rng.uniform(0, L, (n, 3)), list(rng.choice(["Ar", "Ne", "Kr"], n)), [L] * 3)
    p = None
    for t, names in enumerate(TERMS[case]):
        rc = 3.0 if case == "one_cutoff" else 3.0 - 0.4 * t
        q = (0.5 + 0.25 * t) * ipg.Morse(0.1 + 0.1 * t, 0.5, 1.5, rc, list(names))
        p = q if p is None else p + q
    e, f, w = ipg.empirical.pair_eval(s, ipg.empirical.empirical_terms(p), ctx=ipg.Context(0))
    eo, fo, wo = oracle_eval(s, p)
    assert abs(e - eo) <= TOL * max(abs(eo), 1e-300)
    assert np.max(np.abs(f - fo), initial=0.0) <= TOL * max(np.max(np.abs(fo)), 1e-300)
    assert rel_err(w, wo) <= TOL
