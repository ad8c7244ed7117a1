"""A context per thread: bases of different size at once, whose kernels take different amounts of shared memory.
Every call has to succeed and to repeat its thread's first result bit for bit.
"""
import threading

import numpy as np
import pytest

import ipg

pytestmark = pytest.mark.gpu

WORK = [(8, 200, "forces", 300), (3, 200, "forces", 600), (2, 100, "pullback", 300), (8, 64, "pullback", 150),
        (6, 100, "descriptors", 150), (4, 300, "descriptors", 150)]


def test_bases_of_different_size():
    wrong = []

    def work(twojmax, n, call, reps):
        try:
            rng = np.random.default_rng(twojmax + n)
            L = (n / 0.06) ** (1 / 3)
            s = ipg.System(rng.uniform(0, L, (n, 3)), ["A"] * n, [L] * 3)
            snap = ipg.SNAP(n, twojmax, ["A"], 4.5, 0.0, 0.99363, [0.5], [1.0], switch_flag=True, ctx=ipg.Context(0))
            beta, gF = rng.normal(size=(1, snap.K)), rng.normal(size=(n, 3))
            run = {"forces": lambda: snap.energy_forces(s, beta)[1], "pullback": lambda: snap.vjp(s, beta, 0.3, gF)[2],
                   "descriptors": lambda: ipg.compute_all_descriptors(s, snap)[1]}[call]
            first = run().copy()
            if not all(np.array_equal(run(), first) for _ in range(reps)):
                wrong.append((twojmax, call))
        except Exception as e:  # noqa: BLE001
            wrong.append((twojmax, call, str(e)))

    threads = [threading.Thread(target=work, args=w) for w in WORK]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
