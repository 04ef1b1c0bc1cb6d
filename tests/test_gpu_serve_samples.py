"""Served samples are the simulator's for the same seed (as a set: the server
returns them in the order of their uniforms): dense states over one and several
65536-amplitude chunks, and states whose probability sits in a few amplitudes
at the edges of chunks and 256-amplitude runs."""
import numpy as np
import pytest

import kate_b200 as K
from kate_b200 import circuits

pytestmark = pytest.mark.gpu


def ghz(n):
    return [(2, [0], 0, None)] + [(3, [q + 1, q], 0, None) for q in range(n - 1)]


def edge(n, bits):
    # H on one qubit, X on others: two amplitudes, 2^bit apart, inside one run or in different ones.
    x = np.array([[0, 1], [1, 0]], dtype=complex)
    return [(2, [bits[0]], 0, None)] + [(0, [b], 0, x) for b in bits[1:]]


CASES = [(n, "layered") for n in (12, 13, 16, 17, 18)] + [(12, "ghz"), (17, "ghz"), (16, (7, 8)), (16, (8, 0, 1, 2)),
                                                          (18, (16, 15, 14)), (13, (12, 11, 10, 9, 8))]


def test_served_samples_are_the_simulators():
    srv = K.Server(K.C128, budget_bytes=1 << 30, aux_bytes=256 << 20)
    todo = []
    for i, (n, what) in enumerate(CASES):
        g = circuits.layered(n, 3, seed=n) if what == "layered" else ghz(n) if what == "ghz" else edge(n, what)
        c = K.Circuit(n, g)
        shots = (1, 777, 4096)[i % 3]
        todo.append((c, shots, 100 + i, srv.submit(c, shots=shots, seed=100 + i)))
    for c, shots, seed, rid in todo:
        _, got, _ = srv.wait(rid, timeout=120)
        sim = K.Simulator(c)
        sim.execute()
        assert np.array_equal(np.sort(got), np.sort(sim.sample(shots, seed=seed)))
    srv.close()
