"""States of fewer than 12 qubits: the whole circuit in one launch of one CTA
(every tile size from the padded one to four warps), against the oracle."""
import numpy as np
import pytest

import kate_b200 as K
from kate_b200 import circuits
from common import random_circuit

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(K.C128, 1e-12), (K.C64, 2e-6)])
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 8, 9, 10, 11])
def test_every_gate_kind_over_several_programs(n, prec, tol, oracle):
    # 400 gates: more than one program (96 gates each), three- to five-qubit
    # dense gates between register stages. One rounding to FP32 at the end of
    # a complex64 run (the norm is 1): far below 2e-6.
    rng = np.random.default_rng(n)
    gates = random_circuit(n, 400, rng) if n > 1 else random_circuit(n, 400, rng, kinds=("h", "d1", "diag1"))
    sim = K.Simulator(K.Circuit(n, gates), 1, prec, 0)
    assert sim.launches_per_run() == (1 if prec == K.C128 else 3)
    want = oracle.simulate(n, gates)
    for _ in range(2):
        got = sim.execute()
        assert np.abs(sim.state() - want).max() <= tol
    assert np.abs(got.as_array() - sim.proba().as_array()).max() <= 1e-9 if prec == K.C128 else True


@pytest.mark.parametrize("n", [3, 7, 10, 11])
def test_product_start_and_timed_run(n, oracle):
    gates = circuits.layered(n, 12, seed=n)
    r = np.random.default_rng(n)
    tp = np.stack([r.uniform(0.1, 0.9, n), r.uniform(-3, 3, n)], axis=1)
    sim = K.Simulator(K.Circuit(n, gates))
    sim.execute(K.proba_state(tp))
    # The product state as the oracle's start: each qubit's factor as a dense gate on |0>.
    first = []
    for q in range(n):
        t, p = tp[q, 0] * np.pi / 2, tp[q, 1]
        a = np.array([[np.cos(t), -np.sin(t)], [np.exp(1j * p) * np.sin(t), np.exp(1j * p) * np.cos(t)]])
        first.append((0, [q], 0, a))
    want = oracle.simulate(n, first + gates)
    assert np.abs(sim.state() - want).max() <= 1e-12
    init_ms, ms = sim.profile_passes()  # one launch per program, from |0...0>
    assert len(ms) == len(sim.passes())
    assert np.abs(sim.state() - oracle.simulate(n, gates)).max() <= 1e-12
