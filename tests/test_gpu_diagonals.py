"""Diagonals and phases in the pass-specialised kernels are gathered per thread
(factors of thread bits, of coset bits, of one register bit) and multiplied in
late: circuits made of little else, against the oracle, over one and many
cosets and from every kind of start."""
import numpy as np
import pytest

import kate_b200 as K
from kate_b200 import circuits

pytestmark = pytest.mark.gpu


def phases(n, count, seed):
    # Phases and diagonals on random qubits between H, CNOT and TOFFOLI gates that move the bits they depend on.
    r = np.random.default_rng(seed)
    g = []
    for i in range(count):
        q = [int(x) for x in r.choice(n, 3, replace=False)]
        k = i % 8
        if k in (0, 3):
            g.append((2, q[:1], 0, None))
        elif k in (1, 4, 6):
            g.append((4, q[:2], int(r.integers(1, 9)), None))
        elif k == 2:
            g.append((0, q[:1], 0, np.diag(np.exp(1j * r.uniform(0, 6, 2)))))
        elif k == 5:
            g.append((0, q, 0, np.diag(np.exp(1j * r.uniform(0, 6, 8)))))
        else:
            g.append((3, q[:2], 0, None) if i % 16 == 7 else (5, q, 0, None))
    return g


@pytest.mark.parametrize("n,count", [(12, 200), (13, 300), (17, 400), (20, 300)])
def test_phase_circuits_match_oracle(n, count, oracle):
    # Unit factors: each costs an amplitude a few roundings, far below 1e-12 over 400 gates.
    g = phases(n, count, n)
    sim = K.Simulator(K.Circuit(n, g))
    assert all(k == 2 for k in sim.pass_kernels())
    sim.execute()
    assert np.abs(sim.state() - oracle.simulate(n, g)).max() <= 1e-12
    r = np.random.default_rng(n + 1)
    tp = np.stack([r.uniform(0.1, 0.9, n), r.uniform(-3, 3, n)], axis=1)
    first = []
    for q in range(n):
        t, p = tp[q, 0] * np.pi / 2, tp[q, 1]
        first.append((0, [q], 0, np.array([[np.cos(t), -np.sin(t)],
                                           [np.exp(1j * p) * np.sin(t), np.exp(1j * p) * np.cos(t)]])))
    sim.execute(K.proba_state(tp))
    assert np.abs(sim.state() - oracle.simulate(n, first + g)).max() <= 1e-12


@pytest.mark.parametrize("n", [12, 15, 19])
def test_qft_and_ansatz_match_oracle(n, oracle):
    for g in (circuits.qft(n), circuits.hea(n, 6, seed=n)):
        sim = K.Simulator(K.Circuit(n, g))
        sim.execute()
        assert np.abs(sim.state() - oracle.simulate(n, g)).max() <= 1e-12
