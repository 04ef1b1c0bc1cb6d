"""Dense gates of three to five qubits in pass-specialised kernels: on the
shared tile between register stages, first or last in a pass, against the
oracle; a pass with more matrices than kernel parameters hold keeps the
interpreter."""
import os

import numpy as np
import pytest

import kate_b200 as K
from kate_b200 import circuits
from common import haar

pytestmark = pytest.mark.gpu


def dense(n, sizes, seed, between):
    r = np.random.default_rng(seed)
    g = []
    for i, k in enumerate(sizes):
        g.append((0, [int(x) for x in r.choice(n, k, replace=False)], 0, haar(1 << k, r)))
        for _ in range(between):
            q = [int(x) for x in r.choice(n, 2, replace=False)]
            g.append((2, q[:1], 0, None) if r.random() < 0.5 else (3, q, 0, None))
    return g


@pytest.mark.parametrize("n", [12, 13, 16])
@pytest.mark.parametrize("sizes,between", [([3], 0), ([4], 2), ([5], 3), ([3, 4, 5, 2], 0), ([5, 3, 4], 6),
                                           ([1, 3, 2, 3, 4], 4)])
def test_dense_gates_match_oracle(n, sizes, between, oracle):
    # At most 40 gates: a few roundings of 32-term sums each, below 1e-13.
    g = dense(n, sizes, n + len(sizes), between)
    for gates in (g, circuits.layered(n, 1, seed=n) + g):
        sim = K.Simulator(K.Circuit(n, gates))
        assert all(k == 2 for k in sim.pass_kernels())
        sim.execute()
        assert np.abs(sim.state() - oracle.simulate(n, gates)).max() <= 1e-12


def test_more_matrices_than_parameters_keep_the_interpreter(oracle):
    n = 12
    g = dense(n, [5, 5, 5, 5], 3, 0)
    sim = K.Simulator(K.Circuit(n, g))
    assert 1 in sim.pass_kernels()
    sim.execute()
    assert np.abs(sim.state() - oracle.simulate(n, g)).max() <= 1e-12


@pytest.mark.parametrize("family", ["layered", "hea"])
def test_compiled_circuits_match_the_interpreter(family):
    # The compile passes relabel qubits, so the interpreter (checked against
    # the reference's compiled states elsewhere) gives the state to compare.
    n = 17
    c = K.Circuit(n, getattr(circuits, family)(n, 4, seed=5))
    c.compileOPT(5, 1e-6, 10)
    states = []
    for jit in ("1", "0"):
        old = os.environ.get("KATE_JIT")
        os.environ["KATE_JIT"] = jit
        try:
            sim = K.Simulator(c)
        finally:
            if old is None:
                del os.environ["KATE_JIT"]
            else:
                os.environ["KATE_JIT"] = old
        sim.execute()
        states.append(sim.state())
    assert np.abs(states[0] - states[1]).max() <= 1e-12


@pytest.mark.parametrize("n", [12, 13, 16])
@pytest.mark.parametrize("sizes,between", [([3], 0), ([4], 1), ([5], 2), ([4, 3, 5], 0), ([5, 4], 4)])
def test_first_pass_starting_with_a_dense_gate(n, sizes, between, oracle):
    # It makes |0...0> or the product state itself: no launch besides the passes.
    g = dense(n, sizes, 31 * n + len(sizes), between)
    rng = np.random.default_rng(n)
    tp = np.stack([rng.uniform(0, 1, n), rng.uniform(-np.pi, np.pi, n)], axis=1)
    sim = K.Simulator(K.Circuit(n, g))
    assert sim.launches_per_run() == len(sim.pass_kernels())
    sim.execute()
    assert np.abs(sim.state() - oracle.simulate(n, g)).max() <= 1e-12
    sim.execute(K.proba_state(tp))
    assert np.abs(sim.state() - oracle.simulate(n, g, proba_in=tp)).max() <= 1e-12
