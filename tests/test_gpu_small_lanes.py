"""States whose programs have fewer threads than a warp: its other lanes
repeat them, through stages whose ops only some lanes take."""
import numpy as np
import pytest

import kate_b200 as K
from common import haar

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(K.C128, 1e-12), (K.C64, 2e-6)])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 6])
def test_repeated_lanes(n, prec, tol, oracle):
    # Gates on every pair in turn: a phase or a NOT controlled by a qubit that
    # is often a thread bit, and a dense gate that brings its target into the
    # registers. One rounding to FP32 at the end of a complex64 run.
    rng = np.random.default_rng(n)
    gates = [(2, [q], 0, None) for q in range(n)]
    for layer in range(6):
        for a in range(n):
            b = (a + 1 + layer % (n - 1)) % n
            gates += [(0, [a], 0, haar(2, rng)), (4, [b, a], 1 + layer, None), (3, [b, a], 0, None)]
    sim = K.Simulator(K.Circuit(n, gates), 1, prec, 0)
    assert sim.launches_per_run() == (1 if prec == K.C128 else 3)
    sim.execute()
    first = sim.state()
    assert np.abs(first - oracle.simulate(n, gates)).max() <= tol
    for _ in range(50):
        sim.execute()
        assert np.array_equal(sim.state(), first)
