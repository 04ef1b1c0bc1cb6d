"""Runs from |0...0> skip the cosets of qubits that no pass has held yet (they
are zero); runs from a product state skip nothing. Circuits that leave qubits
out, reach them late or take them in any order, on every kernel, against the
oracle, with both starts on one simulator so that the buffer holds an old
state."""
import ctypes
import os

import numpy as np
import pytest

import kate_b200 as K
from kate_b200 import _lib, circuits
from common import haar, random_circuit

pytestmark = pytest.mark.gpu


def late(n, seed):
    # Layers on a window that moves over the qubits in a random order.
    r = np.random.default_rng(seed)
    perm = [int(q) for q in r.permutation(n)]
    g = []
    for w in range(0, n, 3):
        qs = perm[max(0, w - 6):w + 3]
        for _ in range(3 * len(qs)):
            g.append((2, [qs[r.integers(len(qs))]], 0, None))
            if len(qs) > 1:
                a, b = (int(x) for x in r.choice(qs, 2, replace=False))
                g.append((3, [a, b], 0, None))
                g.append((0, [a, b], 0, haar(4, r)))
    return g


def cases(n):
    yield "late", late(n, n)
    yield "part", late(n - 2, n + 1)  # the last two qubits are never touched
    yield "layered", circuits.layered(n, 2, seed=n)
    yield "random", random_circuit(n, 90, np.random.default_rng(n))


@pytest.mark.parametrize("jit", ["1", "0"])
@pytest.mark.parametrize("n", [12, 13, 16, 21])
def test_complex128(n, jit, oracle):
    rng = np.random.default_rng(n)
    tp = np.stack([rng.uniform(0, 1, n), rng.uniform(-np.pi, np.pi, n)], axis=1)
    for name, g in cases(n):
        old = os.environ.get("KATE_JIT")
        os.environ["KATE_JIT"] = jit
        try:
            sim = K.Simulator(K.Circuit(n, g))
        finally:
            if old is None:
                del os.environ["KATE_JIT"]
            else:
                os.environ["KATE_JIT"] = old
        zero, prod = oracle.simulate(n, g), oracle.simulate(n, g, proba_in=tp)
        for start in (0, 1, 0):
            sim.execute(K.proba_state(tp)) if start else sim.execute()
            # A few hundred gates, each some roundings of the amplitudes it touches.
            assert np.abs(sim.state() - (prod if start else zero)).max() <= 1e-12, (name, start)
        sim.close()


@pytest.mark.parametrize("n", [13, 16, 21])
def test_complex64(n, oracle):
    for name, g in (("late", late(n, n)), ("part", late(n - 2, n + 1)), ("brickwork", circuits.brickwork_su4(n, 3))):
        sim = K.Simulator(K.Circuit(n, g), 1, K.C64, 0)
        assert set(sim.pass_kernels()) == {3}
        ref = oracle.simulate(n, g)
        for _ in range(2):
            sim.execute()
            assert np.abs(sim.state() - ref).max() <= 1e-4, name
        sim.close()


@pytest.mark.parametrize("prec,blocks,tol", [(K.C128, 0, 1e-12), (K.C64, 0, 2e-5), (K.C64, 1, 2e-5)])
def test_batch(oracle, prec, blocks, tol):
    # Bars as for the batch engine; two runs, so that the arena holds old states.
    specs = [(n, g) for n in (13, 16, 18) for g in (late(n, n), late(n - 2, n + 1), circuits.hea(n, n, seed=n), [])]
    opts = _lib.BatchOptions()
    _lib.lib().kate_batch_options_default(ctypes.byref(opts))
    for n, _ in specs:
        opts.tune[n].blocks = blocks
    b = K.Batch([K.Circuit(n, g) for n, g in specs], precision=prec, options=opts)
    for _ in range(2):
        b.run()
        for (n, g), z in zip(specs, b.expect_z()):
            p = np.abs(oracle.simulate(n, g)) ** 2
            x = np.arange(1 << n)
            want = [p[(x >> q) & 1 == 0].sum() - p[(x >> q) & 1 == 1].sum() for q in range(n)]
            assert np.abs(z - want).max() <= tol, (n, len(g))
