"""The batch engine's task queue at its edges: one task, fewer and many more
tasks than CTAs, tasks without steps, one coset, a few and many. Every copy of
a circuit gives the same bits, and they are right. Bars as for the batch engine:
complex128 1e-12, complex64 (FP32 arithmetic) 2e-5."""
import numpy as np
import pytest

import kate_b200 as K
from kate_b200 import circuits

pytestmark = pytest.mark.gpu


def zexp(n, st):
    p = np.abs(st) ** 2
    idx = np.arange(1 << n)
    return np.array([p[((idx >> q) & 1) == 0].sum() - p[((idx >> q) & 1) == 1].sum() for q in range(n)])


@pytest.mark.parametrize("prec,tol", [(K.C128, 1e-12), (K.C64, 2e-5)])
@pytest.mark.parametrize("sizes,copies", [((3,), 1), ((13,), 1), ((1, 12, 13), 40), ((16, 18), 3), ((2, 13), 700)])
def test_queue_lengths(oracle, prec, tol, sizes, copies):
    kinds = [(n, circuits.hea(n, 2 * n, seed=n)) for n in sizes] + [(n, []) for n in sizes]
    b = K.Batch([K.Circuit(n, g) for _ in range(copies) for n, g in kinds], precision=prec)
    b.run()
    got = b.expect_z()
    for i, (n, g) in enumerate(kinds):
        assert np.abs(got[i] - zexp(n, oracle.simulate(n, g))).max() <= tol, (n, len(g))
        for c in range(1, copies):
            assert np.array_equal(got[i], got[i + c * len(kinds)]), (n, len(g), c)
