"""Measurement reductions at the sizes where their split of the index changes:
single CTA, one tile per CTA, several rounds per CTA, both amplitude types."""
import math

import numpy as np
import pytest

import kate_b200 as K

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,tol", [(K.C128, 1e-12), (K.C64, 2e-5)])
@pytest.mark.parametrize("n", [1, 2, 5, 8, 11, 12, 13, 17, 22, 23, 25, 26, 27, 28])
def test_product_state_measures_its_own_angles(n, prec, tol):
    # An empty circuit leaves the product state: the amplitudes' sums factor
    # per qubit, so (theta, phi) come back (phi folded into (-pi/2, pi/2) by
    # the reference's atan), and <Z> is cos^2 - sin^2. Sums of 2^n products
    # of n factors carry n + log2(dim) roundings: far below the bounds.
    r = np.random.default_rng(n)
    th = r.uniform(0.2, 0.8, n)
    ph = r.uniform(-1.2, 1.2, n)
    sim = K.Simulator(K.Circuit(n), 1, prec, 0)
    out = sim.execute(K.proba_state(np.stack([th, ph], axis=1))).as_array()
    assert np.abs(out[:, 0] - th).max() <= tol
    assert np.abs(out[:, 1] - ph).max() <= tol
    assert np.abs(sim.proba().as_array() - out).max() <= tol
    z = np.cos(th * math.pi / 2) ** 2 - np.sin(th * math.pi / 2) ** 2
    assert np.abs(sim.expect_z() - z).max() <= tol


@pytest.mark.parametrize("shots", [1, 2048, 2049, 5000])
@pytest.mark.parametrize("n", [3, 12, 14, 18])
def test_samples_at_chunk_edges(n, shots):
    # A few amplitudes at the edges of 4096-amplitude chunks, whole chunks of
    # probability 0 between and after them.
    dim = 1 << n
    at = sorted({i for i in (0, 1, 511, 512, 4095, 4096, 8191, 3 * 4096 + 7, dim // 2 + 1) if i < dim})
    st = np.zeros(dim, dtype=np.complex128)
    st[at] = np.sqrt(np.arange(1.0, len(at) + 1)) * np.exp(1j * np.arange(len(at)))
    st /= np.linalg.norm(st)
    sim = K.Simulator(K.Circuit(n))
    sim.set_state(st)
    got = sim.sample(shots, seed=5)
    state, want = 5, []
    p = np.abs(st) ** 2
    cdf = np.cumsum(p)
    for _ in range(shots):
        state = (state + 0x9E3779B97F4A7C15) & (2 ** 64 - 1)
        z = state
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & (2 ** 64 - 1)
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & (2 ** 64 - 1)
        z ^= z >> 31
        want.append(int(np.searchsorted(cdf, (z >> 11) * 2.0 ** -53 * cdf[-1], side="right")))
    assert np.array_equal(got.astype(np.int64), np.array(want))
