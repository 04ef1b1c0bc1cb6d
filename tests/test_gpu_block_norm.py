"""A complex64 run's last tensor-core block pass sums ||psi||^2 of what it
stores: against a FP64 sum over the same amplitudes (profile_passes leaves the
state as the passes stored it, not rescaled). One CTA, one tile per group, several;
one pass from |0...0>, whose other cosets are zero, and many passes."""
import numpy as np
import pytest

import kate_b200 as K
from kate_b200 import circuits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("layers", [1, 5])
@pytest.mark.parametrize("n", [12, 13, 17, 22])
def test_norm_from_the_last_pass(n, layers):
    sim = K.Simulator(K.Circuit(n, circuits.brickwork_su4(n, layers)), 1, K.C64, 0)
    assert sim.pass_kernels()[-1] == 3
    assert sim.launches_per_run() == len(sim.pass_kernels()) + 1
    sim.execute()
    got = sim.norm2_before_renorm()
    scaled = sim.state()
    sim.profile_passes()
    assert sim.norm2_before_renorm() == got
    raw = sim.state().astype(np.complex128)
    want = float(np.sum(raw.real ** 2 + raw.imag ** 2))
    # FP64 sums of non-negative terms, at most 100 roundings of 2^-53 deep on either side.
    assert abs(got - want) <= 200 * 2.0 ** -53 * want
    # Each amplitude is the raw one times 1/||psi||, rounded once to FP32.
    ref = raw / np.sqrt(want)
    assert np.all(np.abs(scaled.real - ref.real) <= 2.0 ** -23 * np.abs(ref.real) + 1e-40)
    assert np.all(np.abs(scaled.imag - ref.imag) <= 2.0 ** -23 * np.abs(ref.imag) + 1e-40)
