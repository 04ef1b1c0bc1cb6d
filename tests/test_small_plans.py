"""Plans of simulators: every pass holds what the kernel that runs it needs.
Below 12 qubits one launch runs every pass's program or, when a pass has none,
the generic kernel runs the device ops of every pass."""
import numpy as np
import pytest

import kate_b200 as K
from common import random_circuit
from plan_emulator import PlanView

SIMULATOR, C64 = 32, 4


def diagonals_between_layers(n, diags):
    """An H on every qubit, `diags` diagonals of five qubits with generic
    phases (26 controlled phases each: eight of them are more than a program
    holds), then a pass and more of CNOTs and one-qubit gates."""
    rng = np.random.default_rng((n, diags))
    gates = [(2, [q], 0, None) for q in range(n)]
    for _ in range(diags):
        q = [int(x) for x in rng.choice(n, 5, replace=False)]
        gates.append((0, q, 0, np.diag(np.exp(1j * rng.uniform(0, 2 * np.pi, 32)))))
    return gates + random_circuit(n, 90, rng, kinds=("h", "cnot", "d1"))


@pytest.mark.parametrize("flags", [SIMULATOR, SIMULATOR | C64])
@pytest.mark.parametrize("n", [5, 6, 8, 10, 11, 12, 14])
@pytest.mark.parametrize("diags", [1, 9, 20])
def test_every_pass_has_what_its_kernel_runs(n, diags, flags, oracle):
    gates = diagonals_between_layers(n, diags)
    pv = PlanView(K.Circuit(n, gates), 12, 4, flags)
    has = [p is not None for p in (pv.block_programs if n >= 12 and flags & C64 else pv.programs)]
    if n >= 12:  # each pass on the kernel that takes it
        assert all(h or p["nops"] for h, p in zip(has, pv.passes))
        return
    assert all(has) or not any(has)
    assert all(has) or diags > 1
    assert not any(has) or diags < 20
    if not all(has):
        start = np.zeros(1 << n, dtype=np.complex128)
        start[0] = 1.0
        assert np.abs(pv.run(start) - oracle.simulate(n, gates)).max() <= 1e-12


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [K.C128, K.C64])
@pytest.mark.parametrize("n,diags", [(5, 9), (5, 20), (8, 20), (10, 20), (11, 20)])
def test_plans_with_passes_too_large_for_a_program(n, diags, prec, oracle):
    gates = diagonals_between_layers(n, diags)
    sim = K.Simulator(K.Circuit(n, gates), 1, prec, 0)
    assert len(sim.passes()) > 1 and set(sim.pass_kernels()) == {0}
    got = sim.execute()
    # Every gate is a sum of at most two products per amplitude (or one
    # phase): four roundings of 2^-24 a gate in the 2-norm in complex64.
    tol = 1e-12 if prec == K.C128 else 4 * len(gates) * 2.0**-24
    want = oracle.simulate(n, gates)
    assert np.abs(sim.state() - want).max() <= tol
    if prec == K.C128:
        assert np.abs(got.as_array() - oracle.measure(n, want)).max() <= 1e-9
    sim.profile_passes()
    assert np.abs(sim.state() - want).max() <= tol
