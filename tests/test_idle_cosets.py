"""The coset order of plans on the CPU: a program's coset bits are the bits
outside its tile, those that a pass before has held first, and a run from
|0...0> over the cosets of those bits alone equals the run over all of them."""
import numpy as np
import pytest

import kate_b200 as K
from kate_b200 import circuits
from common import random_circuit
from plan_emulator import PlanView, _deposit

CASES = [(13, "layered", 0), (16, "layered", 0), (15, "random", 0), (16, "random", 16), (16, "brickwork", 0),
         (15, "hea", 1), (16, "part", 0), (15, "brickwork", 4)]


def gates(n, what):
    if what == "layered":
        return circuits.layered(n, 2, seed=n)
    if what == "brickwork":
        return circuits.brickwork_su4(n, 3)
    if what == "hea":
        return circuits.hea(n, 3, seed=n)
    if what == "part":  # the last two qubits stay out
        return circuits.layered(n - 2, 2, seed=n)
    return random_circuit(n, 70, np.random.default_rng(n))


@pytest.mark.parametrize("n,what,flags", CASES)
def test_idle_cosets_are_zero(n, what, flags):
    pv = PlanView(K.Circuit(n, gates(n, what)), 12, 4, flags)
    progs = pv.block_programs if flags & 4 else pv.programs
    held, idles = set(), []
    for p, prog in zip(pv.passes, progs):
        tphys = [int(b) for b in p["tphys"]]
        out = [int(b) for b in prog["cphys"][: n - len(tphys)]]
        assert sorted(out + tphys) == list(range(n))
        idle = [b for b in out if b not in held]
        assert out[len(out) - len(idle):] == idle
        idles.append(len(idle))
        held |= set(tphys)
    if flags & 4:
        return
    st = np.zeros(1 << n, dtype=np.complex128)
    st[0] = 1.0
    want = pv.run(st)
    for p, prog, u in zip(pv.passes, progs, idles):
        m = p["m"]
        out = [int(b) for b in prog["cphys"][: n - m]]
        bases = _deposit(np.arange(1 << (n - m - u), dtype=np.int64), out)
        idx = bases[:, None] + _deposit(np.arange(1 << m, dtype=np.int64), p["tphys"])[None, :]
        tile = st[idx]
        for op in pv.ops[p["op0"]:p["op0"] + p["nops"]]:
            pv._apply(tile, bases, m, op)
        o = np.arange(1 << m, dtype=np.int64)
        src = np.zeros(1 << m, dtype=np.int64)
        for b in range(m):
            src |= ((o >> b) & 1) << int(p["outsrc"][b])
        st[idx] = tile[:, src]
    x = np.arange(1 << n, dtype=np.int64)
    got = st[_deposit(x, [pv.final_phys[pv.label_to_logical[b]] for b in range(n)])]
    assert np.array_equal(got, want)  # the same operations on the same amplitudes
