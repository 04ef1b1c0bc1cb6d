"""What this library is timed on: calls a user's program makes, as dicts of
plain values.

Kinds of case (``kind``):

* ``execute``  a Simulator kept by the program runs its circuit and measures
  (``Simulator.execute``), from |0...0> or from a product state;
* ``fresh``    the program has a new circuit each time, as in a variational
  loop: ``Simulator(circuit).execute()``;
* ``batch``    many independent circuits in one launch, <Z_q> of each;
* ``serve``    a burst of requests to the server, <Z_q> and samples of each;
* ``measure``  <Z_q> and seeded samples of a state that a Simulator holds.

Circuits are those of ``kate_b200.circuits``, with seeded angles.
"""
import ctypes
import math

import numpy as np
import torch

import kate_b200 as K
from kate_b200 import _lib, circuits


def listed():
    return [
        # The smallest calls: latency, launches and copies.
        {"name": "execute-n10", "kind": "execute", "family": "layered", "n": 10, "layers": 10, "prec": "c128",
         "start": "zero", "opt": False},
        # A variational loop's step on a small ansatz: every circuit is new.
        {"name": "fresh-hea-n16", "kind": "fresh", "family": "hea", "n": 16, "layers": 16, "prec": "c128",
         "start": "zero", "opt": False},
        # The 20-qubit layered circuit that a CPU can check.
        {"name": "execute-n20", "kind": "execute", "family": "layered", "n": 20, "layers": 10, "prec": "c128",
         "start": "zero", "opt": False},
        # A circuit that went through the compile passes (compileOPT): fused dense gates of up to 5 qubits.
        {"name": "execute-opt-n23", "kind": "execute", "family": "layered", "n": 23, "layers": 4, "prec": "c128",
         "start": "zero", "opt": True},
        # The reference's own benchmark circuit, from a product state.
        {"name": "execute-qulacs-n25", "kind": "execute", "family": "qulacs", "n": 25, "layers": 1, "prec": "c128",
         "start": "product", "opt": False},
        # Dense two-qubit gates in complex128.
        {"name": "execute-su4-n26", "kind": "execute", "family": "brickwork", "n": 26, "layers": 8, "prec": "c128",
         "start": "zero", "opt": False},
        # The full-size layered circuit: 30 qubits, 20 layers.
        {"name": "execute-n30", "kind": "execute", "family": "layered", "n": 30, "layers": 20, "prec": "c128",
         "start": "zero", "opt": False},
        # Complex64 on tensor cores: a small state and a large one.
        {"name": "execute-c64-n21", "kind": "execute", "family": "brickwork", "n": 21, "layers": 12, "prec": "c64",
         "start": "zero", "opt": False},
        {"name": "execute-c64-n30", "kind": "execute", "family": "brickwork", "n": 30, "layers": 20, "prec": "c64",
         "start": "zero", "opt": False},
        # A batch of ansatz circuits of mixed widths, tensor-core blocks on (what the autotuner picks for them).
        {"name": "batch-192", "kind": "batch", "count": 192, "lo": 10, "hi": 20, "blocks": True},
        # A burst of requests of mixed widths.
        {"name": "serve-48", "kind": "serve", "count": 48, "lo": 12, "hi": 21, "shots": 1024},
        # Measuring a state that the program holds.
        {"name": "measure-n26", "kind": "measure", "n": 26, "layers": 2, "prec": "c128", "shots": 1024},
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["execute"] * 5 + ["fresh", "batch", "serve", "measure"])
    if kind == "batch":
        lo = rng.randint(4, 14)
        return {"kind": kind, "count": logint(16, 192), "lo": lo, "hi": rng.randint(lo + 1, 20),
                "blocks": rng.random() < 0.5}
    if kind == "serve":
        return {"kind": kind, "count": logint(4, 48), "lo": 12, "hi": rng.randint(14, 21),
                "shots": logint(64, 2048)}
    if kind == "measure":
        return {"kind": kind, "n": rng.randint(9, 28), "layers": 2, "prec": "c128", "shots": logint(64, 4096)}
    if kind == "fresh":
        return {"kind": kind, "family": rng.choice(["hea", "layered"]), "n": rng.randint(5, 20),
                "layers": rng.randint(2, 16), "prec": "c128", "start": rng.choice(["zero", "product"]), "opt": False}
    prec = rng.choice(["c128", "c128", "c128", "c64"])
    if prec == "c64":
        return {"kind": kind, "family": rng.choice(["brickwork", "layered"]), "n": rng.randint(13, 29),
                "layers": logint(2, 12), "prec": prec, "start": "zero", "opt": False}
    family = rng.choice(["layered", "hea", "qulacs", "qft", "brickwork"])
    opt = family in ("layered", "hea") and rng.random() < 0.25
    return {"kind": kind, "family": family, "n": rng.randint(8, 23 if opt else 28),
            "layers": 1 if family in ("qulacs", "qft") else logint(2, 16), "prec": prec,
            "start": "product" if family in ("qulacs", "qft") else rng.choice(["zero", "product"]), "opt": opt}


# ---- circuits ----

def _gates(family, n, layers, seed):
    if family == "layered":
        return circuits.layered(n, layers, seed=seed)
    if family == "hea":
        return circuits.hea(n, layers, seed=seed)
    if family == "brickwork":
        return circuits.brickwork_su4(n, layers, seed=seed)
    return circuits.qulacs_bench(n) if family == "qulacs" else circuits.qft(n)


def _prec(case):
    return K.C64 if case["prec"] == "c64" else K.C128


def _input(case, seed):
    """The product state that the run starts from: (theta, phi) per qubit, or None for |0...0>."""
    if case["start"] == "zero":
        return None
    r = np.random.default_rng(seed + 17)
    n = case["n"]
    return np.stack([r.uniform(0.1, 0.9, n), r.uniform(0.0, 2.0 * math.pi, n)], axis=1)


def _widths(case, seed):
    """Widths of a batch's circuits (uniform) or of a server's requests (truncated geometric, p = 0.3). They
    depend on the case alone, so that every seed is the same amount of work."""
    r = np.random.default_rng(1000 + case["count"])
    if case["kind"] == "batch":
        return [int(x) for x in r.integers(case["lo"], case["hi"] + 1, case["count"])]
    out = []
    while len(out) < case["count"]:
        n = case["lo"] + int(r.geometric(0.3)) - 1
        if n <= case["hi"]:
            out.append(n)
    return out


def _many(case, seed):
    """The gates of each circuit of a batch or burst."""
    for i, n in enumerate(_widths(case, seed)):
        s = seed * 4096 + i
        yield n, (circuits.hea(n, 2 * n, seed=s) if case["kind"] == "batch" else circuits.layered(n, n, seed=s))


# ---- the calls ----

def prepare(case, seed):
    kind = case["kind"]
    if kind in ("execute", "fresh", "measure"):
        n = case["n"]
        c = K.Circuit(n, _gates(case.get("family", "layered"), n, case["layers"], seed))
        if kind == "measure":
            sim = K.Simulator(c, 1, _prec(case), 0)
            sim.execute()
            return {"kind": kind, "sim": sim, "shots": case["shots"], "seed": seed}
        if case["opt"]:
            c.compileOPT(5, 1e-6, min(n, 10))
        tp = _input(case, seed)
        start = False if tp is None else K.proba_state(tp)
        s = {"kind": kind, "start": start, "prec": _prec(case)}
        if kind == "fresh":
            s["circuit"] = c
        else:
            s["sim"] = K.Simulator(c, 1, _prec(case), 0)
        return s
    if kind == "batch":
        circs = []
        for i, n in enumerate(_widths(case, seed)):
            c = K.Circuit(n)
            c.appendFlat(*circuits.hea_flat(n, 2 * n, seed=seed * 4096 + i))
            circs.append(c)
        options = _lib.BatchOptions()
        _lib.lib().kate_batch_options_default(ctypes.byref(options))
        if case["blocks"]:
            for n in range(13, _lib.KATE_BATCH_MAX_QUBITS + 1):
                options.tune[n].blocks = 1
        return {"kind": kind, "batch": K.Batch(circs, precision=K.C64, options=options)}
    circs = [K.Circuit(n, g) for n, g in _many(case, seed)]
    srv = K.Server(K.C64, 0, budget_bytes=4 << 30, aux_bytes=1 << 30)
    return {"kind": kind, "server": srv, "circuits": circs, "shots": case["shots"], "seed": seed}


def run(state):
    kind = state["kind"]
    if kind in ("execute", "fresh"):
        sim = state["sim"] if kind == "execute" else K.Simulator(state["circuit"], 1, state["prec"], 0)
        tp = sim.execute(state["start"]).as_array()
        # The measurement of a complex64 state carries that type's precision.
        return tp.astype(np.float32) if state["prec"] == K.C64 else tp
    if kind == "measure":
        sim = state["sim"]
        return {"z": sim.expect_z(), "samples": sim.sample(state["shots"], seed=state["seed"]).astype(np.int64)}
    if kind == "batch":
        state["batch"].run()
        return state["batch"].expect_z_flat().astype(np.float32)
    srv = state["server"]
    ids = [srv.submit(c, state["shots"], state["seed"] + i) for i, c in enumerate(state["circuits"])]
    got = [srv.wait(i) for i in ids]
    return {"z": np.concatenate([g[0] for g in got]).astype(np.float32),
            "samples": np.concatenate([g[1] for g in got]).astype(np.int64)}


# ---- what a pass cannot do without ----

def _flops(gates):
    """Floating-point operations per amplitude: a dense k-qubit gate 8 * 2^k - 2, a diagonal or phase 6, H 6."""
    f = 0.0
    for gid, q, _, d in gates:
        if gid == K.DENSE:
            diag = not np.any(d - np.diag(np.diag(d)))
            f += 6.0 if diag else 8.0 * (1 << len(q)) - 2.0
        elif gid in (K.Hadamard, K.CRk):
            f += 6.0
    return f


def work(case):
    """The state written once and read once by the measurement; the circuit's gates. A held state is read once
    for <Z_q> and once for its samples."""
    kind = case["kind"]
    if kind == "measure":
        amps = 2.0 ** case["n"]
        return {"bytes": 2 * (16 if case["prec"] == "c128" else 8) * amps, "flops": 8 * amps}
    if kind in ("execute", "fresh"):
        amps = 2.0 ** case["n"]
        return {"bytes": 2 * (16 if case["prec"] == "c128" else 8) * amps,
                "flops": amps * _flops(_gates(case["family"], case["n"], case["layers"], 1))}
    b = f = 0.0
    for n in _widths(case, 1):
        gates = circuits.hea(n, 2 * n, seed=1) if kind == "batch" else circuits.layered(n, n, seed=1)
        b += 16 * 2.0 ** n
        f += 2.0 ** n * _flops(gates)
    return {"bytes": b, "flops": f}


# ---- the same results in complex128 by dense linear algebra and index permutations ----

_CHUNK = 1 << 25


class _State:
    """A state vector, bit q of the index for qubit q. Dense gates on
    neighbouring qubits are collected until one does not fit beside them,
    then applied five qubits at a time: a matrix product on the low qubits
    that moves them to the top, until all have come round."""

    def __init__(self, n, tp=None):
        self.n, self.pend = n, {}
        self.psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
        self.psi[0] = 1.0
        if tp is not None:
            for q in range(n):
                t, p = float(tp[q][0]) * math.pi / 2, float(tp[q][1])
                self.pend[q] = (1, np.array([[math.cos(t), 0], [np.exp(1j * p) * math.sin(t), 0]]))
            self.flush()

    def dense(self, q, m):
        w = len(q)
        assert list(q) == list(range(q[0], q[0] + w))
        old = self.pend.get(q[0])
        if old is not None and old[0] == w == 1:
            self.pend[q[0]] = (1, m @ old[1])
            return
        if any(a < q[0] + w and q[0] < a + b[0] for a, b in self.pend.items()):
            self.flush()
        self.pend[q[0]] = (w, m)

    def flush(self):
        if not self.pend:
            return
        q, first = 0, True
        while q < self.n:
            m, w = np.eye(1), 0
            while q + w < self.n:
                k, g = self.pend.get(q + w, (1, np.eye(2)))
                if w + k > 5:
                    break
                m, w = np.kron(g, m), w + k
            d = 1 << w
            t = torch.from_numpy(np.ascontiguousarray(m.astype(np.complex128))).cuda()
            self.psi = torch.matmul(t, self.psi.view(-1, d).T).view(-1)
            q += w
        self.pend = {}

    def _chunks(self):
        size = 1 << self.n
        for a in range(0, size, _CHUNK):
            yield a, torch.arange(a, min(size, a + _CHUNK), device="cuda")

    def permute(self, flips):
        """CNOTs and TOFFOLIs in order: (target, controls)."""
        self.flush()
        new = torch.empty_like(self.psi)
        for a, x in self._chunks():
            b = x.numel()
            for t, cs in reversed(flips):
                go = torch.ones_like(x)
                for c in cs:
                    go &= x >> c
                x = x ^ ((go & 1) << t)
            new[a:a + b] = self.psi[x]
        self.psi = new

    def phases(self, ps):
        """exp(i angle) where both qubits are 1: (a, b, angle)."""
        self.flush()
        for a, x in self._chunks():
            t = torch.zeros(x.numel(), dtype=torch.float64, device="cuda")
            for p, q, ang in ps:
                t += ((x >> p) & (x >> q) & 1).to(torch.float64) * ang
            self.psi[a:a + x.numel()] *= torch.polar(torch.ones_like(t), t)

    def circuit(self, gates):
        i = 0
        while i < len(gates):
            gid, q, k, d = gates[i]
            run = []
            while i < len(gates) and gates[i][0] in (K.CNOT, K.TOFFOLI):
                g = gates[i][1]
                run.append((g[0], g[1:]) if gates[i][0] == K.CNOT else (g[2], g[:2]))
                i += 1
            if run:
                self.permute(run)
                continue
            while i < len(gates) and (gates[i][0] == K.CRk or (gates[i][0] == K.DENSE and gates[i][3] is circuits.CZ)
                                      or (gates[i][0] == K.DENSE and len(gates[i][1]) == 2
                                          and np.array_equal(gates[i][3], circuits.CZ))):
                g = gates[i]
                run.append((g[1][0], g[1][1], 2 * math.pi / 2 ** g[2] if g[0] == K.CRk else math.pi))
                i += 1
            if run:
                self.phases(run)
                continue
            self.dense(q, d if gid == K.DENSE else np.array([[1, 1], [1, -1]]) * math.sqrt(0.5))
            i += 1
        self.flush()
        return self

    def sums(self, v):
        """Per qubit, the sum of v over the indices with its bit 0 and with its bit 1."""
        out = []
        for q in range(self.n):
            s = v.view(-1, 2, 1 << q).sum(dim=(0, 2))
            out.append((s[0].item(), s[1].item()))
        return out

    def expect_z(self):
        p = torch.empty(self.psi.numel(), dtype=torch.float64, device="cuda")
        for a in range(0, p.numel(), _CHUNK):
            c = self.psi[a:a + _CHUNK]
            p[a:a + _CHUNK] = c.real.square() + c.imag.square()
        return np.array([a - b for a, b in self.sums(p)])

    def proba(self):
        """(theta, phi) per qubit, as the reference measures them from the amplitudes' sums."""
        out = []
        for s0, s1 in self.sums(self.psi):
            s0, s1 = s0 / math.sqrt(2.0) ** self.n, s1 / math.sqrt(2.0) ** self.n
            if abs(s0) < 1e-13:
                out.append((1.0, 0.0))
            elif abs(s1) < 1e-14:
                out.append((0.0, 0.0))
            else:
                r = s1 / s0
                out.append((math.atan(abs(s1) / abs(s0)) / (math.pi / 2), math.atan(r.imag / r.real)))
        return np.array(out)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("execute", "fresh", "measure"):
        family = case.get("family", "layered")
        gates = _gates(family, case["n"], case["layers"], seed)
        s = _State(case["n"], None if kind == "measure" else _input(case, seed)).circuit(gates)
        return {"z": s.expect_z(), "samples": None} if kind == "measure" else s.proba()
    z = np.concatenate([_State(n).circuit(g).expect_z() for n, g in _many(case, seed)])
    return z if kind == "batch" else {"z": z, "samples": None}
