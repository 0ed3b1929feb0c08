"""The work that users of spinoza_gb300 have it do, as cases that can be timed and checked.

Every case goes through the package's public entry points.  ``listed()`` names
the cases, ``draw(rng)`` gives one more of the same ranges, ``prepare`` makes
what a program has in hand before the call (inputs from the seed alone),
``run`` is one pass, ``work`` the bytes and operations a pass cannot do
without, and ``exact`` the same result from plain torch in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from spinoza_gb300 import _native as nat
from spinoza_gb300 import adjoint, batch, core, gates
from spinoza_gb300.circuit import Program, QuantumCircuit, QuantumRegister, execute_host
from spinoza_gb300.core import State
from spinoza_gb300.gates import Gate


def listed():
    return [
        # A small textbook circuit built gate by gate and executed, its state read back: what a
        # script or a notebook does; latency and launches count.
        {"name": "encode-8q", "kind": "encode", "n": 8, "value": 0.3},
        # Noise, mid-circuit measurements and gates conditioned on their outcomes.
        {"name": "measured-17q", "kind": "measured", "n": 17, "layers": 5, "measures": 4},
        # A circuit compiled once and replayed on new input states: the QFT of a 20-qubit state.
        {"name": "qft-20q", "kind": "qft", "n": 20, "fast": False},
        # A deep random circuit in the default (bit-exact) mode.
        {"name": "brickwork-26q", "kind": "brickwork", "n": 26, "layers": 10, "fast": False},
        # The same in the fast mode, at a size near a large user's.
        {"name": "brickwork-29q-fast", "kind": "brickwork", "n": 29, "layers": 10, "fast": True},
        # Gates applied one by one to every qubit (a user's own loop, the reference's benchmark).
        {"name": "gates-27q", "kind": "gates", "n": 27, "lazy": False},
        # The same loop in the lazy per-gate mode.
        {"name": "gates-29q-lazy", "kind": "gates", "n": 29, "lazy": True},
        # Measurement outcomes of a prepared state.
        {"name": "shots-27q", "kind": "shots", "n": 27, "shots": 1_000_000},
        # The energy of an Ising chain and every qubit's magnetisation.
        {"name": "ising-26q", "kind": "ising", "n": 26, "axis": "z"},
        # One training step of a variational circuit: energy and gradients through autograd.
        {"name": "gradient-21q", "kind": "gradient", "n": 21, "layers": 6, "fast": False},
        # Many small variational circuits at once.
        {"name": "batch-256", "kind": "batch", "count": 256, "qmin": 8, "qmax": 18, "dmin": 2, "dmax": 8},
        # A circuit on a state that the caller keeps in (page-locked) host memory.
        {"name": "host-25q", "kind": "host", "n": 25, "layers": 4, "fast": False},
    ]


def draw(rng):
    kind = rng.choice(["encode", "measured", "qft", "brickwork", "gates", "shots", "ising", "gradient", "batch", "host"])
    if kind == "encode":
        return {"kind": kind, "n": rng.randint(2, 14), "value": round(rng.random(), 6)}
    if kind == "measured":
        return {"kind": kind, "n": rng.randint(9, 22), "layers": rng.randint(2, 6), "measures": rng.randint(1, 6)}
    if kind == "qft":
        return {"kind": kind, "n": rng.randint(9, 25), "fast": rng.random() < 0.5}
    if kind == "brickwork":
        fast = rng.random() < 0.5
        return {"kind": kind, "n": rng.randint(13, 28 if fast else 27), "layers": rng.randint(2, 12), "fast": fast}
    if kind == "gates":
        lazy = rng.random() < 0.5
        return {"kind": kind, "n": rng.randint(5, 28 if lazy else 27), "lazy": lazy}
    if kind == "shots":
        return {"kind": kind, "n": rng.randint(4, 28), "shots": int(round(10.0 ** rng.uniform(2.0, 6.0)))}
    if kind == "ising":
        return {"kind": kind, "n": rng.randint(5, 27), "axis": rng.choice("xyz")}
    if kind == "gradient":
        return {"kind": kind, "n": rng.randint(6, 22), "layers": rng.randint(1, 8), "fast": rng.random() < 0.5}
    if kind == "batch":
        qmin = rng.randint(3, 12)
        return {"kind": kind, "count": int(round(2.0 ** rng.uniform(3.0, 8.0))), "qmin": qmin,
                "qmax": rng.randint(qmin, 18), "dmin": 1, "dmax": rng.randint(2, 9)}
    return {"kind": kind, "n": rng.randint(11, 26), "layers": rng.randint(1, 5), "fast": rng.random() < 0.5}


# ------------------------------------------------------------ circuits
# A gate here is (name, angles, target, controls); name "M" measures, "NOISE"
# flips with a probability.
def _encode_circuit(n, value, seed):
    """Value encoding: H on every qubit, a phase per qubit, the inverse QFT."""
    v = 2.0 ** n * ((value + np.random.default_rng(seed).random()) % 1.0)
    gs = [("H", (), q, ()) for q in range(n)]
    gs += [("P", (2.0 * math.pi * v / 2.0 ** (q + 1),), n - 1 - q, ()) for q in range(n)]
    return gs + _iqft(list(range(n))[::-1])


def _iqft(targets):
    gs = []
    for j in range(len(targets) - 1, -1, -1):
        gs.append(("H", (), targets[j], ()))
        gs += [("P", (-math.pi / 2.0 ** (j - k),), targets[k], (targets[j],)) for k in range(j - 1, -1, -1)]
    return gs


def _qft(n):
    gs = []
    for j in range(n - 1, -1, -1):
        gs.append(("H", (), j, ()))
        gs += [("P", (math.pi / 2.0 ** (j - k),), j, (k,)) for k in range(j - 1, -1, -1)]
    return gs + [("SWAP", (), (q, n - 1 - q), ()) for q in range(n // 2)]


def _brickwork(n, layers, seed):
    """U with uniform angles on every qubit, then CX on the even and the odd neighbours."""
    ang = np.random.default_rng(seed).uniform(0.0, 2.0 * math.pi, (layers, n, 3))
    gs = []
    for a in ang:
        gs += [("U", tuple(a[q]), q, ()) for q in range(n)]
        gs += [("X", (), q + 1, (q,)) for q in list(range(0, n - 1, 2)) + list(range(1, n - 1, 2))]
    return gs


def _measured_circuit(n, layers, measures, seed):
    """Rotation layers with CX and CRZ, a little bit-flip noise, then measurements whose outcomes control more gates."""
    r = np.random.default_rng(seed)
    gs = []
    for _ in range(layers):
        for q in range(n):
            gs.append((("RX", "RY", "RZ")[int(r.integers(3))], (float(r.uniform(-3.0, 3.0)),), q, ()))
        gs += [("X", (), q + 1, (q,)) for q in range(0, n - 1, 2)]
        gs += [("RZ", (float(r.uniform(-3.0, 3.0)),), q + 1, (q,)) for q in range(1, n - 1, 2)]
        gs += [("NOISE", (0.1,), q, ()) for q in range(0, n, 3)]
    for q in r.permutation(n)[:measures]:
        q = int(q)
        gs.append(("M", (), q, ()))
        gs.append(("RY", (float(r.uniform(-3.0, 3.0)),), (q + 1) % n, (q,)))
        gs.append(("H", (), q, ()))
    return gs


def _per_gate_loop(n, lazy, seed):
    r = np.random.default_rng(seed)
    gs = []
    for t in range(n):
        th = [float(x) for x in r.uniform(-3.0, 3.0, 6)]
        gs += [("H", (), t, ()), ("RX", (th[0],), t, ()), ("RZ", (th[1],), t, ())]
        if lazy:
            gs.append(("RY", (th[2],), t, ()))
        else:
            gs += [("U", tuple(th[3:]), t, ()), ("X", (), t, ((t + 1) % n,)), ("X", (), t, ((t + 1) % n, (t + 2) % n, (t + 3) % n))]
    return gs


_KIND = {"H": nat.H, "X": nat.X, "Z": nat.Z, "P": nat.P, "RX": nat.RX, "RY": nat.RY, "RZ": nat.RZ, "U": nat.U, "SWAP": nat.SWAP}


def _op_array(gs):
    ops = np.zeros(len(gs), dtype=nat.OP_DTYPE)
    for i, (name, ang, t, ctl) in enumerate(gs):
        p = tuple(ang) + (0.0,) * (3 - len(ang))
        q0, q1 = t if name == "SWAP" else (0, 0)
        kind = (nat.CONTROLS_NONE, nat.CONTROLS_SINGLE, nat.CONTROLS_ONES)[min(2, len(ctl))]
        ops[i] = ((_KIND[name], q0, q1, 0, p), 0 if name == "SWAP" else t, kind, sum(1 << c for c in ctl), 0)
    return ops


def _add(qc, gs):
    """The circuit through the builder's methods."""
    for name, ang, t, ctl in gs:
        if name == "M":
            qc.measure(t)
        elif name == "NOISE":
            qc.bit_flip_noise(ang[0], t)
        else:
            getattr(qc, ("c" if ctl else "") + name.lower())(*ang, *ctl, t)


def _gate(name, ang):
    return getattr(Gate, name)(*ang) if ang else getattr(Gate, name)


# ------------------------------------------------------------ inputs
def _random_state(n, seed):
    """reals and imags i.i.d. N(0,1), normalised, on the GPU."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    v = torch.randn(2, 1 << n, generator=g, dtype=torch.float64, device="cuda")
    v *= 1.0 / math.sqrt(float(torch.linalg.vector_norm(v)) ** 2)
    return v[0].contiguous(), v[1].contiguous()


def _zero_state(n):
    re = torch.zeros(1 << n, dtype=torch.float64, device="cuda")
    re[0] = 1.0
    return re, torch.zeros_like(re)


def _ising(n, seed):
    r = np.random.default_rng(seed)
    return r.standard_normal(n - 1), r.standard_normal(n)


def prepare(case, seed):
    kind, s = case["kind"], {"case": case, "seed": int(seed)}
    if kind == "encode":
        s["gates"] = _encode_circuit(case["n"], case["value"], seed)
    elif kind == "measured":
        s["gates"] = _measured_circuit(case["n"], case["layers"], case["measures"], seed)
        s["re"], s["im"] = _zero_state(case["n"])
        s["state"] = State.from_torch(s["re"], s["im"])
    elif kind == "qft":
        s["input"] = State.from_torch(*_random_state(case["n"], seed))
        s["re"], s["im"] = _zero_state(case["n"])
        s["state"] = State.from_torch(s["re"], s["im"])
        s["program"] = Program(case["n"], _op_array(_qft(case["n"])), fast=case["fast"])
    elif kind == "brickwork":
        s["ops"] = _op_array(_brickwork(case["n"], case["layers"], seed))
        s["re"], s["im"] = _zero_state(case["n"])
        s["state"] = State.from_torch(s["re"], s["im"])
    elif kind == "gates":
        s["gates"] = [(_gate(name, ang), t, ctl) for name, ang, t, ctl in _per_gate_loop(case["n"], case["lazy"], seed)]
        s["re"], s["im"] = _random_state(case["n"], seed)
        s["state"] = State.from_torch(s["re"], s["im"])
        s["state"].set_lazy(case["lazy"])
    elif kind == "shots":
        s["state"] = State.from_torch(*_random_state(case["n"], seed))
        s["u"] = np.random.default_rng(seed).random(case["shots"])
    elif kind == "ising":
        s["state"] = State.from_torch(*_random_state(case["n"], seed))
        s["terms"] = core.ising_hamiltonian(*_ising(case["n"], seed))
    elif kind == "gradient":
        s["ops"], s["params"] = adjoint.hardware_efficient_ansatz(case["n"], case["layers"])
        s["theta"] = torch.from_numpy(_angles(len(s["params"]), seed)).requires_grad_(True)
        s["terms"] = core.ising_hamiltonian(*_ising(case["n"], seed))
    elif kind == "batch":
        s["batch"] = batch.Batch([(n, *adjoint.hardware_efficient_ansatz(n, d), th, core.ising_hamiltonian(a, b))
                                  for n, d, th, a, b in _batch_instances(case, seed)])
    else:
        s["ops"] = _op_array(_brickwork(case["n"], case["layers"], seed))
        s["in"] = [_pinned(v) for v in _random_state(case["n"], seed)]
        s["out"] = [_pinned(torch.zeros(1 << case["n"], dtype=torch.float64)) for _ in range(2)]
        s["state"] = State(case["n"])
    return s


def _pinned(v):
    t = torch.empty(v.numel(), dtype=torch.float64, pin_memory=True)
    t.copy_(v)
    return t.numpy()


def _angles(count, seed):
    return np.random.default_rng(seed).uniform(-math.pi, math.pi, count)


def _batch_instances(case, seed):
    """(qubits, depth, angles, couplings, fields) of each instance: the sizes are the case's, the numbers the seed's."""
    shape, r = np.random.default_rng(8), np.random.default_rng(seed)
    for _ in range(case["count"]):
        n = int(shape.integers(case["qmin"], case["qmax"] + 1))
        d = int(shape.integers(case["dmin"], case["dmax"] + 1))
        yield n, d, r.uniform(-math.pi, math.pi, 2 * n * d), r.standard_normal(n - 1), r.standard_normal(n)


# ------------------------------------------------------------ one pass
def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "encode":
        qc = QuantumCircuit(QuantumRegister(case["n"]))
        _add(qc, s["gates"])
        qc.execute()
        return qc.get_statevector().to_numpy()
    if kind == "measured":
        gates.seed_noise(s["seed"] + 1)
        s["state"].reset_zero()
        qc = QuantumCircuit.from_state(s["state"], seed=s["seed"])
        _add(qc, s["gates"])
        qc.execute()
        values = [qc.qubit_tracker.get_qubit_measured_val(q) for q in range(case["n"])]
        return s["re"], s["im"], np.array([-1 if v is None else v for v in values])
    if kind == "qft":
        s["state"].copy_from(s["input"])
        s["program"].run(s["state"])
        return s["re"], s["im"]
    if kind == "brickwork":
        s["state"].reset_zero()
        QuantumCircuit.from_state(s["state"], fast=case["fast"]).execute_ops(s["ops"])
        return s["re"], s["im"]
    if kind == "gates":
        state = s["state"]
        for gate, t, ctl in s["gates"]:
            if not ctl:
                gates.apply(gate, state, t)
            elif len(ctl) == 1:
                gates.c_apply(gate, state, ctl[0], t)
            else:
                gates.mc_apply(gate, state, ctl, None, t)
        state.settle()
        return s["re"], s["im"]
    if kind == "shots":
        return core.sample(s["state"], s["u"]).view(np.int64)
    if kind == "ising":
        energy = core.pauli_expectation(s["state"], s["terms"])
        return np.array(energy), np.array(core.xyz_expectation_value(case["axis"], s["state"], range(case["n"])))
    if kind == "gradient":
        s["theta"].grad = None
        energy = adjoint.energy(s["theta"], case["n"], s["ops"], s["params"], s["terms"], fast=case["fast"])
        energy.backward()
        return energy, s["theta"].grad
    if kind == "batch":
        return s["batch"].run()
    execute_host(s["ops"], *s["in"], out=tuple(s["out"]), state=s["state"], fast=case["fast"])
    return s["out"]


# ------------------------------------------------------------ what a pass cannot do without
# Multiplies and adds of each gate per pair of amplitudes (an FMA counts two).
_FLOPS = {"H": 8, "RX": 12, "RY": 12, "U": 24, "P": 6, "RZ": 12, "X": 0, "Z": 0, "SWAP": 0, "NOISE": 0, "M": 4}


def _circuit_flops(n, gs):
    return float(sum((_FLOPS[name] << (n - 1)) >> (len(ctl) if name != "M" else 0) for name, _, _, ctl in gs))


def work(case):
    kind, n = case["kind"], case.get("n", 0)
    N = 1 << n
    if kind == "encode":
        return {"bytes": 16 * N, "flops": _circuit_flops(n, _encode_circuit(n, case["value"], 0))}
    if kind == "measured":
        return {"bytes": 16 * N, "flops": _circuit_flops(n, _measured_circuit(n, case["layers"], case["measures"], 0))}
    if kind == "qft":
        return {"bytes": 32 * N, "flops": _circuit_flops(n, _qft(n))}
    if kind == "brickwork":
        return {"bytes": 16 * N, "flops": _circuit_flops(n, _brickwork(n, case["layers"], 0))}
    if kind == "gates":  # each call reads and writes the amplitudes that its gate touches
        gs = _per_gate_loop(n, case["lazy"], 0)
        return {"bytes": sum((32 * N) >> len(ctl) for _, _, _, ctl in gs), "flops": _circuit_flops(n, gs)}
    if kind == "shots":
        return {"bytes": 16 * N + 16 * case["shots"], "flops": 4.0 * N}
    if kind == "ising":
        return {"bytes": 16 * N, "flops": 4.0 * N + 4.0 * N * n + 2.0 * N}
    if kind == "gradient":
        return {"bytes": 16 * N, "flops": _gradient_flops(n, case["layers"])}
    if kind == "batch":
        sizes = [(m, d) for m, d, _, _, _ in _batch_instances(case, 0)]
        return {"bytes": sum(32 * m * d for m, d in sizes), "flops": sum(_gradient_flops(m, d) for m, d in sizes)}
    return {"bytes": 32 * N, "flops": _circuit_flops(n, _brickwork(n, case["layers"], 0))}


def _gradient_flops(n, layers):
    """Forward once, the inverse on two states, a product per parameter."""
    return float(((12 + 12) * 3 + 8 + 8) * layers * n) * (1 << (n - 1))


# ------------------------------------------------------------ the same in plain torch, 64 bits
def _pick(psi, bits):
    """The amplitudes of psi whose qubits read `bits` ({qubit: 0 or 1}), as a view."""
    prev = psi.numel().bit_length() - 1
    shape, index = [], []
    for q in sorted(bits, reverse=True):
        shape += [1 << (prev - q - 1), 2]
        index += [slice(None), bits[q]]
        prev = q
    return psi.view(*shape, 1 << prev)[tuple(index)]


def _matrix(name, ang):
    if name == "H":
        r = math.sqrt(0.5)
        return r, r, r, -r
    if name == "P":
        return 1.0, 0.0, 0.0, complex(math.cos(ang[0]), math.sin(ang[0]))
    if name == "Z":
        return 1.0, 0.0, 0.0, -1.0
    c, s = math.cos(ang[0] / 2.0), math.sin(ang[0] / 2.0)
    if name == "RX":
        return c, -1j * s, -1j * s, c
    if name == "RY":
        return c, -s, s, c
    if name == "RZ":
        return complex(c, -s), 0.0, 0.0, complex(c, s)
    e = lambda a: complex(math.cos(a), math.sin(a))  # noqa: E731
    return c, -e(ang[2]) * s, e(ang[1]) * s, e(ang[1] + ang[2]) * c


def _apply(psi, name, ang, t, ctl=()):
    on = {c: 1 for c in ctl}
    if name == "SWAP":
        a, b = _pick(psi, {t[0]: 0, t[1]: 1}), _pick(psi, {t[0]: 1, t[1]: 0})
        keep = a.clone()
        a.copy_(b)
        b.copy_(keep)
        return
    a, b = _pick(psi, {**on, t: 0}), _pick(psi, {**on, t: 1})
    if name == "X":
        keep = a.clone()
        a.copy_(b)
        b.copy_(keep)
        return
    m00, m01, m10, m11 = _matrix(name, ang)
    if m01 == 0.0 and m10 == 0.0:
        if m00 != 1.0:
            a.mul_(m00)
        b.mul_(m11)
        return
    new = b * m01
    new.add_(a, alpha=m00)
    b.mul_(m11).add_(a, alpha=m10)
    a.copy_(new)


def _zero(n):
    psi = torch.zeros(1 << n, dtype=torch.complex128, device="cuda")
    psi[0] = 1.0
    return psi


def _parts(psi):
    return psi.real.contiguous(), psi.imag.contiguous()


def _uniform(seed, i):
    """Value i of the seeded counter stream that resolves noise and measurements (splitmix64)."""
    m = (1 << 64) - 1

    def mix(z):
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
        return z ^ (z >> 31)

    golden = 0x9E3779B97F4A7C15
    return (mix((mix((seed + golden) & m) + (i + 1) * golden) & m) >> 11) * 2.0 ** -53


def _energy(psi, a, b, lam=None):
    """Re<psi|H|psi> of H = sum a Z Z + b X, with lam = H psi left in `lam` when given."""
    n = psi.numel().bit_length() - 1
    d = torch.zeros(psi.numel(), dtype=torch.float64, device="cuda")
    for q in range(n - 1):
        for x in (0, 1):
            for y in (0, 1):
                _pick(d, {q: x, q + 1: y}).add_(float(a[q]) if x == y else -float(a[q]))
    out = psi * d if lam is None else torch.mul(psi, d, out=lam)
    for q in range(n):
        _pick(out, {q: 0}).add_(_pick(psi, {q: 1}), alpha=float(b[q]))
        _pick(out, {q: 1}).add_(_pick(psi, {q: 0}), alpha=float(b[q]))
    return (psi.real * out.real + psi.imag * out.imag).sum()


def _gradient(n, layers, theta, a, b):
    """Energy and gradient of the layered RY / RZ / CZ-ring ansatz: forward, then gates taken back on psi and H psi."""
    th = np.asarray(theta).reshape(layers, 2, n)
    pairs = [(i, (i + 1) % n) for i in range(n)] if n > 2 else [(0, 1)][: n - 1]
    psi = _zero(n)
    for layer in range(layers):
        for j, name in enumerate(("RY", "RZ")):
            for q in range(n):
                _apply(psi, name, (th[layer, j, q],), q)
        for c, t in pairs:
            _apply(psi, "Z", (), t, (c,))
    lam = torch.empty_like(psi)
    energy = _energy(psi, a, b, lam)
    grads = [[[None] * n, [None] * n] for _ in range(layers)]
    for layer in range(layers - 1, -1, -1):
        for c, t in pairs:
            _apply(psi, "Z", (), t, (c,))
            _apply(lam, "Z", (), t, (c,))
        for j, name in ((1, "RZ"), (0, "RY")):
            for q in range(n):
                p0, p1, l0, l1 = _pick(psi, {q: 0}), _pick(psi, {q: 1}), _pick(lam, {q: 0}), _pick(lam, {q: 1})
                if name == "RZ":  # Im<lam|Z|psi>
                    g = (l0.conj() * p0).imag.sum() - (l1.conj() * p1).imag.sum()
                else:  # Im<lam|Y|psi>
                    g = (l1.conj() * p0).real.sum() - (l0.conj() * p1).real.sum()
                grads[layer][j][q] = g
                _apply(psi, name, (-th[layer, j, q],), q)
                _apply(lam, name, (-th[layer, j, q],), q)
    flat = [g for per in grads for axis in per for g in axis]
    return energy, torch.stack(flat)


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "shots":
        return None
    if kind == "batch":
        got = [_gradient(m, d, th, a, b) for m, d, th, a, b in _batch_instances(case, seed)]
        return torch.stack([e for e, _ in got]).cpu(), torch.cat([g for _, g in got]).cpu()
    if kind == "gradient":
        energy, grad = _gradient(n, case["layers"], _angles(2 * n * case["layers"], seed), *_ising(n, seed))
        return energy.cpu(), grad.cpu()
    if kind in ("qft", "gates", "ising", "host"):
        psi = torch.complex(*_random_state(n, seed))
    else:
        psi = _zero(n)
    if kind == "ising":
        if case["axis"] == "z":
            p = psi.real ** 2 + psi.imag ** 2
            mags = [float(_pick(p, {q: 0}).sum() - _pick(p, {q: 1}).sum()) for q in range(n)]
        else:
            w = [(_pick(psi, {q: 0}).conj() * _pick(psi, {q: 1})).sum() for q in range(n)]
            mags = [2.0 * float(v.real if case["axis"] == "x" else v.imag) for v in w]
        return _energy(psi, *_ising(n, seed)), np.array(mags)
    gs = {"encode": lambda: _encode_circuit(n, case["value"], seed),
          "measured": lambda: _measured_circuit(n, case["layers"], case["measures"], seed),
          "qft": lambda: _qft(n),
          "gates": lambda: _per_gate_loop(n, case["lazy"], seed)}.get(kind, lambda: _brickwork(n, case.get("layers"), seed))()
    draws, flips, seen = 0, 0, {}
    for name, ang, t, ctl in gs:
        if name == "NOISE":
            if _uniform(seed + 1, flips) <= ang[0]:
                _apply(psi, "X", (), t)
            flips += 1
        elif name == "M":
            lo, hi = _pick(psi, {t: 0}), _pick(psi, {t: 1})
            p0 = float((lo.real ** 2 + lo.imag ** 2).sum())
            seen[t] = int(_uniform(seed, draws) < 1.0 - p0)
            draws += 1
            if seen[t]:
                lo.copy_(hi)
            lo.mul_(1.0 / math.sqrt(1.0 - p0 if seen[t] else p0))
            hi.zero_()
        elif len(ctl) == 1 and ctl[0] in seen:
            if seen[ctl[0]]:
                _apply(psi, name, ang, t)
        else:
            _apply(psi, name, ang, t, ctl)
    if kind == "measured":
        return (*_parts(psi), None)
    return _parts(psi)
