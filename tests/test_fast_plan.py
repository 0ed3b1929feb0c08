"""Fast mode's planner on circuits dense in controlled phases: it returns (host
only), and what it plans matches the oracle."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from spinoza_gb300 import _native as nat
from spinoza_gb300 import circuit

ROOT = Path(__file__).resolve().parent.parent


def _ops(rows):
    """Rows of (kind, target, control or None, angle) as an op array."""
    ops = np.zeros(len(rows), dtype=nat.OP_DTYPE)
    for i, (kind, t, c, angle) in enumerate(rows):
        ctl = (nat.CONTROLS_NONE, 0) if c is None else (nat.CONTROLS_SINGLE, 1 << c)
        ops[i] = ((kind, 0, 0, 0, (angle, 0.0, 0.0)), t, ctl[0], ctl[1], 0)
    return ops


def edges_then_h(pairs, hs):
    return _ops([(nat.P, t, c, 0.1 + 0.05 * i) for i, (c, t) in enumerate(pairs)] + [(nat.H, q, None, 0.0) for q in hs])


def phase_layers(n, seed):
    """H on every qubit, then twice: random CP / CZ / CX-RZ-CX edges and a layer of RX or H."""
    r = np.random.default_rng(seed)
    rows = [(nat.H, q, None, 0.0) for q in range(n)]
    density = r.uniform(0.1, 0.9)
    for _ in range(2):
        for a in range(n):
            for b in range(a + 1, n):
                if r.random() > density:
                    continue
                th, kind = float(r.uniform(0.1, 3.0)), int(r.integers(3))
                if kind == 0:
                    rows.append((nat.P, b, a, th))
                elif kind == 1:
                    rows.append((nat.Z, b, a, 0.0))
                else:
                    rows += [(nat.X, b, a, 0.0), (nat.RZ, b, None, th), (nat.X, b, a, 0.0)]
        last = nat.RX if r.random() < 0.5 else nat.H
        rows += [(last, q, None, 0.7) for q in range(n)]
    return _ops(rows)


def controlled_phase_mix(n, count, seed):
    """Random CP and, for three in ten, H."""
    r = np.random.default_rng(seed)
    rows = []
    for _ in range(count):
        t = int(r.integers(n))
        c = int((t + 1 + r.integers(n - 1)) % n)
        rows.append((nat.P, t, c, float(r.uniform(0.1, 3.0))) if r.random() < 0.7 else (nat.H, t, None, 0.0))
    return _ops(rows)


def circuits(which):
    if which == "two-tables":
        # qubits 0 and 1 with four phases each: their tables hold more masks
        # together than one op can, and either could go with a third qubit's
        yield 12, edges_then_h([(9, 0), (2, 0), (3, 0), (4, 0), (9, 1), (5, 1), (6, 1), (7, 1)], [0, 1, 9])
        yield 8, edges_then_h([(2, 0), (3, 0), (4, 0), (5, 0), (2, 1), (3, 1), (4, 1), (5, 1)], [0, 1, 2])
    elif which == "layers":
        for seed in range(150):
            yield 10 + seed % 11, phase_layers(10 + seed % 11, seed)
    else:
        for seed in range(200):
            yield 8 + seed % 9, controlled_phase_mix(8 + seed % 9, 60 + seed % 50, seed)


def plan_all(which):
    for n, ops in circuits(which):
        st = circuit.plan_stats(n, ops, fast=True)
        masks, device_ops = circuit.plan_passes(n, ops, fast=True)
        assert st["gates"] == len(ops) and len(masks) == len(device_ops) == st["passes"]
    print("planned")


@pytest.mark.parametrize("which", ["two-tables", "layers", "mix"])
def test_the_planner_returns(native, which):
    # in a child process: a planner that loops holds its thread for ever
    code = f"import sys; sys.path[:0] = ['.', 'tests']; import test_fast_plan; test_fast_plan.plan_all({which!r})"
    p = subprocess.run([sys.executable, "-c", code], cwd=ROOT, capture_output=True, text=True, timeout=240)
    assert p.returncode == 0 and p.stdout.strip() == "planned", p.stderr[-2000:]


@pytest.mark.gpu
@pytest.mark.parametrize("which", ["two-tables", "layers", "mix"])
def test_phase_dense_circuits_match_the_oracle(gpu, which):
    import oracle
    from spinoza_gb300 import rng
    from spinoza_gb300.circuit import QuantumCircuit
    from spinoza_gb300.core import State

    for i, (n, ops) in enumerate(circuits(which)):
        if n > 15 or i % 5 and which != "two-tables":
            continue
        re, im = rng.normal_state(n, i)
        s = State.from_arrays(re, im)
        QuantumCircuit.from_state(s, fast=True).execute_ops(ops)
        gre, gim = s.to_numpy()
        oracle.execute(ops, re, im)
        # a norm of 1, each gate within four 2^-53 of it (a phase: of its angle, 3 at most)
        atol = 4.0 * 3.0 * len(ops) * 2.0 ** -53
        np.testing.assert_allclose(gre, re, atol=atol, rtol=0)
        np.testing.assert_allclose(gim, im, atol=atol, rtol=0)
