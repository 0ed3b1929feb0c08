"""X, CX and SWAP inside a pass move nothing (an index map follows them): long
mixes of them with controls inside and outside the tile, on 1 and on 0, with
gates of every other class between them, at the sizes where the launch shape
changes."""
import numpy as np
import pytest

import oracle
from spinoza_gb300 import _native as nat
from spinoza_gb300 import rng
from spinoza_gb300.circuit import Program, QuantumCircuit
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu


def _moves(n, count, seed, others):
    r = np.random.default_rng(seed)
    rows = []
    for _ in range(count):
        q = [int(v) for v in r.permutation(n)[:4]]
        kind, ctl, zeros, ck = nat.X, 0, 0, nat.CONTROLS_NONE
        pick = r.random()
        if pick < 0.2 and n > 1:
            rows.append(((nat.SWAP, q[0], q[1], 0, (0, 0, 0)), 0, 0, 0, 0))
            continue
        if others and pick < 0.5:
            kind = (nat.H, nat.RY, nat.Y, nat.Z, nat.P, nat.RZ, nat.U)[int(r.integers(7))]
        nc = min(n - 1, int(r.integers(0, 4)))
        if nc:
            ctl = sum(1 << c for c in q[1:1 + nc])
            zeros = sum(1 << c for c in q[1:1 + nc] if r.random() < 0.4)
            ck = nat.CONTROLS_MIXED
        rows.append(((kind, 0, 0, 0, tuple(r.uniform(-3, 3, 3))), q[0], ck, ctl, zeros))
    ops = np.zeros(len(rows), dtype=nat.OP_DTYPE)
    for i, row in enumerate(rows):
        ops[i] = row
    return ops


@pytest.mark.parametrize("others", [False, True])
@pytest.mark.parametrize("n", [1, 2, 3, 6, 10, 11, 13, 17, 18])
def test_moves_match_the_oracle(gpu, n, others):
    re, im = rng.normal_state(n, 60 + n)
    for seed in range(3):
        ops = _moves(n, 120, seed, others)
        ore, oim = re.copy(), im.copy()
        oracle.execute(ops, ore, oim)
        s = State.from_arrays(re, im)
        QuantumCircuit.from_state(s).execute_ops(ops)
        assert all(np.array_equal(a, b) for a, b in zip(s.to_numpy(), (ore, oim)))
        p = State.from_arrays(re, im)
        Program(n, ops).run(p)
        assert all(np.array_equal(a, b) for a, b in zip(p.to_numpy(), (ore, oim)))
        f = State.from_arrays(re, im)
        QuantumCircuit.from_state(f, fast=True).execute_ops(ops)
        assert max(float(np.max(np.abs(a - b))) for a, b in zip(f.to_numpy(), (ore, oim))) <= 1e-12
