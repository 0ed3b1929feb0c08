"""Fast mode's reordering of a pass for rotation pairs: rotations between gates
that commute with them and gates that do not."""
import numpy as np
import pytest

import oracle
from spinoza_gb300 import _native as nat
from spinoza_gb300 import rng
from spinoza_gb300.circuit import QuantumCircuit
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu


def _circuit(n, count, seed):
    r = np.random.default_rng(seed)
    ops = np.zeros(count, dtype=nat.OP_DTYPE)
    for i in range(count):
        th = tuple(r.uniform(-3.0, 3.0, 3))
        t = int(r.integers(n))
        c = 1 << int((t + 1 + r.integers(n - 1)) % n)
        kind, ctl = [(nat.H, 0), (nat.RX, 0), (nat.RY, 0), (nat.RY, 0), (nat.P, 0), (nat.RZ, 0), (nat.X, c), (nat.P, c),
                     (nat.RX, c), (nat.U, 0), (nat.Y, 0)][int(r.integers(11))]
        ops[i] = ((kind, 0, 0, 0, th), t, nat.CONTROLS_SINGLE if ctl else 0, ctl, 0)
    return ops


@pytest.mark.parametrize("n", [2, 3, 10, 11, 14])
def test_reordered_rotations_match_the_oracle(gpu, n):
    for seed in range(12):
        ops = _circuit(n, 90, 100 * n + seed)
        re, im = rng.normal_state(n, seed)
        s = State.from_arrays(re, im)
        QuantumCircuit.from_state(s, fast=True).execute_ops(ops)
        gre, gim = s.to_numpy()
        oracle.execute(ops, re, im)
        # 90 gates, each within a few 2^-53 of a norm of 1
        np.testing.assert_allclose(gre, re, atol=1e-13, rtol=0)
        np.testing.assert_allclose(gim, im, atol=1e-13, rtol=0)
