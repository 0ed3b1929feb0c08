"""Fast mode leaves zeros zero: imaginary parts of real-valued circuits, and
amplitudes that no gate reaches or that cancel exactly."""
import numpy as np
import pytest

import oracle
from spinoza_gb300 import _native as nat
from spinoza_gb300.circuit import QuantumCircuit
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu


def _fast(rows, n):
    ops = np.zeros(len(rows), dtype=nat.OP_DTYPE)
    for i, (kind, q, c, th) in enumerate(rows):
        ctl = (nat.CONTROLS_NONE, 0) if c is None else (nat.CONTROLS_SINGLE, 1 << c)
        ops[i] = ((kind, 0, 0, 0, (th, 0.0, 0.0)), q, ctl[0], ctl[1], 0)
    s = State(n)
    QuantumCircuit.from_state(s, fast=True).execute_ops(ops)
    want = oracle.zero_state(n)
    oracle.execute(ops, *want)
    return s.to_numpy(), want


@pytest.mark.parametrize("angles", [(0.3, 2.8), (1e-6, 0.06)])
@pytest.mark.parametrize("n", [4, 11, 13])
def test_real_circuits_stay_real(gpu, n, angles):
    r = np.random.default_rng(n)
    rows = []
    for _ in range(4):
        rows += [(nat.H if r.random() < 0.2 else nat.RY, q, None, float(r.choice([-1, 1]) * r.uniform(*angles))) for q in range(n)]
        rows += [(nat.X, q + 1, q, 0.0) for q in range(n - 1)]
    (re, im), (ore, oim) = _fast(rows, n)
    assert not np.any(oim) and not np.any(im)
    np.testing.assert_allclose(re, ore, atol=8 * len(rows) * 2.0 ** -53, rtol=0)


@pytest.mark.parametrize("n", [5, 12])
def test_amplitudes_that_nothing_reaches(gpu, n):
    rows = [(nat.RX, 2, None, 0.7), (nat.RY, 2, None, 1e-3)] + [(nat.X, q, 2, 0.0) for q in range(n) if q != 2]
    rows += [(nat.RY, 0, None, 0.4), (nat.RX, 0, None, 1e-9)]
    (re, im), (ore, oim) = _fast(rows, n)
    nothing = (ore == 0.0) & (oim == 0.0)
    assert nothing.sum() == (1 << n) - 4 and not np.any(re[nothing]) and not np.any(im[nothing])


@pytest.mark.parametrize("n", [4, 11])
def test_exact_cancellation(gpu, n):
    rows = [(nat.H, q, None, 0.0) for q in range(n)] * 2  # H H = 1: all but one amplitude cancel
    (re, im), _ = _fast(rows, n)
    assert not np.any(im) and not np.any(re[1:]) and abs(re[0] - 1.0) <= 2 * n * 2.0 ** -53
