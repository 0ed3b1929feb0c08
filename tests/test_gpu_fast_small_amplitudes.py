"""Fast mode holds every amplitude to the relative precision of 64-bit floating
point, small ones beside large ones too: rotations by tiny angles, products of
small amplitudes, states over many magnitudes."""
import math

import numpy as np
import pytest

import oracle
from spinoza_gb300 import _native as nat
from spinoza_gb300.circuit import QuantumCircuit
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu

EPS = 2.0 ** -53


def _ops(rows):
    ops = np.zeros(len(rows), dtype=nat.OP_DTYPE)
    for i, (kind, q, th) in enumerate(rows):
        ops[i] = ((kind, 0, 0, 0, tuple(th) + (0.0,) * (3 - len(th))), q, nat.CONTROLS_NONE, 0, 0)
    return ops


def _reach(rows, size):
    """|U| as a product of the gates' absolute values, as a function of |psi|: what an
    amplitude's rounding errors are measured by, gate by gate, in floating point."""
    def apply(mag):
        mag = mag.copy()
        for kind, q, th in rows:
            if kind in (nat.P, nat.RZ):
                continue
            c, s = (abs(math.cos(th[0] / 2)), abs(math.sin(th[0] / 2))) if kind != nat.H else (math.sqrt(0.5),) * 2
            v = mag.reshape(-1, 2, 1 << q)
            a, b = v[:, 0].copy(), v[:, 1].copy()
            v[:, 0], v[:, 1] = c * a + s * b, s * a + c * b
        return mag
    return apply


def _check(rows, re, im, per_gate=16.0):
    """Each gate within per_gate 2^-53 of the magnitudes that flow into an amplitude."""
    ops = _ops(rows)
    s = State.from_arrays(re, im)
    QuantumCircuit.from_state(s, fast=True).execute_ops(ops)
    got = s.to_numpy()
    ore, oim = re.copy(), im.copy()
    oracle.execute(ops, ore, oim)
    err = np.hypot(got[0] - ore, got[1] - oim)
    bound = per_gate * EPS * len(rows) * _reach(rows, re.size)(np.hypot(re, im))
    assert np.all(err <= bound), np.max(err / np.maximum(bound, 1e-300))


@pytest.mark.parametrize("theta", [0.0, 1e-12, 1e-8, 1e-4, 1e-2, 0.06, 0.063, 0.125, -1e-8, math.pi - 1e-8, math.pi + 1e-3])
@pytest.mark.parametrize("kind", [nat.RX, nat.RY, nat.U])
def test_one_rotation_by_a_small_angle(gpu, kind, theta):
    n = 11
    for q in (0, 4, 10):
        re, im = np.zeros(1 << n), np.zeros(1 << n)
        re[0], im[0] = 0.6, -0.8
        _check([(kind, q, (theta, 0.3, 0.4)), (nat.P, q, (0.7,))], re, im)


def test_a_large_neighbour_leaves_a_small_amplitude_alone(gpu):
    n = 10
    r = np.random.default_rng(1)
    re, im = r.standard_normal(1 << n), r.standard_normal(1 << n)
    re[1::2] *= 1e-9
    im[1::2] *= 1e-9
    for kind in (nat.RX, nat.RY):
        _check([(kind, 0, (0.0,)), (nat.RZ, 0, (0.3,)), (kind, 0, (1e-12,))], re, im)


@pytest.mark.parametrize("low, high", [(0.05, 0.3), (0.1, 1.0), (0.3, 1.5), (1e-6, 0.2)])
def test_products_of_small_amplitudes(gpu, low, high):
    n = 12
    r = np.random.default_rng(3)
    rows = [(nat.RY if r.random() < 0.5 else nat.RX, q, (float(r.choice([-1, 1]) * r.uniform(low, high)),)) for q in range(n)]
    re, im = np.zeros(1 << n), np.zeros(1 << n)
    re[0] = 1.0
    _check(rows, re, im)


@pytest.mark.parametrize("seed", range(8))
def test_states_over_many_magnitudes(gpu, seed):
    n = 11
    r = np.random.default_rng(seed)
    scale = 2.0 ** -r.integers(0, 60, 1 << n).astype(np.float64)
    re, im = r.standard_normal(1 << n) * scale, r.standard_normal(1 << n) * scale
    rows = []
    for _ in range(3):
        for q in r.permutation(n):
            kind = (nat.H, nat.RX, nat.RY, nat.P, nat.RZ)[int(r.integers(5))]
            th = float(r.uniform(-3, 3)) if r.random() < 0.7 else float(r.uniform(-1, 1) * 2.0 ** -r.integers(1, 40))
            rows.append((kind, int(q), (th,)))
    _check(rows, re, im)
