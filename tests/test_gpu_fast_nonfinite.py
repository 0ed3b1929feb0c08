"""Fast mode with angles that are infinite or NaN on gates that keep their exact
form (controlled ones), and amplitudes near the top of the range: what is NaN
and what stays finite is the oracle's."""
import math

import numpy as np
import pytest

import oracle
from spinoza_gb300 import _native as nat
from spinoza_gb300.circuit import QuantumCircuit
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu


def _ops(bad):
    """`bad`, controlled by qubit 1 (and 4), between rotations that mix what it touched."""
    rows = [((nat.RY, 0, 0, 0, (0.4, 0, 0)), 2, 0, 0, 0), ((nat.RX, 0, 0, 0, (1.1, 0, 0)), 3, 0, 0, 0), bad,
            ((nat.H, 0, 0, 0, (0, 0, 0)), 2, 0, 0, 0), ((nat.RY, 0, 0, 0, (0.9, 0, 0)), 3, 0, 0, 0),
            ((nat.H, 0, 0, 0, (0, 0, 0)), 0, 0, 0, 0)]
    ops = np.zeros(len(rows), dtype=nat.OP_DTYPE)
    for i, row in enumerate(rows):
        ops[i] = row
    return ops


def _bad(kind, angle):
    if kind == nat.P:  # two controls: a diagonal gate that is not pushed as a phase
        return ((kind, 0, 0, 0, (angle, 0, 0)), 2, nat.CONTROLS_ONES, 0b10010, 0)
    return ((kind, 0, 0, 0, (angle, 0.3, 0.2)), 2, nat.CONTROLS_SINGLE, 0b10, 0)


@pytest.mark.parametrize("state", ["normal", "zeros"])
@pytest.mark.parametrize("angle", [math.nan, math.inf])
@pytest.mark.parametrize("kind", [nat.RX, nat.RY, nat.RZ, nat.U, nat.P])
def test_nan_where_the_oracle_has_it(gpu, kind, angle, state):
    n = 13  # tiles of 10 qubits
    r = np.random.default_rng(5)
    re, im = r.standard_normal(1 << n), r.standard_normal(1 << n)
    if state == "zeros":  # all tiles but one
        re[1 << 10:], im[1 << 10:] = 0.0, 0.0
    ops = _ops(_bad(kind, angle))
    s = State.from_arrays(re, im)
    QuantumCircuit.from_state(s, fast=True).execute_ops(ops)
    got = s.to_numpy()
    oracle.execute(ops, re, im)
    if kind == nat.RZ:  # one control: pushed as phases, which reach every amplitude
        assert np.all(np.isnan(got[0][(np.arange(1 << n) & 2) != 0]) )
        return
    for g, w in zip(got, (re, im)):
        assert np.array_equal(np.isnan(g), np.isnan(w)) and not np.any(np.isinf(g))
        ok = ~np.isnan(w)
        assert np.max(np.abs(g[ok] - w[ok])) <= 6 * 8 * 2.0 ** -53 * np.max(np.abs(w[ok]))


def test_amplitudes_that_leave_the_range_are_not_finite(gpu):
    # 340 H on one qubit grow the amplitudes by 2^170 until the carried scale takes it back at the end
    n, count = 10, 340
    r = np.random.default_rng(6)
    re, im = r.standard_normal(1 << n) * 2.0 ** 870, r.standard_normal(1 << n) * 2.0 ** 870
    ops = np.zeros(count + 2, dtype=nat.OP_DTYPE)
    ops[:count] = ((nat.H, 0, 0, 0, (0, 0, 0)), 1, 0, 0, 0)
    ops[count] = ((nat.RY, 0, 0, 0, (0.7, 0, 0)), 2, nat.CONTROLS_SINGLE, 1, 0)
    ops[count + 1] = ((nat.RY, 0, 0, 0, (0.9, 0, 0)), 3, 0, 0, 0)
    s = State.from_arrays(re, im)
    QuantumCircuit.from_state(s, fast=True).execute_ops(ops)
    got = s.to_numpy()
    oracle.execute(ops, re, im)
    for g, w in zip(got, (re, im)):
        wrong = np.abs(g - w) > count * 8 * 2.0 ** -53 * np.max(np.abs(w))
        assert not np.any(wrong & np.isfinite(g))
