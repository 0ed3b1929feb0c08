"""Fast mode's fixed-point tiles: amplitudes over many magnitudes, zeros, values
that fixed point cannot hold (which take the FP64 path), every lazy kind with
either sign of its coefficient, and angles that are not finite."""
import math

import numpy as np
import pytest

import oracle
from spinoza_gb300 import _native as nat
from spinoza_gb300.circuit import QuantumCircuit
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu


def _state(n, kind, seed):
    r = np.random.default_rng(seed)
    re, im = r.standard_normal(1 << n), r.standard_normal(1 << n)
    if kind == "wide":  # magnitudes over 2^60 inside a tile
        s = 2.0 ** -r.integers(0, 60, 1 << n).astype(np.float64)
        return re * s, im * s
    if kind == "sparse":
        keep = r.random(1 << n) < 0.02
        return re * keep, im * keep
    if kind == "basis":
        re[:], im[:] = 0.0, 0.0
        re[(1 << n) // 3] = 1.0
        return re, im
    scale = {"tiny": 1e-290, "small": 1e-250, "huge": 1e280}.get(kind, 1.0)
    return re * scale, im * scale * 1e-3


def _circuit(n, seed):
    r = np.random.default_rng(seed)
    rows = []
    for layer in range(3):
        for q in range(n):
            kind = (nat.H, nat.RX, nat.RY, nat.U, nat.RZ, nat.P)[int(r.integers(6))]
            th = r.uniform(-7.0, 7.0, 3)
            if r.random() < 0.2:
                th[:] = (0.0, math.pi, -math.pi / 2, math.pi / 2)[int(r.integers(4))]
            rows.append(((kind, 0, 0, 0, tuple(th)), q, 0, 0, 0))
        for q in range(layer % 2, n - 1, 2):
            rows.append(((nat.X, 0, 0, 0, (0, 0, 0)), q + 1, nat.CONTROLS_SINGLE, 1 << q, 0))
        if n > 1:
            rows.append(((nat.RY, 0, 0, 0, (0.7, 0, 0)), 0, nat.CONTROLS_SINGLE, 1 << (n - 1), 0))
        rows.append(((nat.Y, 0, 0, 0, (0, 0, 0)), n // 2, 0, 0, 0))
        rows.append(((nat.SWAP, 0, n - 1, 0, (0, 0, 0)), 0, 0, 0, 0))
    ops = np.zeros(len(rows), dtype=nat.OP_DTYPE)
    for i, row in enumerate(rows):
        ops[i] = row
    return ops


def _fast(ops, re, im):
    s = State.from_arrays(re, im)
    QuantumCircuit.from_state(s, fast=True).execute_ops(ops)
    return s.to_numpy()


@pytest.mark.parametrize("kind", ["normal", "wide", "sparse", "basis", "tiny", "small", "huge"])
@pytest.mark.parametrize("n", [1, 2, 5, 10, 13])
def test_fixed_point_tiles_match_the_oracle(gpu, kind, n):
    re, im = _state(n, kind, 3 * n)
    ops = _circuit(n, n)
    got = _fast(ops, re, im)
    ore, oim = re.copy(), im.copy()
    oracle.execute(ops, ore, oim)
    # at most about 120 ops, each within a few 2^-53 of the state's norm
    top = np.abs(re).max() or 1.0  # the squares of "tiny" and "huge" leave the range
    tol = 1e-13 * math.hypot(np.linalg.norm(re / top), np.linalg.norm(im / top)) * top
    assert max(np.max(np.abs(got[0] - ore)), np.max(np.abs(got[1] - oim))) <= tol


def test_values_that_are_not_finite_stay_in_their_tile(gpu):
    n = 13
    re, im = _state(n, "normal", 9)
    ops = _circuit(10, 4)  # qubits 0-9: one tile per value of the upper three
    want = _fast(ops, re, im)
    re[5], im[(3 << 10) + 7] = math.inf, math.nan
    got = _fast(ops, re, im)
    for tile in range(8):
        part = slice(tile << 10, (tile + 1) << 10)
        for g, w in zip(got, want):
            if tile in (0, 3):
                assert not np.all(np.isfinite(g[part]))
            else:
                assert np.array_equal(g[part], w[part])


def test_angles_that_are_not_finite_give_nan(gpu):
    n = 6
    re, im = _state(n, "normal", 2)
    ops = _circuit(n, 1)
    ops[0] = ((nat.RY, 0, 0, 0, (math.nan, 0, 0)), 2, 0, 0, 0)
    got = _fast(ops, re, im)
    assert np.all(np.isnan(got[0])) and np.all(np.isnan(got[1]))
