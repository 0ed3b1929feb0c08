"""States with zeros between ordinary amplitudes (real-valued ones, qubits still
in |0>): the reference's bits, signs of zeros among them, whichever way a warp
forms its products."""
import math

import numpy as np
import pytest

import oracle
from spinoza_gb300 import gates
from spinoza_gb300.circuit import Controls, QuantumCircuit
from spinoza_gb300.core import State
from spinoza_gb300.gates import Gate

pytestmark = pytest.mark.gpu


def _state(n, kind, seed):
    r = np.random.default_rng(seed)
    re, im = r.standard_normal(1 << n), r.standard_normal(1 << n)
    i = np.arange(1 << n)
    if "real" in kind:
        im[:] = 0.0
    if "imaginary" in kind:
        re[:] = -0.0
    if "empty" in kind:  # a qubit in |0>: neighbouring lanes, or groups of them
        hole = (i >> int(kind[-1])) & 1 == 1
        re[hole], im[hole] = 0.0, -0.0
    if "scattered" in kind:
        re[r.random(re.size) < 0.2] = 0.0
        im[r.random(im.size) < 0.2] = -0.0
    return re, im


def _same(a, b):
    return all(np.array_equal(x, y) and np.array_equal(np.signbit(x), np.signbit(y)) for x, y in zip(a, b))


@pytest.mark.parametrize("kind", ["real", "imaginary", "empty-0", "empty-1", "empty-4", "real, empty-1", "scattered"])
@pytest.mark.parametrize("n", [5, 9, 13])
def test_bits_match_the_oracle(gpu, kind, n):
    re, im = _state(n, kind, n)
    for j, th in enumerate((0.7, -2.9, math.pi, 0.0, 1e-160)):
        t, c = (3 * j) % n, (3 * j + 2) % n
        for g in (Gate.H, Gate.P(th), Gate.RX(th), Gate.RY(th), Gate.RZ(th), Gate.U(th, 0.4, 0.3)):
            for control in (None, c):
                ore, oim = re.copy(), im.copy()
                og = oracle.gate(g.kind, g.params)
                s, f = State.from_arrays(re, im), State.from_arrays(re, im)
                qc = QuantumCircuit.from_state(f)
                qc.x(0)
                qc.x(0)
                if control is None:
                    oracle.apply(og, ore, oim, t)
                    gates.apply(g, s, t)
                    qc._add(g, t)
                else:
                    oracle.c_apply(og, ore, oim, c, t)
                    gates.c_apply(g, s, c, t)
                    qc._add(g, t, Controls.single(c))
                assert _same(s.to_numpy(), (ore, oim)), (g, t, control)
                qc.execute()
                assert _same(f.to_numpy(), (ore, oim)), ("fused", g, t, control)

