"""Gradients of circuits that touch few of the qubits: backward passes whose gates
need fewer qubits than a tile has."""
import math

import numpy as np
import pytest

import oracle
from spinoza_gb300 import _native as nat
from spinoza_gb300 import adjoint, core, rng
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fast", [False, True])
@pytest.mark.parametrize("n,qubits", [(5, [4]), (11, [5]), (12, [11, 6]), (13, [0]), (13, list(range(13)))])
def test_narrow_circuits(gpu, n, qubits, fast):
    ops = np.zeros(len(qubits), dtype=nat.OP_DTYPE)
    for i, q in enumerate(qubits):
        ops[i] = ((nat.RY if i % 2 else nat.RX, 0, 0, 0, (0.3 + i, 0, 0)), q, nat.CONTROLS_NONE, 0, 0)
    pidx = np.arange(len(qubits), dtype=np.uint32)
    re0, im0 = rng.normal_state(n, n)
    terms = core.pauli_terms([(0.5 + q, 1 << q, 0) for q in range(n)] + [(1.0, 0, 1 << q) for q in range(n)])

    def energy(k, shift):
        o = ops.copy()
        o["gate"]["p"][k, 0] += shift
        re, im = re0.copy(), im0.copy()
        oracle.execute(o, re, im)
        return oracle.pauli_expectation(re, im, terms)

    _, g = adjoint.adjoint_gradient(State.from_arrays(re0, im0), ops, pidx, terms, fast=fast)
    want = [0.5 * (energy(k, math.pi / 2) - energy(k, -math.pi / 2)) for k in range(len(qubits))]
    # a few gates on a state of norm 1, |H| < 120
    np.testing.assert_allclose(g, want, atol=1e-11, rtol=0)
