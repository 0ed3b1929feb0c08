"""RZ in the backward sweeps: uncontrolled (goes back as P), controlled, with and
without a parameter, on tile qubits and above them."""
import math

import numpy as np
import pytest

import oracle
from spinoza_gb300 import _native as nat
from spinoza_gb300 import adjoint, batch, core
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu


def _problem(n, seed):
    r = np.random.default_rng(seed)
    rows, pidx = [], []
    for layer in range(2):
        for q in range(n):
            rows.append(((nat.RX, 0, 0, 0, (r.uniform(-3, 3), 0, 0)), q, nat.CONTROLS_NONE, 0, 0))
            if (q + layer) % 3:
                pidx.append(len(rows))
            rows.append(((nat.RZ, 0, 0, 0, (r.uniform(-6, 6), 0, 0)), q, nat.CONTROLS_NONE, 0, 0))
        for q in range(n - 1):
            rows.append(((nat.RZ, 0, 0, 0, (r.uniform(-3, 3), 0, 0)), q, nat.CONTROLS_SINGLE, 1 << (n - 1), 0))
            pidx.append(len(rows))
            rows.append(((nat.RY, 0, 0, 0, (r.uniform(-3, 3), 0, 0)), q, nat.CONTROLS_NONE, 0, 0))
    ops = np.zeros(len(rows), dtype=nat.OP_DTYPE)
    for i, row in enumerate(rows):
        ops[i] = row
    terms = core.ising_hamiltonian(r.standard_normal(n - 1), 1.0 + r.standard_normal(n))
    return ops, np.array(pidx, dtype=np.uint32), terms


def _energy(n, ops, pidx, theta, terms):
    re, im = oracle.zero_state(n)
    oracle.execute(adjoint.set_params(ops, pidx, theta), re, im)
    return oracle.pauli_expectation(re, im, terms)


@pytest.mark.parametrize("n", [1, 2, 6, 12])
def test_rz_gradients_match_parameter_shift(gpu, n):
    ops, pidx, terms = _problem(n, n)
    if n == 1:
        pidx = np.array([1, 3], dtype=np.uint32)  # both RZ
    theta = np.array([ops[int(k)]["gate"]["p"][0] for k in pidx])
    want = []
    for j in range(len(pidx)):
        step = np.zeros(len(pidx))
        step[j] = math.pi / 2
        want.append(0.5 * (_energy(n, ops, pidx, theta + step, terms) - _energy(n, ops, pidx, theta - step, terms)))
    # rounding of some 60 gates on a state of norm 1, times |H| < 100: below 1e-11
    _, g = adjoint.adjoint_gradient(State(n), ops, pidx, terms)
    np.testing.assert_allclose(g, want, atol=1e-11, rtol=0)
    for kw in ({}, {"tile_qubits": 4, "threads": 64}):
        e, grads = batch.Batch([(n, ops, pidx, theta, terms)], **kw).run()
        np.testing.assert_allclose(np.asarray(grads).ravel(), want, atol=1e-11, rtol=0)
