"""A long run of equal RZ gates in the backward sweeps: the rounding of the
coefficients (the same for every amplitude, so it adds up) may scale both halves
alike, but not one of them alone."""
import math

import numpy as np
import pytest

from spinoza_gb300 import _native as nat
from spinoza_gb300 import adjoint, batch, core
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu

GATES = 2000


def _modulus_and_angle_error(x):
    c, s = np.longdouble(math.cos(x)), np.longdouble(math.sin(x))
    dc, ds = c - np.cos(np.longdouble(x)), s - np.sin(np.longdouble(x))
    return float(c * dc + s * ds), float(c * ds - s * dc)


def _angle():
    """An angle whose half has coefficients of modulus 1 and the right argument to
    2^-59, while its own have a modulus off by 2^-54 or more."""
    for k in range(400_000):
        theta = 0.3 + k * 1e-5
        half = _modulus_and_angle_error(theta / 2)
        if max(map(abs, half)) < 2.0 ** -59 and abs(_modulus_and_angle_error(theta)[0]) > 2.0 ** -53.9:
            return theta
    raise AssertionError("no such angle")


def test_both_halves_keep_their_weight(gpu):
    theta, a = _angle(), 0.1
    ops = np.zeros(GATES + 1, dtype=nat.OP_DTYPE)
    ops[0] = ((nat.RY, 0, 0, 0, (a, 0, 0)), 0, nat.CONTROLS_NONE, 0, 0)
    ops[1:] = ((nat.RZ, 0, 0, 0, (theta, 0, 0)), 0, nat.CONTROLS_NONE, 0, 0)
    pidx = np.array([0], dtype=np.uint32)
    turn = np.longdouble(theta) * GATES
    # <cos x X + sin x Y> with x the whole turn: its slope in a is cos a
    terms = core.pauli_terms([(float(np.cos(turn)), 1, 0), (float(np.sin(turn)), 1, 1)])
    # the coefficients' own errors, forward and back, and the roundings of 3 GATES
    # results of either sign (four standard deviations of at most 2^-53 / sqrt 3 each)
    tol = 4 * GATES * 2.0 ** -59 + 4 * math.sqrt(3 * GATES / 3) * 2.0 ** -53
    _, g = adjoint.adjoint_gradient(State(2), ops, pidx, terms)
    assert abs(g[0] - math.cos(a)) <= tol
    _, g = batch.Batch([(2, ops, pidx, np.array([a]), terms)]).run()
    assert abs(float(np.asarray(g).ravel()[0]) - math.cos(a)) <= tol
