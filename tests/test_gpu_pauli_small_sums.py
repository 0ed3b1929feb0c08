"""Pauli sums that are small against the largest probability: every product and
partial sum keeps the relative precision of 64-bit floating point."""
import numpy as np
import pytest

from spinoza_gb300 import core
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu

# The products of a term are added in chains of at most 32 a thread and a tree of
# some 30 levels: 2^-53 each, of the sum of the magnitudes so far.
BOUND = 64 * 2.0 ** -53


def _sums(re, im, q, obs):
    """(2 sum Re or Im conj(psi_x) psi_y, the sum of its products' magnitudes) in extended precision."""
    v, w = (a.astype(np.longdouble).reshape(-1, 2, 1 << q) for a in (re, im))
    a, b, c, d = v[:, 0], w[:, 0], v[:, 1], w[:, 1]
    p = (a * c, b * d) if obs == "x" else (a * d, -b * c)
    return 2 * (p[0].sum() + p[1].sum()), 2 * (np.abs(p[0]).sum() + np.abs(p[1]).sum())


@pytest.mark.parametrize("obs", ["x", "y"])
@pytest.mark.parametrize("eps", [2.0 ** -6, 2.0 ** -12, 2.0 ** -18])
def test_a_qubit_almost_in_zero(gpu, eps, obs):
    n = 14  # the same amplitude for all others: what a product loses, every one loses
    re, im = np.full(1 << n, 0.9), np.full(1 << n, 0.7)
    re[1::2] = 1.2345 * eps
    im[1::2] = 0.4321 * eps
    got = core.xyz_expectation_value(obs, State.from_arrays(re, im), [0, 1])[0]
    want, weight = _sums(re, im, 0, obs)
    assert abs(got - want) <= BOUND * weight


@pytest.mark.parametrize("rest", [1e-4, 3e-6])
@pytest.mark.parametrize("n", [15, 18])
def test_a_few_large_amplitudes(gpu, n, rest):
    r = np.random.default_rng(n)
    re, im = (rest * r.uniform(0.5, 1.0, 1 << n) * r.choice([-1.0, 1.0], 1 << n) for _ in range(2))
    re[:: 1 << 11] = 1.0  # near a basis state, in every tile
    s = State.from_arrays(re, im)
    for obs in "xy":
        got = core.xyz_expectation_value(obs, s, range(n))
        for q in range(n):
            want, weight = _sums(re, im, q, obs)
            assert abs(got[q] - want) <= BOUND * weight
    b = r.standard_normal(n)
    got = core.pauli_expectation(s, core.pauli_terms([(b[q], 1 << q, 0) for q in range(n)]))
    sums = [_sums(re, im, q, "x") for q in range(n)]
    assert abs(got - sum(b[q] * sums[q][0] for q in range(n))) <= 2 * BOUND * sum(abs(b[q]) * sums[q][1] for q in range(n))
