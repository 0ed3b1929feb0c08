"""Pauli sums on the integer pipes: the sizes about the one that they start at,
tiles that fixed point cannot hold (which go the FP64 way in the same call), and
every form of term."""
import numpy as np
import pytest

import oracle
from spinoza_gb300 import core, rng
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu


def _state(n, form):
    re, im = rng.normal_state(n, 90 + n)
    if form == "zero tiles":
        re[: re.size // 2] = 0.0
        im[: re.size // 2] = 0.0
    elif form == "real":
        im[:] = 0.0
    elif form == "near basis":  # one large amplitude in some tiles
        re[:: 1 << 15] *= 1e9
    elif form == "wide":  # neighbours 2^30 apart
        re[1::2] *= 2.0 ** -30
        im[1::2] *= 2.0 ** -30
    elif form == "huge":
        re *= 2.0 ** 480
        im *= 2.0 ** 480
    elif form == "tiny":
        re *= 2.0 ** -490
        im *= 2.0 ** -490
    return re, im


def _terms(n, r):
    c = iter(r.standard_normal(400))
    bit = lambda *qs: sum(1 << q for q in qs)
    terms = [(next(c), 0, bit(i, i + 1)) for i in range(n - 1)]
    terms += [(next(c), bit(i), 0) for i in range(n)]                       # X
    terms += [(next(c), bit(i), bit(i)) for i in range(0, n, 3)]            # Y
    terms += [(next(c), bit(i), bit((i + 5) % n)) for i in range(0, n, 4)]  # XZ
    terms += [(next(c), bit(i), bit(i, (i + 1) % n)) for i in range(0, n, 5)]           # YZ
    terms += [(next(c), bit(0, n - 1), bit(0, n - 1)), (next(c), bit(2, 7, 9), bit(2, 7, 9))]  # YY, YYY
    terms += [(next(c), bit(1, 2, 3, 4), bit(1, 2, 3, 8)), (0.0, bit(3), 0)]
    return core.pauli_terms(terms)


@pytest.mark.parametrize("form", ["normal", "zero tiles", "real", "near basis", "wide", "huge", "tiny"])
@pytest.mark.parametrize("n", [19, 20, 21])
def test_sums_match_the_oracle(gpu, n, form):
    re, im = _state(n, form)
    s = State.from_arrays(re, im)
    norm = float(np.sum(np.square(re)) + np.sum(np.square(im)))
    terms = _terms(n, np.random.default_rng(n))
    weight = float(np.sum(np.abs(terms["coeff"])))
    # 2^-53 of the sum of the terms' magnitudes, a few partial sums deep on either
    # side (the oracle adds 2^20 products one after another: 2^-53 sqrt(2^20))
    tol = 1e-12 * norm * weight
    got = core.pauli_expectation(s, terms)
    assert abs(got - oracle.pauli_expectation(re, im, terms)) <= tol
    assert got == core.pauli_expectation(s, terms)  # fixed order: the same bits again
    for obs in "xy":
        got = core.xyz_expectation_value(obs, s, list(range(n)))
        want = oracle.xyz_expectation_value(obs, re, im, list(range(n)))
        np.testing.assert_allclose(got, want, atol=1e-12 * norm, rtol=0)


def test_small_components_keep_their_bits(gpu):
    """A qubit almost in |0>: its <X> is small against the tile's largest
    probability, and neither side of the range that fixed point takes loses it."""
    n = 20
    for eps in (2.0 ** -12, 2.0 ** -18, 2.0 ** -30):
        re, im = rng.normal_state(n, 7)
        re = 0.5 + np.abs(re) / np.abs(re).max()  # all of one sign: no cancellation
        im[:] = 0.0
        re[1::2] *= eps
        s = State.from_arrays(re, im)
        got = core.xyz_expectation_value("x", s, [0, 1])[0]
        want = 2.0 * float(np.sum(re[::2] * re[1::2]))
        # at 2^-18 a product's parts that fixed point leaves out are below 2^-36 of it,
        # of either sign, over 2^19 pairs: 2^-45; rounding a component: 2^-41 / 2^9
        assert abs(got - want) <= 2.0 ** -41 * want


def test_infinities_and_nan_still_reach_the_sum(gpu):
    n = 20
    for bad in (np.inf, np.nan):
        re, im = rng.normal_state(n, 3)
        re[12345] = bad
        s = State.from_arrays(re, im)
        assert not np.isfinite(core.pauli_expectation(s, core.pauli_terms([(1.0, 2, 0), (0.5, 0, 1)])))


@pytest.mark.parametrize("n", [12, 13, 20])
def test_strings_of_many_x_use_the_larger_tile(gpu, n):
    re, im = rng.normal_state(n, n)
    s = State.from_arrays(re, im)
    nine = sum(1 << q for q in range(n - 9, n))
    terms = core.pauli_terms([(0.7, nine, 0), (-0.4, nine, nine), (0.3, nine, 5), (0.2, 1, 0), (0.9, 0, 3)])
    # as above
    assert abs(core.pauli_expectation(s, terms) - oracle.pauli_expectation(re, im, terms)) <= 1e-12 * 2.5
