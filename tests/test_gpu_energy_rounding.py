"""An energy's diagonal part: rounding the terms' coefficients together must not
shift every amplitude's value alike."""
import numpy as np
import pytest

from spinoza_gb300 import core
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [14, 18])
def test_many_z_strings_on_equal_probabilities(gpu, n):
    r = np.random.default_rng(n)
    worst = 0.0
    for seed in range(6):
        # |+...+> up to signs: every Z string's value is exactly 0, whatever the coefficients
        re = np.full(1 << n, 2.0 ** (-n / 2)) * r.choice([-1.0, 1.0], 1 << n)
        c = r.standard_normal(40) * 3.0
        masks = [int(r.integers(1, 1 << n)) for _ in range(40)]
        got = core.pauli_expectation(State.from_arrays(re, np.zeros(1 << n)), core.pauli_terms(
            [(float(x), 0, m) for x, m in zip(c, masks)]))
        worst = max(worst, abs(got))
    # Per amplitude a value of about |c| = 20 with five roundings of 2^-53 of it, of
    # either sign and independent over the 2^n strings' values, and as many in the sum
    # over 2^n equal probabilities; a shift common to all would be 2^-53 20 by itself.
    assert worst <= 0.25 * 20 * 2.0 ** -53
