"""<X>, <Y>, <Z> of several targets in one call: the sizes at which the path
changes (one launch, a block per target, up to 13 qubits; tiles above), target
lists in any order, with repeats, and longer than the qubits."""
import numpy as np
import pytest

import oracle
from spinoza_gb300 import core, rng
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("obs", ["x", "y", "z"])
@pytest.mark.parametrize("n", [1, 2, 6, 13, 14, 15, 20])
def test_several_targets_match_the_oracle(gpu, n, obs):
    re, im = rng.normal_state(n, 40 + n)
    s = State.from_arrays(re, im)
    every = list(range(n))
    for targets in (every, every[::-1], [n - 1, 0, n - 1], every * (70 // n + 1)):
        got = core.xyz_expectation_value(obs, s, targets)
        want = oracle.xyz_expectation_value(obs, re, im, targets)
        # a sum of 2^n terms of total magnitude 1 in any order: 2^-53 times a few
        # partial sums deep, far under 1e-13
        np.testing.assert_allclose(got, want, atol=1e-13, rtol=0)
        assert got == core.xyz_expectation_value(obs, s, targets)  # fixed order: the same bits again
    assert core.xyz_expectation_value(obs, s, []) == []
