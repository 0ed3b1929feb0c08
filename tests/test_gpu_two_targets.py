"""Expectation values of two and three targets about the sizes where the route changes."""
import numpy as np
import pytest

import oracle
from spinoza_gb300 import core, rng
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("targets", [(0, 1), (5, 2), (3, 3), (12, 0), (7, 11, 4)])
@pytest.mark.parametrize("n", [13, 14, 18])
def test_two_and_three_targets(gpu, n, targets):
    re, im = rng.normal_state(n, n)
    s = State.from_arrays(re, im)
    for obs in "xyz":
        got = core.xyz_expectation_value(obs, s, targets)
        # sums of at most 2^18 probabilities of a norm of 1
        np.testing.assert_allclose(got, oracle.xyz_expectation_value(obs, re, im, list(targets)), atol=1e-13, rtol=0)
        if obs == "z" and len(targets) == 2 and n > 13:
            assert got == [core.xyz_expectation_value("z", s, [t])[0] for t in targets]
