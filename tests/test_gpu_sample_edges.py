"""Sampling at the sizes where its hierarchy changes (a sub-chunk of 32, a chunk
of 256, a super-chunk of 2^18 amplitudes) and at shot counts around a warp, on
dense and mostly empty states: outcomes equal the oracle's."""
import numpy as np
import pytest

import oracle
from spinoza_gb300 import core, rng
from spinoza_gb300.core import State

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 4, 5, 6, 8, 9, 13, 18, 19])
def test_outcomes_equal_the_oracle(gpu, n):
    re, im = rng.normal_state(n, 80 + n)
    for sparse in (False, True):
        if sparse:
            keep = np.random.default_rng(n).random(1 << n) < 0.02
            keep[(1 << n) - 1] = True
            re, im = re * keep, im * keep
        s = State.from_arrays(re, im)
        for shots in (1, 31, 33, 1000, 20001):
            u = rng.uniforms(n + shots, shots)
            u[0] = 0.0
            u[-1] = 1.0 - 2.0 ** -53
            assert np.array_equal(core.sample(s, u), oracle.sample(re, im, u)), (n, sparse, shots)
