"""rng.uniform, one draw in plain integers, against the array path (host only)."""
import numpy as np
import pytest

from spinoza_gb300 import rng

TOP = (1 << 64) - 1


@pytest.mark.parametrize("seed", [0, 1, 3, 1 << 31, (1 << 63) - 1, 1 << 63, TOP - 1, TOP])
def test_one_draw_is_the_arrays_draw(seed):
    for index in (0, 1, 2, 1000, (1 << 32) - 1, 1 << 40, (1 << 63) - 1):
        assert rng.uniform(seed, index) == rng.uniforms(seed, 1, index)[0]
    draws = [rng.uniform(seed, i) for i in range(64)]
    assert np.array_equal(draws, rng.uniforms(seed, 64)) and all(type(u) is float and 0.0 <= u < 1.0 for u in draws)


@pytest.mark.parametrize("seed", [-1, TOP + 1])
def test_what_the_arrays_refuse_is_refused(seed):
    with pytest.raises(OverflowError):
        rng.uniforms(seed, 1)
    with pytest.raises(OverflowError):
        rng.uniform(seed, 0)
