"""Gate products formed on the integer pipes: the reference's bits for every
kind of amplitude and coefficient, in the plain kernels and in fused tiles."""
import math

import numpy as np
import pytest

import oracle
from spinoza_gb300 import gates
from spinoza_gb300.circuit import QuantumCircuit
from spinoza_gb300.core import State
from spinoza_gb300.gates import Gate

pytestmark = pytest.mark.gpu


def _amplitudes(n, kind, seed):
    """2^n doubles of one kind, as reals and imags."""
    r = np.random.default_rng(seed)
    size = 2 << n
    if kind == "any-bits":  # every exponent, subnormals, infinities and NaN among them
        v = r.integers(0, 1 << 64, size, dtype=np.uint64).view(np.float64)
    elif kind == "mixed":  # ordinary values with zeros, subnormals and extremes between them
        v = r.standard_normal(size)
        v[::7] = 0.0
        v[3::11] = -0.0
        v[5::13] = 5e-324 * r.integers(1, 1 << 20, v[5::13].size)
        v[1::17] = 1.7e308
        v[2::19] = 2.3e-308
        v[4::23] = math.inf
    else:  # few significant bits: products that end in exact halves
        v = (r.integers(1, 1 << 27, size) | 1) * 2.0 ** r.integers(-40, 5, size).astype(np.float64)
    v = v.astype(np.float64)
    return v[0::2].copy(), v[1::2].copy()


# angles whose sine or cosine is 0, 1, a power of two, tiny or ordinary
ANGLES = [0.0, math.pi, 2.0 * math.pi / 3.0, 1e-160, 1e-310, 0.7, -2.9, 2.0 * math.asin(2.0 ** -26)]


def _same(a, b):
    return all(np.array_equal(x, y, equal_nan=True) and
               np.array_equal(np.signbit(x[~np.isnan(x)]), np.signbit(y[~np.isnan(y)])) for x, y in zip(a, b))


@pytest.mark.parametrize("kind", ["any-bits", "mixed", "few-bits"])
@pytest.mark.parametrize("n", [1, 5, 11])
def test_products_plain_and_fused(gpu, kind, n):
    re, im = _amplitudes(n, kind, 100 + n)
    for j, th in enumerate(ANGLES):
        t = j % n
        for g in (Gate.H, Gate.P(th), Gate.RX(th), Gate.RY(th), Gate.RZ(th), Gate.U(th, 0.0, 0.3), Gate.U(1.1, th, th)):
            ore, oim = re.copy(), im.copy()
            with np.errstate(all="ignore"):
                oracle.apply(oracle.gate(g.kind, g.params), ore, oim, t)
            s = State.from_arrays(re, im)
            gates.apply(g, s, t)
            assert _same(s.to_numpy(), (ore, oim)), (kind, n, g, t)
            # the same gate inside a fused tile (a lone gate runs as a plain kernel: X X adds nothing)
            f = State.from_arrays(re, im)
            qc = QuantumCircuit.from_state(f)
            qc.x(0)
            qc.x(0)
            qc._add(g, t)
            qc.execute()
            assert qc.last_stats.tile_passes >= 1
            assert _same(f.to_numpy(), (ore, oim)), ("fused", kind, n, g, t)


def test_products_controlled(gpu):
    n = 6
    re, im = _amplitudes(n, "mixed", 5)
    for g in (Gate.H, Gate.P(0.4), Gate.RX(-0.8), Gate.RY(2.2), Gate.RZ(1.3), Gate.U(0.3, 0.9, -0.2)):
        for c, t in ((0, 3), (3, 0), (5, 1)):
            ore, oim = re.copy(), im.copy()
            with np.errstate(all="ignore"):
                oracle.c_apply(oracle.gate(g.kind, g.params), ore, oim, c, t)
            s = State.from_arrays(re, im)
            gates.c_apply(g, s, c, t)
            assert _same(s.to_numpy(), (ore, oim)), (g, c, t)
