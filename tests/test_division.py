"""The division by a known divisor of the particle kernels (common.cuh:
divide_by): Markstein's correction of x * RN(1/h) with two fused
multiply-adds gives the correctly rounded quotient, so lattice coordinates
keep the bits of x / h.  Restated here with libm's fma over the magnitudes of
positions, chord extents and spline values, and for the divisors in use."""
import ctypes
import ctypes.util

import numpy as np
import pytest

fma = ctypes.CDLL(ctypes.util.find_library("m")).fma
fma.restype = ctypes.c_double
fma.argtypes = [ctypes.c_double] * 3


def divide_by(x, h):
    inv = 1.0 / h
    q = x * inv
    return fma(fma(-q, h, x), inv, q)


@pytest.mark.parametrize("h", [5e-6, 4e-6, 2e-6, 1e-6, 3.3333333333333335e-6, 2.0, 3.0, 4.0, 5.0,
                               1.9999999999999998])
def test_same_bits_as_the_division(h):
    rng = np.random.default_rng(int(h * 1e9) % 1000003)
    scale = h * 10.0 ** rng.uniform(-14, 5, 20000)
    for x in (scale * rng.standard_normal(scale.size)).tolist() + [0.0, h, -h, 7 * h, h / 3]:
        assert divide_by(x, h) == x / h


def test_non_finite_stays_non_finite():
    for x in (np.inf, -np.inf, np.nan):
        assert not np.isfinite(divide_by(x, 5e-6))
