"""The division by a known divisor of the particle kernels (common.cuh:
divide_by): Markstein's correction of x * RN(1/h) with two fused
multiply-adds gives the correctly rounded quotient, so lattice coordinates
keep the bits of x / h.  Restated here with libm's fma over the magnitudes of
positions, chord extents and spline values, and for the divisors in use; the
device's own function, in both precisions, is compared on the GPU."""
import ctypes
import ctypes.util

import numpy as np
import pytest

import checkers
import device_arithmetic
from aprl_b200 import native, workloads

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


@pytest.fixture(scope="module")
def device(tmp_path_factory):
    return device_arithmetic.load(tmp_path_factory.mktemp("device_arithmetic"))


@pytest.mark.gpu
@pytest.mark.parametrize("h", [1.0, 2.0, 3.0, 4.0, 5.0])
def test_device_binary32_over_the_splines_divisors(device, h):
    """Every significand; numpy's binary32 division is correctly rounded."""
    x = (np.arange(2**23, dtype=np.uint32) + 0x3f800000).view(np.float32)
    got = device_arithmetic.divide(device, x, np.full_like(x, h))
    np.testing.assert_array_equal(got, x / np.float32(h))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_device_division_near_the_midpoints(device, dtype):
    """Random divisors, and numerators one rounding from h times the midpoint
    between two neighbouring quotients, where a wrong last bit would show."""
    rng = np.random.default_rng(13)
    n = 1 << 20
    h = (1.0 + rng.random(n)).astype(dtype) * dtype(5e-6)
    q = (0.5 + 3.5 * rng.random(n)).astype(dtype)
    wide = np.longdouble if dtype is np.float64 else np.float64
    middle = (q.astype(wide) + np.nextafter(q, dtype(np.inf)).astype(wide)) / 2
    x = (middle * h.astype(wide)).astype(dtype)
    for v in (x, np.nextafter(x, dtype(np.inf)), np.nextafter(x, dtype(0)), -x,
              (x * (10.0 ** rng.uniform(-10, 5, n))).astype(dtype), q * h):
        np.testing.assert_array_equal(device_arithmetic.divide(device, v, h), v / h)


@pytest.mark.gpu
def test_device_division_of_non_finite_values(device):
    for dtype in (np.float32, np.float64):
        x = np.array([np.inf, -np.inf, np.nan, 0.0, -0.0], dtype=dtype)
        got = device_arithmetic.divide(device, x, np.full_like(x, 5e-6))
        assert not np.any(np.isfinite(got[:3]))
        np.testing.assert_array_equal(got[3:], x[3:])


@pytest.mark.gpu
def test_lattice_coordinates_use_the_divisors_of_the_run():
    """Uneven spacings: a chord's lattice coordinates come from this run's
    reciprocals, or the particles' own cells would be missed."""
    w = workloads.small_case(steps=2)
    cfg = w.config
    cfg.dx, cfg.dy = 4.7e-6, 5.3e-6
    cfg.reference_origin[0], cfg.reference_origin[1] = -8 * cfg.dx, -8 * cfg.dy
    g = native.Run(native.load(), w.config).load_workload(w)
    o = checkers.run(checkers.oracle(), w)
    for _ in range(2):
        g.step(1)
        o.step(1)
        for a in range(6):
            assert checkers.max_relative(g.get_field(a), o.get_field(a)) <= 1e-12, a
