"""tests/cpp/device_arithmetic.cu, built with the library's flags and loaded."""
import ctypes as C
import os
import subprocess

import numpy as np

from aprl_b200 import build

SOURCE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp", "device_arithmetic.cu")


def load(directory):
    out = os.path.join(str(directory), "device_arithmetic.so")
    subprocess.check_call([build.nvcc(), "-shared", "-o", out, SOURCE] + build.flags())
    return C.CDLL(out)


def _ptr(a):
    return a.ctypes.data_as(C.c_void_p)


def divide(lib, x, h):
    f = lib.test_divide64 if x.dtype == np.float64 else lib.test_divide32
    x, h = np.ascontiguousarray(x), np.ascontiguousarray(h, dtype=x.dtype)
    out = np.empty_like(x)
    assert f(_ptr(x), _ptr(h), _ptr(out), C.c_longlong(x.size)) == 0
    return out


def fixed_add(lib, values, scale, merged):
    """Per value: whether it was accepted and its pair's value, an int."""
    v = np.ascontiguousarray(values, dtype=np.float64)
    pairs = np.empty((v.size, 2), dtype=np.uint64)
    accepted = np.empty(v.size, dtype=np.int32)
    assert lib.test_fixed_add(_ptr(v), C.c_longlong(v.size), C.c_double(scale), int(merged),
                              _ptr(pairs), _ptr(accepted)) == 0
    high = pairs[:, 1].astype(np.int64)
    return accepted != 0, [int(h) * 2**32 + int(l) for h, l in zip(high, pairs[:, 0])]
