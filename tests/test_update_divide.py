"""The FP64 update's division by the spectral half-width (div_shared in
mw3_kernels.cu) on the CPU: one multiply and two FMAs with the rounded reciprocal
give the bits of the division, at the exponents that the kernel sends there."""
import ctypes
import ctypes.util

import numpy as np
import pytest

_fma = ctypes.CDLL(ctypes.util.find_library("m")).fma
_fma.restype = ctypes.c_double
_fma.argtypes = [ctypes.c_double] * 3


def _div_shared(a, b, z):
    hi = (int(np.float64(a).view(np.uint64)) >> 32) & 0x7FFFFFFF
    q = a * z
    if 200 << 20 <= hi < 1800 << 20:
        return _fma(_fma(-q, b, a), z, q)
    if a == 0.0:
        return q
    return a / b


_ONES = 1.0 + (1.0 - 2.0 ** -52)          # every mantissa bit set


@pytest.mark.parametrize("b", [1.0, 3.0, 0.1, 0.37419, 7.1e-3, _ONES, 2.0 ** -100, 2.0 ** 100 * (1 - 2.0 ** -53),
                               1.0 + 2.0 ** -52])
def test_division_bits(b):
    rng = np.random.default_rng(7)
    m = 1.0 + rng.integers(0, 2 ** 52, 4000) * 2.0 ** -52
    a = np.concatenate([m, -m * b, m * 2.0 ** rng.integers(-822, 776, 4000).astype(np.float64),
                        rng.integers(1, 2 ** 53, 2000) * b,
                        [0.0, -0.0, 5e-324, 2.0 ** -823, 2.0 ** -824, 2.0 ** 777, np.nextafter(2.0 ** 777, 0), _ONES]])
    z = 1.0 / b
    got = np.array([_div_shared(float(x), b, z) for x in a])
    assert np.array_equal(got.view(np.int64), (a / b).view(np.int64))
