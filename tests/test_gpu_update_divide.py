"""The FP64 update's division by a shared divisor (csrc/mw3_div.cuh) as compiled: the bits of the
division for every kind of dividend, and for divisors on both sides of the range it is made for."""
import ctypes as ct
import subprocess

import numpy as np
import pytest

from madwave3_gb300 import build

pytestmark = pytest.mark.gpu

SOURCE = r"""
#include "mw3_div.cuh"

__global__ void divide(const double *a, double *q, int n, double b, double z, bool ok)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) q[i] = mw3::div_shared(a[i], b, z, ok);
}

extern "C" int divide_all(const double *a, double *q, int n, double b)
{
    double *d = nullptr;
    if (cudaMalloc(&d, sizeof(double) * 2 * n) != cudaSuccess) return 1;
    cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
    divide<<<(n + 255) / 256, 256>>>(d, d + n, n, b, 1.0 / b, mw3::zdiv_ok(b));
    cudaMemcpy(q, d + n, sizeof(double) * n, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return cudaGetLastError();
}
"""


@pytest.fixture(scope="module")
def divide(tmp_path_factory):
    d = tmp_path_factory.mktemp("divide")
    src, lib = str(d / "divide.cu"), str(d / "libdivide.so")
    with open(src, "w") as f:
        f.write(SOURCE)
    subprocess.run([build._nvcc()] + build.ARCH + build.NVCC_FLAGS + ["-I" + build.CSRC, "-shared", "-o", lib, src], check=True)
    L = ct.CDLL(lib)
    L.divide_all.argtypes = [ct.c_void_p, ct.c_void_p, ct.c_int, ct.c_double]
    return L.divide_all


ONES = 1.0 + (1.0 - 2.0 ** -52)          # every mantissa bit set


@pytest.mark.parametrize("b", [1.0, 3.0, 0.1, 0.37419, 7.1e-3, ONES, 2.0 ** -100, 2.0 ** 100 * (1 - 2.0 ** -53), 1.0 + 2.0 ** -52,
                               np.nextafter(2.0 ** -100, 0), 2.0 ** 100, 3.0e-300, 1.7e300])
def test_division_bits(divide, b):
    rng = np.random.default_rng(11)
    m = 1.0 + rng.integers(0, 2 ** 52, 20000) * 2.0 ** -52
    with np.errstate(over="ignore", under="ignore"):
        a = np.concatenate([m, -m * b, m * 2.0 ** rng.integers(-1074, 1024, 20000).astype(np.float64),
                            rng.integers(1, 2 ** 53, 20000) * b,
                            [0.0, -0.0, 5e-324, -5e-324, 2.0 ** -823, 2.0 ** -824, 2.0 ** 777, np.nextafter(2.0 ** 777, 0), ONES,
                             np.inf, -np.inf, np.finfo(float).max, 2.0 ** -1022, np.nextafter(2.0 ** -1022, 0)]])
        want = a / b
    q = np.empty_like(a)
    assert divide(a.ctypes.data, q.ctypes.data, len(a), float(b)) == 0
    assert np.array_equal(q.view(np.int64), want.view(np.int64))
    nan = np.array([np.nan, -np.nan])
    assert divide(nan.ctypes.data, q.ctypes.data, 2, float(b)) == 0 and np.isnan(q[:2]).all()
