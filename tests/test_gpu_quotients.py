"""The FP64 state's reciprocal and Exner factor on their own, over the ranges
they are used in, against extended precision.

crcp refines the hardware's approximation by one step of a third-order
iteration.  The approximation reads the upper word of its operand and fills the
upper word of its result, 20 mantissa bits each: two relative errors of 2^-20,
and as much again for the approximation itself.  What the step leaves is the
cube of that, 27 2^-60 or 0.22 roundings, beside the last rounding.  quot(a, b) =
a crcp(b) rounds once more.  exner(x) = x^(-2/7) takes one third-order step from the FP32
power: seven roundings of the residual count a seventh each, the last rounding
one, and the step's own remainder, 0.06 e^3 with a residual e below 6e-6 over
1e-6 <= x <= 1.3, is a tenth of a rounding."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from gdpy import build

pytestmark = pytest.mark.gpu

U = 2.0**-53
SOURCE = r"""
#include "gd_common.cuh"
namespace gd { long long g_launches = 0; }
__global__ void k(int what, const double* a, const double* b, double* y, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    double r;
    if (what == 0) asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(a[i]));
    else if (what == 1) r = gd::crcp(a[i]);
    else if (what == 2) r = gd::quot(a[i], b[i]);
    else r = gd::exner(a[i]);
    y[i] = r;
  }
}
extern "C" int run(int what, const double* a, const double* b, double* y, long n) {
  double *d[3];
  for (auto& p : d) if (cudaMalloc(&p, n * 8) != cudaSuccess) return 1;
  cudaMemcpy(d[0], a, n * 8, cudaMemcpyHostToDevice);
  cudaMemcpy(d[1], b, n * 8, cudaMemcpyHostToDevice);
  k<<<1024, 256>>>(what, d[0], d[1], d[2], n);
  int rc = cudaMemcpy(y, d[2], n * 8, cudaMemcpyDeviceToHost) != cudaSuccess;
  for (auto p : d) cudaFree(p);
  return rc;
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("quotients")
    src, so = str(d / "q.cu"), str(d / "q.so")
    open(src, "w").write(SOURCE)
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-shared", src, "-o", so], check=True)
    lib = ctypes.CDLL(so)

    def f(what, a, b=None):
        a = np.ascontiguousarray(a)
        b = a if b is None else np.ascontiguousarray(b)
        y = np.empty_like(a)
        p = [x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, y)]
        assert lib.run(what, *p, ctypes.c_long(a.size)) == 0
        return y

    return f


def mantissas():
    # every mantissa the approximation reads (its upper 20 bits), the bits below them all zero, all one, random
    rng = np.random.default_rng(0)
    top = np.arange(1 << 20, dtype=np.uint64) << np.uint64(32)
    low = [np.zeros(1 << 20, np.uint64), np.full(1 << 20, 0xffffffff, np.uint64),
           rng.integers(0, 1 << 32, 1 << 20, dtype=np.uint64)]
    return np.concatenate([(np.uint64(1023) << np.uint64(52) | top | l).view(np.float64) for l in low])


def worst(y, ref):
    assert np.all(np.isfinite(y))
    return float(np.max(np.abs((y.astype(np.longdouble) - ref) / ref)))


def test_reciprocal(run):
    x = mantissas()
    one = np.longdouble(1)
    assert worst(run(0, x), one / x) <= 3 * 2.0**-20
    for s in (1.0, -1.0, 2.0**-1000, 2.0**-300, 2.0**40, 2.0**1000):
        assert worst(run(1, s * x), one / (s * x).astype(np.longdouble)) <= 1.22 * U


def test_quotient(run):
    rng = np.random.default_rng(1)
    b = mantissas() * 2.0 ** rng.integers(-40, 40, 3 << 20)
    a = rng.standard_normal(3 << 20) * 10.0 ** rng.uniform(-12, 12, 3 << 20)
    assert worst(run(2, a, b), a.astype(np.longdouble) / b) <= 2.23 * U


def test_exner(run):
    rng = np.random.default_rng(2)
    x = np.concatenate([10.0 ** rng.uniform(-6, np.log10(1.3), 1 << 20), np.linspace(0.2, 1.1, 1 << 20)])
    ref = np.exp(-np.longdouble(2) / 7 * np.log(x.astype(np.longdouble)))
    assert worst(run(3, x), ref) <= 2.2 * U
