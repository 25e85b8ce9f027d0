"""The FP64 quotient, root and comparisons of xg_fp64.cuh, called as they are from
a kernel compiled here.

Bounds, with u = 2^-53 (half a unit in the last place, relative): recip ends in
one rounding of x (1 + e + e^2), e below 2^-21 from the FP32 approximation (within
an FP32 ulp of an argument cut to 24 bits), exact up to e^3 < 2^-63: u (1 + 2^-9).
A quotient over(a, b) is a product with it: 2 u (1 + 2^-8).  xsqrt rounds s = x y
(half of that error is left by the correction) and its last sum: 3/2 u (1 +
2^-9).  Outside FP32's range, for zeros, infinities, NaN and (roots) negative
numbers they are CUDA's own IEEE division and root, bit for bit."""

import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from xyst_gb300 import build

pytestmark = pytest.mark.gpu

U = 2.0 ** -53

CODE = r"""
#include "xg_fp64.cuh"
using namespace xg;
__global__ void k(int n, const double* a, const double* b, double* o, int* t) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  o[i] = recip(a[i]);
  o[n + i] = xsqrt(a[i]);
  o[2 * n + i] = over(b[i], a[i], recip(a[i]));
  o[3 * n + i] = flip_if(a[i], i & 1);
  t[i] = less(a[i], b[i]) | less_neg(a[i], b[i]) << 1 | at_most(a[i], b[i]) << 2 |
         is_nan(a[i]) << 3 | (side(a[i], b[i]) + 1) << 4;
}
extern "C" int run(int n, const double* a, const double* b, double* o, int* t) {
  double *da, *db, *dout;
  int* dt;
  if (cudaMalloc(&da, n * 8) || cudaMalloc(&db, n * 8) || cudaMalloc(&dout, n * 32) ||
      cudaMalloc(&dt, n * 4))
    return 1;
  cudaMemcpy(da, a, n * 8, cudaMemcpyHostToDevice);
  cudaMemcpy(db, b, n * 8, cudaMemcpyHostToDevice);
  k<<<(n + 255) / 256, 256>>>(n, da, db, dout, dt);
  if (cudaGetLastError()) return 2;
  cudaMemcpy(o, dout, n * 32, cudaMemcpyDeviceToHost);
  cudaMemcpy(t, dt, n * 4, cudaMemcpyDeviceToHost);
  cudaFree(da), cudaFree(db), cudaFree(dout), cudaFree(dt);
  return int(cudaGetLastError());
}
"""


@pytest.fixture(scope="module")
def run(tmp_path_factory):
    d = tmp_path_factory.mktemp("fp64")
    (d / "h.cu").write_text(CODE)
    subprocess.run([build.nvcc()] + build.ARCH +
                   ["-O3", "-std=c++17", "-I" + build.CSRC, "-shared", "-Xcompiler", "-fPIC",
                    str(d / "h.cu"), "-o", str(d / "h.so"), "-cudart", "static"], check=True)
    lib = C.CDLL(os.path.join(d, "h.so"))

    def call(a, b):
        a, b = np.ascontiguousarray(a), np.ascontiguousarray(b)
        o, t = np.empty((4, a.size)), np.empty(a.size, np.int32)
        p = [x.ctypes.data_as(C.c_void_p) for x in (a, b, o, t)]
        assert lib.run(a.size, *p) == 0
        return o, t

    return call


def _numbers(rng, n, lo, hi):
    """Random signs and mantissas (some all ones, some zero) at exponents lo .. hi."""
    m = rng.uniform(1, 2, n)
    m[::17] = 1.0
    m[1::17] = 2.0 - 2.0 ** -52
    m[2::17] = 1.0 + 2.0 ** -52
    m[3::17] = 2.0 - 2.0 ** -23  # the last FP32 below a power of two
    return np.ldexp(m * rng.choice([-1, 1], n), rng.integers(lo, hi, n))


def _err(got, exact):
    return float(np.abs((got.astype(np.longdouble) - exact) / exact).max())


@pytest.mark.parametrize("lo,hi", [(-1, 2), (-120, 120), (-120, -117), (117, 120)])
def test_inside_fp32_range(run, lo, hi):
    assert np.finfo(np.longdouble).eps < 2.0 ** -62
    rng = np.random.default_rng(hi - lo)
    a, b = _numbers(rng, 400000, lo, hi), _numbers(rng, 400000, -100, 100)
    o, _ = run(a, b)
    al = a.astype(np.longdouble)
    assert _err(o[0], 1 / al) < U * (1 + 2.0 ** -9)
    assert _err(o[2], b / al) < 2 * U * (1 + 2.0 ** -8)
    pos = a > 0
    assert _err(o[1][pos], np.sqrt(al[pos])) < 1.5 * U * (1 + 2.0 ** -9)
    assert np.isnan(o[1][~pos]).all()


SPECIAL = np.array([0.0, -0.0, np.inf, -np.inf, np.nan, 5e-324, -5e-324, 2.2250738585072014e-308,
                    1.7976931348623157e308, -1.7976931348623157e308, 2.0 ** -120,
                    np.nextafter(2.0 ** -120, 0), 2.0 ** 120, np.nextafter(2.0 ** 120, 0), 1.0,
                    -1.0, 1e-9, -1e-9])


def _same(x, y):
    return np.all((x.view(np.int64) == y.view(np.int64)) | (np.isnan(x) & np.isnan(y)))


def test_outside_fp32_range(run):
    rng = np.random.default_rng(1)
    a = np.concatenate([SPECIAL, _numbers(rng, 50000, -1022, -120), _numbers(rng, 50000, 120, 1023),
                        rng.integers(1, 1 << 52, 5000).view(np.float64)])
    mag = np.abs(a)
    a = a[~((mag >= 2.0 ** -120) & (mag < 2.0 ** 120))]
    o, _ = run(a, a)
    with np.errstate(all="ignore"):
        assert _same(o[0], 1.0 / a) and _same(o[1], np.sqrt(a))


def test_comparisons(run):
    rng = np.random.default_rng(2)
    a = np.concatenate([np.repeat(SPECIAL, SPECIAL.size), rng.standard_normal(1000)])
    b = np.concatenate([np.tile(SPECIAL, SPECIAL.size), rng.standard_normal(1000)])
    b[-300:] = a[-300:]
    o, t = run(a, b)
    with np.errstate(all="ignore"):
        assert np.array_equal(t & 1, a < b)
        assert np.array_equal(t >> 1 & 1, a < -b)
        assert np.array_equal(t >> 2 & 1, a <= b)
        assert np.array_equal(t >> 3 & 1, np.isnan(a))
        ok = ~np.isnan(b)  # side's second argument is a number
        assert np.array_equal((t >> 4)[ok] - 1, np.where(a > b, 1, np.where(a < b, -1, 0))[ok])
    odd = np.arange(a.size) % 2 == 1
    assert _same(o[3], np.where(odd, -a, a))
