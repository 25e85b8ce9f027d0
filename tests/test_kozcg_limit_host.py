"""The limit coefficients of KozCG's FCT on rounding noise: the node pass's and
the element pass's own text on the CPU.  In the FP32 mode a node's extremes are
floats and its low-order solution a double, so at a node that is its own extreme
their difference is the float's rounding, of either sign; the coefficients are
shares of an allowed change (KozCG.cpp:1004-1024) and lie in [0, 1] all the same,
and an element's is the least of its nodes'."""

import ctypes as C

import numpy as np
import pytest

import host_kernel as hk

CODE = r"""
constexpr int kBlock = 256;
%s
template <class F>
void limit(int64_t n, const int32_t* aoff, const int32_t* aw, const int32_t* nbr, const F* ext,
           const double* R, const double* P, F* Q) {
  auto* K = new typename KozT<F>::Key[n * rec10<F>()]();
  for (int64_t i = 0; i < n; ++i)
    for (int k = 0; k < 10; ++k) K[i * rec10<F>() + k] = okey(ext[i * 10 + k]);
  blockDim.x = kBlock;
  for (int64_t i = 0; i < n; ++i) {
    blockIdx.x = unsigned(i / kBlock);
    threadIdx.x = unsigned(i %% kBlock);
    k_node_limit<F>(n, aoff, aw, nbr, K, R, P, Q);
  }
  delete[] K;
}
extern "C" void limit32(int64_t n, const int32_t* aoff, const int32_t* aw, const int32_t* nbr,
                        const float* ext, const double* R, const double* P, float* Q) {
  limit<float>(n, aoff, aw, nbr, ext, R, P, Q);
}
extern "C" void limit64(int64_t n, const int32_t* aoff, const int32_t* aw, const int32_t* nbr,
                        const double* ext, const double* R, const double* P, double* Q) {
  limit<double>(n, aoff, aw, nbr, ext, R, P, Q);
}
extern "C" int rec32() { return rec10<float>(); }
extern "C" void elem32(const int32_t* N, const float* Q, int sysmask, const float* aec, float* ca) {
  elem_limit<float>(N, Q, sysmask, reinterpret_cast<const float(*)[5]>(aec),
                    reinterpret_cast<float(*)[5]>(ca));
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    text = hk.source("xg_kozcg.cu")
    piece = hk.cut(text, "dkey", "dval", "KozT", "okey", "oval", "kC64", "rec10", "load10",
                   "store10", "quotients", "k_node_limit", "sbits", "lesser", "elem_limit")
    return hk.build(tmp_path_factory.mktemp("kozlim"), CODE % piece)


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


def _noise(dtype, n, seed):
    """A chain of n nodes whose low-order solution is uniform up to rounding, with
    antidiffusive sums of the size of rounding too; the extremes as node_low
    forms them (the low-order solution in the mode's precision)."""
    rng = np.random.default_rng(seed)
    base = rng.uniform(-2, 2, 5)
    R = base[:, None] * (1 + 1e-16 * rng.integers(-3, 4, (5, n)))
    P = np.empty((10, n))
    P[0::2] = 10.0 ** rng.uniform(-17, -7, (5, n))
    P[1::2] = -(10.0 ** rng.uniform(-17, -7, (5, n)))
    ext = np.repeat(R.T.astype(dtype), 2, axis=1)
    ns = (n + 31) // 32
    aoff = (np.arange(ns + 1) * 64).astype(np.int32)
    aw = np.full(ns, 2, np.int32)
    nbr = np.full(ns * 64, -1, np.int32)
    for i in range(n):
        o = aoff[i >> 5] + (i & 31)
        if i > 0:
            nbr[o] = i - 1
        if i + 1 < n:
            nbr[o + 32] = i + 1
    return aoff, aw, nbr, np.ascontiguousarray(ext), R, P


@pytest.mark.parametrize("seed", range(8))
@pytest.mark.parametrize("bits", [32, 64])
def test_coefficients_are_shares(lib, bits, seed):
    dtype = np.float32 if bits == 32 else np.float64
    n = 100
    aoff, aw, nbr, ext, R, P = _noise(dtype, n, seed)
    rec = lib.rec32() if bits == 32 else 10
    Q = np.full(n * rec, np.nan, dtype)
    getattr(lib, f"limit{bits}")(C.c_int64(n), _p(aoff), _p(aw), _p(nbr), _p(ext), _p(R), _p(P),
                                 _p(Q))
    Q = Q.reshape(n, rec)[:, :10]
    assert np.all(Q >= 0) and np.all(Q <= 1)


@pytest.mark.parametrize("sysmask", [0, 0b10011, 0b11111])
def test_element_takes_the_least(lib, sysmask):
    """An element's coefficient is the least of its nodes' for each component's
    sign (of all its components together where the system is limited)."""
    rng = np.random.default_rng(sysmask)
    rec = lib.rec32()
    for seed in range(8):
        n = 64
        aoff, aw, nbr, ext, R, P = _noise(np.float32, n, seed)
        Q = np.zeros(n * rec, np.float32)
        lib.limit32(C.c_int64(n), _p(aoff), _p(aw), _p(nbr), _p(ext), _p(R), _p(P), _p(Q))
        for _ in range(20):
            N = rng.choice(n, 4, replace=False).astype(np.int32)
            aec = rng.standard_normal((4, 5)).astype(np.float32)
            ca = np.zeros((4, 5), np.float32)
            lib.elem32(_p(N), _p(Q), C.c_int(sysmask), _p(aec), _p(ca))
            q = Q.reshape(n, rec)[N][:, :10].reshape(4, 5, 2)
            coef = np.minimum(1, np.where(aec > 0, q[..., 0], q[..., 1]).min(0))
            on = [c for c in range(5) if sysmask >> c & 1]
            if on:
                coef[on] = coef[on].min()
            assert np.array_equal(ca, coef.astype(np.float32) * aec)
