// KozCG on one GB300: element Taylor-Galerkin residual and flux-corrected
// transport, FP64, or with FP32 element arithmetic (XG_FP32_FLUX).
//
// Reference path (paths relative to the reference project root):
//   kozak::rhs      src/Physics/Kozak.cpp:29-180
//   KozCG::dt       src/Inciter/KozCG.cpp:613-688
//   KozCG::aec      src/Inciter/KozCG.cpp:772-843
//   KozCG::alw      src/Inciter/KozCG.cpp:865-948
//   KozCG::lim      src/Inciter/KozCG.cpp:978-1097
//   KozCG::solve    src/Inciter/KozCG.cpp:1119-1197
//   KozCG::BC       src/Inciter/KozCG.cpp:590-611 (Dirichlet and symmetry)
//
// Layout: node arrays SoA [ncomp][n] (U, R = rhs then low-order solution,
// P = antidiffusive sums +/- per component, A = limited contributions),
// elements as int32 [T][4].  Element kernels (one thread per tet) hand their
// four nodes' contributions on: in FP64 as plain stores into element-major
// slots that the node passes sum per node in ascending element order (the
// reference's order, the same bits on every run), in FP32 as vector atomic
// adds into node records.  The allowed limits Q+/- (extremes over
// the elements holding a node) are taken per node over the node adjacency,
// which holds the same nodes, and compared as order-preserving keys.  Node
// kernels (one thread per node) do the per-node algebra between the element
// passes.  One step is:
//   step_begin -> node_prim -> elem_rhs -> node_low -> node_limit -> elem_lim -> node_update
// node_low sums the element terms (FP64: from the slots), projects the
// boundary nodes' sums and forms the low-order solution; node_limit takes the
// allowed limits and the limit coefficients; node_update sums the limited
// terms, updates, applies the BCs and forms the CFL minimum for the next step.
// (FP32 zeroes its records first.)
//
// FP32-element mode: the element passes read an FP32 copy of the state (made
// by node_prim) and FP32 element geometry (made at setup), and add into FP32
// node records [n][16] / [n][8] with vector atomics; the allowed limits are
// 32-bit keys of floats.  The node passes (low-order solution, limit
// coefficients, update, dt) stay FP64 on the FP64 state.  GB300's FP64 rate
// is a small fraction of its FP32 rate, and FP32/FP64 conversions run at the
// FP64 rate, so this mode converts per node, not per element.

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <limits>
#include <vector>

#include "xg_fp64.cuh"
#include "xg_internal.hpp"
#include "xg_source.cuh"

namespace xg {

namespace {
constexpr int kBlock = 256;

struct KScalars {
  double dt;
  unsigned long long dtmin;
  int32_t blowup;
  int32_t pad;
  double t, tnext;  // the current step's start time, the next step's
};
}  // namespace

struct KozCGDev {
  Arena arena;
  Arena bcarena;
  int64_t n = 0, ne = 0;
  xg_kozcg_params prm{};
  int32_t* inpoel = nullptr;
  // FP32: per block of kFB elements its distinct nodes and their slots
  int32_t *bptr = nullptr, *bnode = nullptr;
  uint16_t* bstart = nullptr;
  uint8_t* bslot = nullptr;
  double *xyz = nullptr, *ivol = nullptr;  // coordinates, 1/vol
  double* cbrtv = nullptr;                 // cbrt(vol)
  double *U = nullptr, *R = nullptr, *P = nullptr, *A = nullptr;
  double* Q = nullptr;              // FP64 mode: limit coefficients C+/- [n][kC64]
  unsigned long long* K = nullptr;  // and the keys of each node's extremes [n][kC64]
  double* stage = nullptr;
  double* V = nullptr;  // node records of the element passes (see k_node_prim)
  // FP32-element mode: element sums, limit coefficients and 32-bit keys
  // [n][kC32]
  float *R32 = nullptr, *A32 = nullptr, *Q32 = nullptr;
  unsigned int* K32 = nullptr;
  // element geometry in the mode's precision (see k_geo)
  float* geo32 = nullptr;
  double* geo64 = nullptr;
  // FP64 mode: residual and limited slot records (10 and 6 doubles per
  // (element, local node) slot) and each node's slots in element order,
  // SELL-32 like the adjacency
  double *E = nullptr, *L = nullptr;
  int32_t *soff = nullptr, *sw = nullptr, *sslot = nullptr;
  // node adjacency (every pair of nodes sharing a tet) as SELL-32: slice s
  // of 32 nodes, entry k of node i at aoff[s] + 32 k + lane, -1 padding
  int64_t nslice = 0;
  int32_t *aoff = nullptr, *aw = nullptr, *anbr = nullptr;
  // BC program: one thread per BC node
  int64_t nbc = 0;
  int32_t *bcnode = nullptr, *bcdir = nullptr, *bcsymp = nullptr, *dirmask = nullptr;
  double *symn = nullptr, *dirval = nullptr;
  int32_t* bcof = nullptr;  // per node: its BC program entry or -1
  KScalars* scal = nullptr;
  double* dthist = nullptr;
  int64_t dthist_cap = 0;
  double t = 0.0;
  bool dt_valid = false;
  // manufactured source (kozak::rhs with problems::SRC): per step the
  // sources at the nodes at the step's start time S [5][n] and at the
  // element centroids half a step later Se [ne][5]
  SrcPrm src{};
  double *S = nullptr, *Se = nullptr;
};

void destroy_kozcg(KozCGDev* d) {
  if (!d) return;
  if (d->dthist) cudaFree(d->dthist);
  if (d->S) cudaFree(d->S);
  if (d->Se) cudaFree(d->Se);
  delete d;
}
size_t bytes_kozcg(const KozCGDev* d) { return d ? d->arena.bytes() + d->bcarena.bytes() : 0; }

namespace {

// order-preserving map of doubles to unsigned 64-bit keys
__device__ __forceinline__ unsigned long long dkey(double v) {
  unsigned long long b = __double_as_longlong(v);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ull);
}
__device__ __forceinline__ double dval(unsigned long long k) {
  unsigned long long b = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double(b);
}

__device__ __forceinline__ void block_min_atomic(double v, unsigned long long* dst) {
  __shared__ double red[32];
  unsigned long long bits = __double_as_longlong(v);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long other = __shfl_xor_sync(0xffffffffu, bits, o);
    bits = other < bits ? other : bits;
  }
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = __longlong_as_double(bits);
  __syncthreads();
  if (wid == 0) {
    int nw = (blockDim.x + 31) >> 5;
    double x = lane < nw ? red[lane] : DBL_MAX;
    unsigned long long b = __double_as_longlong(x);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long other = __shfl_xor_sync(0xffffffffu, b, o);
      b = other < b ? other : b;
    }
    if (lane == 0) atomicMin(dst, b);
  }
}

template <class F>
struct Geo {
  F J;
  F g[4][3];
};

// Element geometry (Kozak.cpp:76-89): coordinate differences in FP64, the
// cross products and Jacobian in F.
template <class F>
__device__ __forceinline__ Geo<F> tetgeo(const double* xyz, int64_t n, const int32_t N[4]) {
  const double* x = xyz;
  const double* y = xyz + n;
  const double* z = xyz + 2 * n;
  const F ba[3] = {F(x[N[1]] - x[N[0]]), F(y[N[1]] - y[N[0]]), F(z[N[1]] - z[N[0]])};
  const F ca[3] = {F(x[N[2]] - x[N[0]]), F(y[N[2]] - y[N[0]]), F(z[N[2]] - z[N[0]])};
  const F da[3] = {F(x[N[3]] - x[N[0]]), F(y[N[3]] - y[N[0]]), F(z[N[3]] - z[N[0]])};
  Geo<F> t;
  t.g[1][0] = ca[1] * da[2] - da[1] * ca[2];
  t.g[1][1] = ca[2] * da[0] - da[2] * ca[0];
  t.g[1][2] = ca[0] * da[1] - da[0] * ca[1];
  t.g[2][0] = da[1] * ba[2] - ba[1] * da[2];
  t.g[2][1] = da[2] * ba[0] - ba[2] * da[0];
  t.g[2][2] = da[0] * ba[1] - ba[0] * da[1];
  t.g[3][0] = ba[1] * ca[2] - ca[1] * ba[2];
  t.g[3][1] = ba[2] * ca[0] - ca[2] * ba[0];
  t.g[3][2] = ba[0] * ca[1] - ca[0] * ba[1];
  for (int i = 0; i < 3; ++i) t.g[0][i] = -t.g[1][i] - t.g[2][i] - t.g[3][i];
  t.J = ba[0] * t.g[1][0] + ba[1] * t.g[1][1] + ba[2] * t.g[1][2];
  return t;
}

// Types of a precision mode: F is the element arithmetic; FP64 mode sums in
// FP64 and keeps the allowed limits as 64-bit keys of doubles, the
// FP32-element mode sums in FP32 and keys floats in 32 bits.
template <class F>
struct KozT;
template <>
struct KozT<double> {
  using Key = unsigned long long;
};
template <>
struct KozT<float> {
  using Key = unsigned int;
};

__device__ __forceinline__ unsigned long long okey(double v) { return dkey(v); }
__device__ __forceinline__ unsigned int okey(float v) {
  const unsigned int b = __float_as_uint(v);
  return (b >> 31) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ double oval(unsigned long long k) { return dval(k); }
__device__ __forceinline__ float oval(unsigned int k) {
  return __uint_as_float((k >> 31) ? (k & 0x7fffffffu) : ~k);
}

// FP32 element sums are node records, so that a node's contribution is added
// with 16-byte vector atomics (red.global.add.v4.f32) instead of one atomic per
// component: R and P share a [n][16] record (R at 0..4, P+/- at 5..14), A has
// [n][8].
constexpr int kRP = 16;   // FP32 R+P record
constexpr int kAR = 8;    // FP32 A record
constexpr int kGB = 4;    // FP64 node gather: slots loaded together
// Records of ten values per node (extremes' keys, limit coefficients, + and -
// per component interleaved), padded to whole 16-byte accesses.
constexpr int kC64 = 10, kC32 = 12;
template <class T>
constexpr int rec10() {
  return sizeof(T) == 8 ? kC64 : kC32;
}
__device__ __forceinline__ void load10(const double* p, double o[10]) {
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const double2 t = __ldg(reinterpret_cast<const double2*>(p) + k);
    o[2 * k] = t.x;
    o[2 * k + 1] = t.y;
  }
}
__device__ __forceinline__ void load10(const unsigned long long* p, unsigned long long o[10]) {
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    const ulonglong2 t = __ldg(reinterpret_cast<const ulonglong2*>(p) + k);
    o[2 * k] = t.x;
    o[2 * k + 1] = t.y;
  }
}
__device__ __forceinline__ void load10(const unsigned int* p, unsigned int o[10]) {
  const uint4 a = __ldg(reinterpret_cast<const uint4*>(p));
  const uint4 b = __ldg(reinterpret_cast<const uint4*>(p) + 1);
  const uint2 c = __ldg(reinterpret_cast<const uint2*>(p + 8));
  o[0] = a.x, o[1] = a.y, o[2] = a.z, o[3] = a.w;
  o[4] = b.x, o[5] = b.y, o[6] = b.z, o[7] = b.w;
  o[8] = c.x, o[9] = c.y;
}
__device__ __forceinline__ void load10(const float* p, float o[10]) {
  unsigned int t[10];
  load10(reinterpret_cast<const unsigned int*>(p), t);
#pragma unroll
  for (int k = 0; k < 10; ++k) o[k] = __uint_as_float(t[k]);
}
template <class T>
__device__ __forceinline__ void store10(T* p, const T o[10]) {
  if constexpr (sizeof(T) == 8) {
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const longlong2 t = make_longlong2(reinterpret_cast<const long long*>(o)[2 * k],
                                         reinterpret_cast<const long long*>(o)[2 * k + 1]);
      reinterpret_cast<longlong2*>(p)[k] = t;
    }
  } else {
    const int* q = reinterpret_cast<const int*>(o);
    reinterpret_cast<int4*>(p)[0] = make_int4(q[0], q[1], q[2], q[3]);
    reinterpret_cast<int4*>(p)[1] = make_int4(q[4], q[5], q[6], q[7]);
    reinterpret_cast<int2*>(p + 8)[0] = make_int2(q[8], q[9]);
  }
}
// What the element passes read of a node, one record of eight values (density,
// momenta, total energy, pressure, 1/density, pad): 32 or 64 bytes in one or two
// accesses, where component arrays take a sector each.  The node-wise
// quotients kozak::rhs forms for every element holding the node
// (Kozak.cpp:93-118) are formed once.
template <class F>
__global__ void __launch_bounds__(kBlock) k_node_prim(int64_t n, const double* __restrict__ U,
                                                       double gamma_d, F* __restrict__ V) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const F gamma = F(gamma_d);
  F u[5];
#pragma unroll
  for (int c = 0; c < 5; ++c) u[c] = F(U[c * n + i]);
  const F ir = F(1.0) / u[0];
  const F p =
      (gamma - F(1.0)) * (u[4] - F(0.5) * (u[1] * u[1] + u[2] * u[2] + u[3] * u[3]) * ir);
  if constexpr (sizeof(F) == 8) {
    double2* o = reinterpret_cast<double2*>(V + i * 8);
    o[0] = make_double2(u[0], u[1]);
    o[1] = make_double2(u[2], u[3]);
    o[2] = make_double2(u[4], p);
    o[3] = make_double2(ir, 0.0);
  } else {
    float4* o = reinterpret_cast<float4*>(V + i * 8);
    o[0] = make_float4(u[0], u[1], u[2], u[3]);
    o[1] = make_float4(u[4], p, ir, 0.f);
  }
}
__device__ __forceinline__ void load_node(const float* V, int32_t i, float o[8]) {
  asm volatile("ld.global.nc.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=f"(o[0]), "=f"(o[1]), "=f"(o[2]), "=f"(o[3]), "=f"(o[4]), "=f"(o[5]),
                 "=f"(o[6]), "=f"(o[7])
               : "l"(V + int64_t(i) * 8));
}
__device__ __forceinline__ void load_node(const double* V, int32_t i, double o[8]) {
  const double* p = V + int64_t(i) * 8;
  asm volatile("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];"
               : "=d"(o[0]), "=d"(o[1]), "=d"(o[2]), "=d"(o[3])
               : "l"(p));
  asm volatile("ld.global.nc.v4.f64 {%0,%1,%2,%3}, [%4];"
               : "=d"(o[4]), "=d"(o[5]), "=d"(o[6]), "=d"(o[7])
               : "l"(p + 4));
}

// Element geometry in the mode's precision, formed once at setup from the
// FP64 coordinates: J/120, 1/(2J), g1, g2, g3 as [kGeo][T] (g0 = -g1 - g2 - g3
// is re-formed in the element passes).  In FP64 the 88 bytes a tet replace
// some 60 FP64 instructions a step (the cross products and two divisions),
// about 0.18 ms of arithmetic for 0.02 ms of memory traffic at 65^3.
constexpr int kGeo = 11;
template <class F>
__global__ void k_geo(int64_t n, int64_t ne, const int32_t* __restrict__ inpoel,
                      const double* __restrict__ xyz, F* __restrict__ geo) {
  const int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (e >= ne) return;
  int32_t N[4];
  for (int a = 0; a < 4; ++a) N[a] = inpoel[e * 4 + a];
  const Geo<double> t = tetgeo<double>(xyz, n, N);
  geo[e] = F(t.J / 120.0);
  geo[ne + e] = F(0.5 / t.J);
  for (int a = 1; a < 4; ++a)
    for (int j = 0; j < 3; ++j) geo[(2 + (a - 1) * 3 + j) * ne + e] = F(t.g[a][j]);
}

template <class F>
struct ElemGeo {
  F j120, ij2;  // J/120, 1/(2J)
  F g[4][3];
};
template <class F>
__device__ __forceinline__ ElemGeo<F> elem_geo(const F* __restrict__ geo, int64_t ne, int64_t e) {
  ElemGeo<F> t;
  t.j120 = __ldg(geo + e);
  t.ij2 = __ldg(geo + ne + e);
#pragma unroll
  for (int a = 1; a < 4; ++a)
#pragma unroll
    for (int j = 0; j < 3; ++j) t.g[a][j] = __ldg(geo + (2 + (a - 1) * 3 + j) * ne + e);
#pragma unroll
  for (int j = 0; j < 3; ++j) t.g[0][j] = -t.g[1][j] - t.g[2][j] - t.g[3][j];
  return t;
}

// KozCG::aec (KozCG.cpp:794-814) in FP32, k = ctau J/120: sum_b k (3 or -1)
// u_b, rounded term by term as the reference's sum.  The rounding it leaves in a
// nearly uniform component keeps the limiter's quotients bounded; formed as
// k (4 u_a - sum), exactly zero there, a run's differences from itself (the
// order of the atomics) grew from 6e-8 to 2e-6 of the state in 40 steps at 97^3.
template <class U>
__device__ __forceinline__ void aec32(float k, const U& u, float aec[4][5]) {
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      float s = 0.f;
#pragma unroll
      for (int b = 0; b < 4; ++b) s += (k * (a == b ? 3.f : -1.f)) * u[b][c];
      aec[a][c] = s;
    }
}

// kozak::rhs for one tet (Kozak.cpp:73-173): the residual r[a][c] of its
// four nodes, and with fct the antidiffusive element contributions of
// KozCG::aec (KozCG.cpp:794-814) aec[a][c], from the node records V.
//
// In FP64 the operation count is the bound (12.6 M tets of a 129^3 cube at 530
// G operations/s), so each flux is contracted with its gradient vector as
// F.g = (v.g) (rho, m, E + p) + p (0, g, 0), 12 operations a node where the
// sum over directions took 36; the fourth node's residual is minus the sum of
// the others (the gradients add to zero); and aec_a = ctau J/120 (4 u_a -
// sum_b u_b), which is exactly zero for a uniform component (FP32: aec32): about 190
// operations a tet for 480, k_elem_rhs64 1259 -> 548 us at 65^3, its FP64
// units busy throughout.
template <class F>
__device__ __forceinline__ void elem_terms(int64_t n, int64_t ne, int64_t e,
                                           const int32_t* __restrict__ inpoel,
                                           const F* __restrict__ geo, const F* __restrict__ V,
                                           const KScalars* __restrict__ sc, F gamma, F ctau,
                                           int fct, const double* __restrict__ S,
                                           const double* __restrict__ Se, int32_t N[4],
                                           F r[4][5], F aec[4][5]) {
  const int4 nd = __ldg(reinterpret_cast<const int4*>(inpoel) + e);
  N[0] = nd.x;
  N[1] = nd.y;
  N[2] = nd.z;
  N[3] = nd.w;
  const ElemGeo<F> t = elem_geo<F>(geo, ne, e);
  F u[4][5], sum[5], acc[5];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    F v[8];
    load_node(V, N[a], v);
#pragma unroll
    for (int c = 0; c < 5; ++c) u[a][c] = v[c];
    const F gv = (t.g[a][0] * v[1] + t.g[a][1] * v[2] + t.g[a][2] * v[3]) * v[6];
    const F h = v[4] + v[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      sum[c] = a == 0 ? u[a][c] : sum[c] + u[a][c];
      const F f = gv * (c == 4 ? h : u[a][c]);
      acc[c] = a == 0 ? f : acc[c] + f;
      if (c > 0 && c < 4) acc[c] += t.g[a][c - 1] * v[5];
    }
  }
  const F dt = F(sc->dt);
  const F coef = dt * t.ij2;
  F ue[5];
#pragma unroll
  for (int c = 0; c < 5; ++c) ue[c] = F(0.25) * sum[c] - coef * acc[c];
  if (S) {  // the nodes' sources at the step's start time, dt/8 each
    const F c8 = dt / F(8.0);
    for (int a = 0; a < 4; ++a)
      for (int c = 0; c < 5; ++c) ue[c] += c8 * F(__ldg(S + c * n + N[a]));
  }
  const F ir = F(1.0) / ue[0];
  const F vx = ue[1] * ir, vy = ue[2] * ir, vz = ue[3] * ir;
  const F pr = (gamma - F(1.0)) * (ue[4] - F(0.5) * (ue[1] * vx + ue[2] * vy + ue[3] * vz));
  ue[4] += pr;
  const F p6 = pr * (F(1.0) / F(6.0));
#pragma unroll
  for (int c = 0; c < 5; ++c) ue[c] *= F(1.0) / F(6.0);
#pragma unroll
  for (int a = 1; a < 4; ++a) {
    const F gv = t.g[a][0] * vx + t.g[a][1] * vy + t.g[a][2] * vz;
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      r[a][c] = gv * ue[c];
      if (c > 0 && c < 4) r[a][c] += t.g[a][c - 1] * p6;
    }
  }
#pragma unroll
  for (int c = 0; c < 5; ++c) r[0][c] = -r[1][c] - r[2][c] - r[3][c];
  if (Se) {  // the centroid's source half a step later, J/24 to each node
    const F cj = F(5.0) * t.j120;
    for (int c = 0; c < 5; ++c) {
      const F se = cj * F(__ldg(Se + e * 5 + c));
      for (int a = 0; a < 4; ++a) r[a][c] += se;
    }
  }
  if (fct) {
    const F k = ctau * t.j120;
    if constexpr (sizeof(F) == 8) {
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = 0; c < 5; ++c) aec[a][c] = k * (F(4.0) * u[a][c] - sum[c]);
    } else {
      aec32(k, u, aec);
    }
  } else {
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 5; ++c) aec[a][c] = F(0.0);
  }
}

// The FP32 residual pass is made of blocks of kFB elements (a slot 4 e + a of a
// block fits a byte).  Atomics would bound it (about 200 G of 16 bytes a second:
// 396 us at 97^3 with four nodes of four each an element).  Consecutive elements
// share nodes (those of 64 hold 50 distinct ones of 256 with locality
// numbering, 71 numbered at random), so a block adds its elements' contributions
// per distinct node in shared memory (lists made once per mesh) and hands one
// record a node to the atomics: 262 us, with 14 blocks an SM (12: 287).  The
// limiting pass, with two atomics a node, gains nothing so (227 against 223).
constexpr int kFB = 64;
constexpr int kFW = kFB / 32;
constexpr int kNG = 6;  // nodes a warp adds together, a lane per component
struct BlockLists {
  const int32_t *ptr, *node;  // the block's distinct nodes, most slots first
  const uint16_t* start;      // a node's first slot in the block's list
  const uint32_t* slot;       // the block's 4 kFB slots, four a word
};
struct BlockNodes {
  int32_t node[4 * kFB];
  uint16_t start[4 * kFB + 1];
  uint32_t slot[kFB];
};
// The block's lists into shared memory; returns its distinct nodes.
__device__ __forceinline__ int block_nodes(const BlockLists& l, int64_t ne, BlockNodes& s) {
  const int32_t b0 = __ldg(l.ptr + blockIdx.x), nu = __ldg(l.ptr + blockIdx.x + 1) - b0;
  for (int j = threadIdx.x; j < nu; j += kFB) {
    s.node[j] = __ldg(l.node + b0 + j);
    s.start[j] = __ldg(l.start + b0 + j);
  }
  s.slot[threadIdx.x] = __ldg(l.slot + int64_t(blockIdx.x) * kFB + threadIdx.x);
  const int64_t left = ne - int64_t(blockIdx.x) * kFB;
  if (threadIdx.x == 0) s.start[nu] = uint16_t(4 * (left < kFB ? left : kFB));
  return nu;
}
// Adds the contributions v[5 a + c][element] of the block, component by
// component (add(sum, v)), per distinct node and the sums (put(record, c, sum))
// to the node records acc [n][S], CH 16-byte pieces each.
template <int S, int CH, class T, class Sum, class A, class P>
__device__ __forceinline__ void block_add(const BlockNodes& s, int nu, const T (*v)[kFB + 1],
                                          float (*rec)[kNG][4 * CH], float* acc, Sum zero, A add,
                                          P put) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint8_t* slot = reinterpret_cast<const uint8_t*>(s.slot);
  const int g = lane / 5, c = lane - 5 * g;
  for (int j0 = w * kNG; j0 < nu; j0 += kFW * kNG) {
    if (g < kNG && j0 + g < nu) {
      Sum t = zero;
      const int k1 = s.start[j0 + g + 1];
#pragma unroll 4
      for (int k = s.start[j0 + g]; k < k1; ++k) {
        const int q = slot[k];
        add(t, v[(q & 3) * 5 + c][q >> 2]);
      }
      put(rec[w][g], c, t);
    }
    __syncwarp();
    if (lane < kNG * CH && j0 + lane / CH < nu) {
      const int h = lane / CH, k = lane % CH;
      atomicAdd(reinterpret_cast<float4*>(acc + int64_t(s.node[j0 + h]) * S) + k,
                *reinterpret_cast<const float4*>(&rec[w][h][4 * k]));
    }
    __syncwarp();
  }
}

// FP32 element pass: per node its residual and its ten antidiffusive sums
// (+, - per component; the sign that does not apply adds 0) in one [16]
// record; without FCT the residual alone.
__global__ void __launch_bounds__(kFB, 14) k_elem_rhs_aec32(int64_t n, int64_t ne,
                                                         const int32_t* __restrict__ inpoel,
                                                         const float* __restrict__ geo,
                                                         const float* __restrict__ V,
                                                         const KScalars* __restrict__ sc,
                                                         double gamma, double ctau, int fct,
                                                         const double* __restrict__ S,
                                                         const double* __restrict__ Se,
                                                         BlockLists lists, float* R) {
  __shared__ float2 v[20][kFB + 1];  // (residual, antidiffusive) per local node and component
  __shared__ __align__(16) float rec[kFW][kNG][16];
  __shared__ BlockNodes s;
  const int64_t e = blockIdx.x * int64_t(kFB) + threadIdx.x;
  const int nu = block_nodes(lists, ne, s);
  for (int k = threadIdx.x; k < kFW * kNG * 16; k += kFB) (&rec[0][0][0])[k] = 0.f;
  if (e < ne) {
    int32_t N[4];
    float r[4][5], aec[4][5];
    elem_terms<float>(n, ne, e, inpoel, geo, V, sc, float(gamma), float(ctau), fct, S, Se, N, r,
                      aec);
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
      for (int c = 0; c < 5; ++c) v[a * 5 + c][threadIdx.x] = make_float2(r[a][c], aec[a][c]);
  }
  __syncthreads();
  if (fct)
    block_add<kRP, 4>(
        s, nu, v, rec, R, make_float3(0.f, 0.f, 0.f),
        [](float3& t, float2 x) {
          t.x += x.x;
          t.y += x.y > 0.f ? x.y : 0.f;
          t.z += x.y < 0.f ? x.y : 0.f;
        },
        [](float* q, int c, float3 t) {
          q[c] = t.x;
          q[5 + 2 * c] = t.y;
          q[6 + 2 * c] = t.z;
        });
  else
    block_add<kRP, 2>(
        s, nu, v, reinterpret_cast<float(*)[kNG][8]>(rec), R, 0.f,
        [](float& t, float2 x) { t += x.x; }, [](float* q, int c, float t) { q[c] = t; });
}

// FP64 element passes hand their node contributions to the node passes through
// slot records, one per (element e, local node a), slot q = 4 e + a: the
// residual pass writes 10 doubles (the five contributions, then the five
// antidiffusive ones), the limiting pass 6 (the five limited contributions
// and a zero).  A warp's 32 elements own 128 consecutive records; each lane
// builds its four in shared memory (kStW double2 per lane: 16-byte stores
// of 8 lanes fall in distinct banks) and the warp moves the run to or from
// global memory with contiguous 512-byte accesses.
constexpr int kEB = 64;    // FP64 element-pass block: an SM's FP64 units take its blocks in turn
constexpr int kStW = 21;   // staged double2 per lane
constexpr int kRecD2 = 5;  // residual slot record, double2
constexpr int kLimD2 = 3;  // limited slot record, double2

template <int D2>  // double2 per element
__device__ __forceinline__ void warp_put(double2* __restrict__ g, const double2* buf, int nv,
                                         int lane) {
  for (int k = lane; k < nv * D2; k += 32) g[k] = buf[(k / D2) * kStW + k % D2];
}
template <int D2>
__device__ __forceinline__ void warp_get(const double2* __restrict__ g, double2* buf, int nv,
                                         int lane) {
  for (int k = lane; k < nv * D2; k += 32) buf[(k / D2) * kStW + k % D2] = __ldg(g + k);
}

__global__ void __launch_bounds__(kEB) k_elem_rhs64(int64_t n, int64_t ne,
                                                     const int32_t* __restrict__ inpoel,
                                                     const double* __restrict__ geo,
                                                     const double* __restrict__ V,
                                                     const KScalars* __restrict__ sc,
                                                     double gamma, double ctau, int fct,
                                                     const double* __restrict__ S,
                                                     const double* __restrict__ Se,
                                                     double* __restrict__ E) {
  __shared__ double2 st[kEB / 32][32 * kStW];
  const int lane = threadIdx.x & 31;
  const int64_t e = blockIdx.x * int64_t(kEB) + threadIdx.x;
  const int64_t e0 = e - lane;
  if (e0 >= ne) return;  // the whole warp is past the last element
  double2* buf = st[threadIdx.x >> 5];
  if (e < ne) {
    int32_t N[4];
    double r[4][5], aec[4][5];
    elem_terms<double>(n, ne, e, inpoel, geo, V, sc, gamma, ctau, fct, S, Se, N, r, aec);
    for (int a = 0; a < 4; ++a) {
      double2* b = buf + lane * kStW + a * kRecD2;
      b[0] = make_double2(r[a][0], r[a][1]);
      b[1] = make_double2(r[a][2], r[a][3]);
      b[2] = make_double2(r[a][4], aec[a][0]);
      b[3] = make_double2(aec[a][1], aec[a][2]);
      b[4] = make_double2(aec[a][3], aec[a][4]);
    }
  }
  __syncwarp();
  const int nv = static_cast<int>(ne - e0 < 32 ? ne - e0 : 32);
  warp_put<4 * kRecD2>(reinterpret_cast<double2*>(E) + e0 * 4 * kRecD2, buf, nv, lane);
}

struct KBC {
  int64_t nbc;
  const int32_t* node;
  const int32_t* dir;
  const int32_t* symp;
  const int32_t* dirmask;
  const double* dirval;
  const double* symn;
  SrcPrm prob;         // the problem whose analytic state mask-1 Dirichlet values take
  const double* xyz;   // [3][n] node coordinates
};

// What the node passes share.
struct NodeArgs {
  int64_t n;
  const double *ivol, *cbrtv;
  const KScalars* sc;
  KBC bc;
  const int32_t* bcof;
  int fct, clip;
  double gamma;
  double *U, *R, *P;  // state, low-order solution, P/vol [10][n]
  unsigned long long* dtmin;
};

// KozCG::alw node part (KozCG.cpp:887-912) at node i from its sums r and p
// (p[2c] positive, p[2c + 1] negative antidiffusive sums of component c):
// the symmetry projection of the momentum sums at BC nodes (KozCG.cpp:816-830),
// P /= vol and the low-order solution lo = U + dt R/vol - P+ - P-, with the
// keys of the node's extremes (lo, and U unless clip) for the allowed limits.
template <class F>
__device__ __forceinline__ void node_low(const NodeArgs& q, int64_t i, const double r[5],
                                         F p[10], typename KozT<F>::Key* __restrict__ K) {
  const int32_t b = __ldg(q.bcof + i);
  if (b >= 0) {
    for (int32_t k = q.bc.symp[b]; k < q.bc.symp[b + 1]; ++k) {
      const F nx = F(q.bc.symn[3 * k]), ny = F(q.bc.symn[3 * k + 1]), nz = F(q.bc.symn[3 * k + 2]);
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const F vn = p[2 + s] * nx + p[4 + s] * ny + p[6 + s] * nz;
        p[2 + s] -= vn * nx;
        p[4 + s] -= vn * ny;
        p[6 + s] -= vn * nz;
      }
    }
  }
  const double iv = q.ivol[i], dv = q.sc->dt * iv;
  typename KozT<F>::Key key[10];
#pragma unroll
  for (int c = 0; c < 5; ++c) {
    const double pp = iv * double(p[2 * c]), pn = iv * double(p[2 * c + 1]);
    q.P[(c * 2 + 0) * q.n + i] = pp;
    q.P[(c * 2 + 1) * q.n + i] = pn;
    const double u = q.U[c * q.n + i];
    const double lo = u + dv * r[c] - pp - pn;
    q.R[c * q.n + i] = lo;
    const F l = F(lo), uf = F(u);
    key[c * 2 + 0] = okey(q.clip ? l : fmax(l, uf));
    key[c * 2 + 1] = okey(q.clip ? l : fmin(l, uf));
  }
  store10(K + i * rec10<F>(), key);
}

// KozCG::solve's state u of node i (KozCG.cpp:1144-1160), its BCs (Dirichlet
// then symmetry at the step's end time, KozCG.cpp:590-611, 1167) and its CFL
// time step.
__device__ __forceinline__ double node_finish(const NodeArgs& q, int64_t i, double u[5]) {
  const int32_t b = __ldg(q.bcof + i);
  if (b >= 0) {
    const int32_t d = q.bc.dir[b];
    if (d >= 0)
      dirichlet(q.bc.prob, q.bc.xyz[i], q.bc.xyz[q.n + i], q.bc.xyz[2 * q.n + i], q.sc->tnext,
                q.bc.dirmask + d * 5, q.bc.dirval + d * 5, u);
    for (int32_t k = q.bc.symp[b]; k < q.bc.symp[b + 1]; ++k) {
      const double* nn = q.bc.symn + 3 * k;
      const double vn = u[1] * nn[0] + u[2] * nn[1] + u[3] * nn[2];
      u[1] -= vn * nn[0];
      u[2] -= vn * nn[1];
      u[3] -= vn * nn[2];
    }
  }
#pragma unroll
  for (int c = 0; c < 5; ++c) q.U[c * q.n + i] = u[c];
  return node_dt(u, q.cbrtv[i], q.gamma);
}

// FP32 mode: the node passes on the element sums in node records.
__global__ void __launch_bounds__(kBlock) k_node_low32(NodeArgs q, const float* __restrict__ acc,
                                                        unsigned int* __restrict__ K) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= q.n) return;
  float v[16];
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const float4 t = __ldg(reinterpret_cast<const float4*>(acc + i * kRP) + k);
    v[4 * k] = t.x;
    v[4 * k + 1] = t.y;
    v[4 * k + 2] = t.z;
    v[4 * k + 3] = t.w;
  }
  double r[5];
#pragma unroll
  for (int c = 0; c < 5; ++c) r[c] = double(v[c]);
  node_low<float>(q, i, r, v + 5, K);
}
__global__ void __launch_bounds__(kBlock) k_node_update32(NodeArgs q,
                                                           const float* __restrict__ acc) {
  // acc: the limited sums [n][8], or without FCT the residual records [n][16]
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  double dtp = DBL_MAX;
  if (i < q.n) {
    const float* a = acc + i * (q.fct ? kAR : kRP);
    const float4 t = __ldg(reinterpret_cast<const float4*>(a));
    const float v[5] = {t.x, t.y, t.z, t.w, __ldg(a + 4)};
    const double iv = q.fct ? q.ivol[i] : q.sc->dt * q.ivol[i];
    double u[5];
#pragma unroll
    for (int c = 0; c < 5; ++c)
      u[c] = (q.fct ? q.R : q.U)[c * q.n + i] + iv * double(v[c]);
    dtp = node_finish(q, i, u);
  }
  block_min_atomic(dtp, q.dtmin);
}

// Two quotients a/p and b/q from one division (batch inversion); the plain
// divisions where the product of the denominators leaves the normal range.
__device__ __forceinline__ void quotients(double a, double p, double b, double q, double& x,
                                          double& y) {
  const double d = p * q, m = fabs(d);
  if (m > 1e-290 && m < 1e290) {
    const double inv = 1.0 / d;
    x = a * (q * inv);
    y = b * (p * inv);
  } else {
    x = a / p;
    y = b / q;
  }
}
__device__ __forceinline__ void quotients(float a, float p, float b, float q, float& x, float& y) {
  x = a / p;
  y = b / q;
}

// KozCG::alw element part and KozCG::lim node part (KozCG.cpp:914-935,
// 1004-1024).  The allowed limits of a node are the maximum / minimum, over
// the elements holding it, of the element's extremes; the nodes of those
// elements are the node and its adjacency, so the same extremes are taken
// here per node over {i} and its neighbours (max and min are exact, so the
// bounds are the element loop's, without atomics), as integer comparisons of
// the keys: FP64 comparisons would hold the FP64 units, 280 a node (with the
// records and the two passes in one, 249 -> 67 us at 65^3).  Then Q -=
// low-order solution and the limit coefficients C+/- into Q.
template <class F>
__global__ void __launch_bounds__(kBlock)
    k_node_limit(int64_t n, const int32_t* __restrict__ aoff, const int32_t* __restrict__ aw,
                 const int32_t* __restrict__ nbr, const typename KozT<F>::Key* __restrict__ K,
                 const double* __restrict__ R, const double* __restrict__ P,
                 F* __restrict__ Q) {
  using Key = typename KozT<F>::Key;
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const int lane = static_cast<int>(i & 31);
  const int64_t s = i >> 5;
  const int32_t off = __ldg(aoff + s), w = __ldg(aw + s);
  constexpr int RL = rec10<F>();
  Key m[10];  // the maximum and minimum of each component, interleaved
  load10(K + i * RL, m);
  // two neighbours together: their records are in flight at once
  for (int k = 0; k < w; k += 2) {
    int32_t q[2];
    Key v[2][10];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      q[j] = k + j < w ? __ldg(nbr + off + (k + j) * 32 + lane) : -1;
      if (q[j] < 0) q[j] = static_cast<int32_t>(i);  // padding: the node itself
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) load10(K + int64_t(q[j]) * RL, v[j]);
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int c = 0; c < 5; ++c) {
        m[2 * c] = v[j][2 * c] > m[2 * c] ? v[j][2 * c] : m[2 * c];
        m[2 * c + 1] = v[j][2 * c + 1] < m[2 * c + 1] ? v[j][2 * c + 1] : m[2 * c + 1];
      }
  }
  const double eps = DBL_EPSILON;
  F out[10];
#pragma unroll
  for (int c = 0; c < 5; ++c) {
    const double lo = R[c * n + i];
    F qp = F(double(oval(m[2 * c])) - lo), qn = F(double(oval(m[2 * c + 1])) - lo);
    if (sizeof(F) == 4) {
      // the extremes hold float(lo), which may lie on the wrong side of lo: at a
      // node that is its own extreme nothing is allowed (FP64: exactly 0)
      qp = qp < F(0) ? F(0) : qp;
      qn = qn > F(0) ? F(0) : qn;
    }
    const double pp = P[(c * 2 + 0) * n + i], pn = P[(c * 2 + 1) * n + i];
    const bool zp = pp < eps, zn = pn > -eps;
    F cp, cn;
    quotients(qp, zp ? F(1) : F(pp), qn, zn ? F(1) : F(pn), cp, cn);
    out[c * 2 + 0] = zp ? F(0) : fmin(F(1), cp);
    out[c * 2 + 1] = zn ? F(0) : fmin(F(1), cn);
  }
  store10(Q + i * RL, out);
}

// KozCG::lim element part (KozCG.cpp:1049-1078): limited antidiffusive
// element contributions, system-limited over the components in sysmask.
// Limit coefficients of one element from its antidiffusive contributions
// aec[a][c] and the nodes' C+/- (Q); ca = the limited ones.  Signs and minima
// are taken on the bits of the values: the coefficients lie in [0, 1] or are -0
// (k_node_limit), which order as signed integers, and FP64 comparisons would
// hold the FP64 units.
__device__ __forceinline__ long long sbits(double v) { return __double_as_longlong(v); }
__device__ __forceinline__ int sbits(float v) { return __float_as_int(v); }
template <class F>
__device__ __forceinline__ F lesser(F a, F b) {
  return sbits(a) < sbits(b) ? a : b;
}
template <class F>
__device__ __forceinline__ void elem_limit(const int32_t N[4], const F* __restrict__ Q,
                                           int sysmask, const F aec[4][5], F ca[4][5]) {
  F coef[5];
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    F q[10];
    load10(Q + int64_t(N[a]) * rec10<F>(), q);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
      const F lim = sbits(aec[a][c]) > 0 ? q[2 * c] : q[2 * c + 1];
      coef[c] = lesser(a == 0 ? F(1.0) : coef[c], lim);
    }
  }
  F cs = F(1.0);
#pragma unroll
  for (int c = 0; c < 5; ++c)
    if (sysmask & (1 << c)) cs = lesser(cs, coef[c]);
#pragma unroll
  for (int c = 0; c < 5; ++c)
    if (sysmask & (1 << c)) coef[c] = cs;
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int c = 0; c < 5; ++c) ca[a][c] = coef[c] * aec[a][c];
}

// FP32: the antidiffusive contributions formed again from the FP32 state and
// geometry (as KozCG::lim does), the limited ones added atomically.
__global__ void __launch_bounds__(kBlock) k_elem_lim32(int64_t n, int64_t ne,
                                                        const int32_t* __restrict__ inpoel,
                                                        const float* __restrict__ geo,
                                                        const float* __restrict__ V,
                                                        const float* __restrict__ Q,
                                                        double ctau_d, int sysmask, float* A) {
  const int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (e >= ne) return;
  const int4 nd = __ldg(reinterpret_cast<const int4*>(inpoel) + e);
  const int32_t N[4] = {nd.x, nd.y, nd.z, nd.w};
  const float k = float(ctau_d) * __ldg(geo + e);  // ctau J/120
  float u[4][8], aec[4][5], ca[4][5];
#pragma unroll
  for (int a = 0; a < 4; ++a) load_node(V, N[a], u[a]);
  aec32(k, u, aec);
  elem_limit<float>(N, Q, sysmask, aec, ca);
  for (int a = 0; a < 4; ++a) {
    float* q = A + int64_t(N[a]) * kAR;
    atomicAdd(reinterpret_cast<float4*>(q), make_float4(ca[a][0], ca[a][1], ca[a][2], ca[a][3]));
    atomicAdd(q + 4, ca[a][4]);
  }
}

// FP64: the antidiffusive contributions are the ones the residual pass
// stored in the residual slot records E (the values KozCG::lim forms again
// from the same state and geometry); the limited ones go to the limited slot
// records L.
__global__ void __launch_bounds__(kEB) k_elem_lim64(int64_t n, int64_t ne,
                                                     const int32_t* __restrict__ inpoel,
                                                     const double* __restrict__ E,
                                                     const double* __restrict__ Q,
                                                     int sysmask, double* __restrict__ L) {
  __shared__ double2 st[kEB / 32][32 * kStW];
  const int lane = threadIdx.x & 31;
  const int64_t e = blockIdx.x * int64_t(kEB) + threadIdx.x;
  const int64_t e0 = e - lane;
  if (e0 >= ne) return;  // the whole warp is past the last element
  double2* buf = st[threadIdx.x >> 5];
  const int nv = static_cast<int>(ne - e0 < 32 ? ne - e0 : 32);
  warp_get<4 * kRecD2>(reinterpret_cast<const double2*>(E) + e0 * 4 * kRecD2, buf, nv, lane);
  __syncwarp();
  double ca[4][5];
  const bool live = e < ne;
  if (live) {
    int32_t N[4];
    for (int a = 0; a < 4; ++a) N[a] = inpoel[e * 4 + a];
    double aec[4][5];
    for (int a = 0; a < 4; ++a) {
      const double* rec = reinterpret_cast<const double*>(buf + lane * kStW + a * kRecD2);
      for (int c = 0; c < 5; ++c) aec[a][c] = rec[5 + c];
    }
    elem_limit<double>(N, Q, sysmask, aec, ca);
  }
  __syncwarp();
  if (live)
    for (int a = 0; a < 4; ++a) {
      double2* b = buf + lane * kStW + a * kLimD2;
      b[0] = make_double2(ca[a][0], ca[a][1]);
      b[1] = make_double2(ca[a][2], ca[a][3]);
      b[2] = make_double2(ca[a][4], 0.0);
    }
  __syncwarp();
  warp_put<4 * kLimD2>(reinterpret_cast<double2*>(L) + e0 * 4 * kLimD2, buf, nv, lane);
}

// FP64 node sums of the element contributions, in a fixed order: node i
// adds the slots (element e, local node a) of the elements holding it in
// ascending e -- the order of the reference's serial element loop
// (Kozak.cpp:73-173 adds R[N[a]] per element, KozCG.cpp:794-814 and
// 1049-1078 likewise P and A) -- so the sums are the same on every run, with
// no atomics.  Slot q's record is RD2 double2 at E + q * RD2: entries 0..4
// the contributions to the node's five components, and with WP entries
// 5..9 the antidiffusive ones, summed by sign into P+ / P- (zero goes to
// neither).  Slots as SELL-32: slice s of 32 nodes, entry k of node i at
// soff[s] + 32 k + lane, value q, -1 padding.  The slots are taken kGB at a
// time, their loads issued together before the adds (in slot order), so
// that a node's loads overlap.
template <int RD2, bool WP>
__device__ __forceinline__ void node_slots(int64_t i, const int32_t* __restrict__ soff,
                                           const int32_t* __restrict__ sw,
                                           const int32_t* __restrict__ slot,
                                           const double* __restrict__ E, double r[5],
                                           double p[10]) {
  constexpr int LD2 = WP ? 5 : 3;  // double2 read per slot
  const int lane = static_cast<int>(i & 31);
  const int64_t s = i >> 5;
  const int32_t off = __ldg(soff + s), w = __ldg(sw + s);
  const double2* E2 = reinterpret_cast<const double2*>(E);
#pragma unroll
  for (int c = 0; c < 5; ++c) r[c] = p[2 * c] = p[2 * c + 1] = 0.0;
  for (int k0 = 0; k0 < w; k0 += kGB) {
    int32_t q[kGB];
#pragma unroll
    for (int j = 0; j < kGB; ++j) q[j] = k0 + j < w ? __ldg(slot + off + (k0 + j) * 32 + lane) : -1;
    double x[kGB][2 * LD2];
#pragma unroll
    for (int j = 0; j < kGB; ++j) {
      const int64_t qq = q[j] >= 0 ? q[j] : 0;  // padding reads slot 0, unused
#pragma unroll
      for (int k = 0; k < LD2; ++k) {
        const double2 t = __ldg(E2 + qq * RD2 + k);
        x[j][2 * k] = t.x;
        x[j][2 * k + 1] = t.y;
      }
    }
#pragma unroll
    for (int j = 0; j < kGB; ++j) {
      if (q[j] < 0) break;  // padding only after a node's last slot
#pragma unroll
      for (int c = 0; c < 5; ++c) r[c] += x[j][c];
      if constexpr (WP) {
#pragma unroll
        for (int c = 0; c < 5; ++c) {
          // one FP64 addition to the sum of v's sign (a zero changes neither, a
          // NaN is left out), chosen on the bits: a branch per sign adds in
          // both where a warp's lanes differ, and a comparison, or a 64-bit NaN
          // test that the compiler makes one of, holds the FP64 pipe as well
          const double v = x[j][5 + c];
          const int hi = __double2hiint(v);
          const bool nan = unsigned(hi & 0x7fffffff) + (__double2loint(v) != 0) > 0x7ff00000u;
          const double t = (hi >= 0 ? p[2 * c] : p[2 * c + 1]) + (nan ? 0.0 : v);
          p[2 * c] = hi >= 0 ? t : p[2 * c];
          p[2 * c + 1] = hi >= 0 ? p[2 * c + 1] : t;
        }
      }
    }
  }
}

// The FP64 node passes: the slots' sums, then the node's algebra, in one
// kernel each (sums, boundary projection and low-order solution in kernels of
// their own moved 240 bytes a node through memory in between).
__global__ void __launch_bounds__(kBlock) k_node_low64(NodeArgs q,
                                                        const int32_t* __restrict__ soff,
                                                        const int32_t* __restrict__ sw,
                                                        const int32_t* __restrict__ slot,
                                                        const double* __restrict__ E,
                                                        unsigned long long* __restrict__ K) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= q.n) return;
  double r[5], p[10];
  node_slots<kRecD2, true>(i, soff, sw, slot, E, r, p);
  node_low<double>(q, i, r, p, K);
}
// FCT: E the limited slot records; otherwise the residual ones.
template <bool FCT>
__global__ void __launch_bounds__(kBlock) k_node_update64(NodeArgs q,
                                                           const int32_t* __restrict__ soff,
                                                           const int32_t* __restrict__ sw,
                                                           const int32_t* __restrict__ slot,
                                                           const double* __restrict__ E) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  double dtp = DBL_MAX;
  if (i < q.n) {
    double r[5], p[10];
    node_slots<FCT ? kLimD2 : kRecD2, false>(i, soff, sw, slot, E, r, p);
    const double iv = FCT ? q.ivol[i] : q.sc->dt * q.ivol[i];
    double u[5];
#pragma unroll
    for (int c = 0; c < 5; ++c) u[c] = (FCT ? q.R : q.U)[c * q.n + i] + iv * r[c];
    dtp = node_finish(q, i, u);
  }
  block_min_atomic(dtp, q.dtmin);
}
// The residual alone (xg_kozcg_rhs).
__global__ void __launch_bounds__(kBlock) k_node_rhs64(int64_t n,
                                                        const int32_t* __restrict__ soff,
                                                        const int32_t* __restrict__ sw,
                                                        const int32_t* __restrict__ slot,
                                                        const double* __restrict__ E,
                                                        double* __restrict__ R) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  double r[5], p[10];
  node_slots<kRecD2, false>(i, soff, sw, slot, E, r, p);
#pragma unroll
  for (int c = 0; c < 5; ++c) R[c * n + i] = r[c];
}

// Nodal BCs (KozCG::BC) on the device state at the caller's time t.
__global__ void __launch_bounds__(kBlock) k_bc(int64_t n, KBC bc, double* U, double t) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= bc.nbc) return;
  const int64_t p = bc.node[i];
  double u[5];
  for (int c = 0; c < 5; ++c) u[c] = U[c * n + p];
  const int32_t d = bc.dir[i];
  if (d >= 0)
    dirichlet(bc.prob, bc.xyz[p], bc.xyz[n + p], bc.xyz[2 * n + p], t, bc.dirmask + d * 5,
              bc.dirval + d * 5, u);
  for (int32_t k = bc.symp[i]; k < bc.symp[i + 1]; ++k) {
    const double* nn = bc.symn + 3 * k;
    double vn = u[1] * nn[0] + u[2] * nn[1] + u[3] * nn[2];
    u[1] -= vn * nn[0];
    u[2] -= vn * nn[1];
    u[3] -= vn * nn[2];
  }
  for (int c = 0; c < 5; ++c) U[c * n + p] = u[c];
}

__global__ void k_dt(int64_t n, const double* __restrict__ U, const double* __restrict__ cbrtv,
                     double gamma, unsigned long long* dtmin) {
  int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  double dtp = DBL_MAX;
  if (p < n) {
    double u[5];
    for (int c = 0; c < 5; ++c) u[c] = U[c * n + p];
    dtp = node_dt(u, cbrtv[p], gamma);
  }
  block_min_atomic(dtp, dtmin);
}

__global__ void k_step_begin(KScalars* s, double cfl, double const_dt, double* hist, int64_t k) {
  double dt;
  if (fabs(const_dt) > DBL_EPSILON)
    dt = const_dt;
  else
    dt = __longlong_as_double(s->dtmin) * cfl;
  if (dt < DBL_EPSILON) s->blowup = 1;
  s->dt = dt;
  s->t = s->tnext;
  s->tnext = s->t + dt;
  s->dtmin = __double_as_longlong(DBL_MAX);
  if (hist) hist[k] = dt;
}
// A step of the caller's dt from time t (its CFL minimum starts afresh).
__global__ void k_set_step(KScalars* s, double t, double dt) {
  s->t = t;
  s->dt = dt;
  s->tnext = t + dt;
  s->dtmin = __double_as_longlong(DBL_MAX);
}
__global__ void k_set_time(KScalars* s, double t) {
  s->t = t;
  s->tnext = t;
}

// The sources kozak::rhs adds (src/Physics/Kozak.cpp:125-132, 161-170): at
// every node at the step's start time, S [5][n], and at every element's
// centroid (the mean of its nodes' coordinates) half a step later, Se [ne][5].
__global__ void k_src_nodes(int64_t n, SrcPrm q, const KScalars* __restrict__ sc,
                            const double* __restrict__ xyz, double* __restrict__ S) {
  const int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (p >= n) return;
  double o[5];
  problem_source(q, xyz[p], xyz[n + p], xyz[2 * n + p], sc->t, o);
  for (int c = 0; c < 5; ++c) S[c * n + p] = o[c];
}
__global__ void k_src_elems(int64_t n, int64_t ne, SrcPrm q, const KScalars* __restrict__ sc,
                            const int32_t* __restrict__ inpoel, const double* __restrict__ xyz,
                            double* __restrict__ Se) {
  const int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (e >= ne) return;
  const int32_t* N = inpoel + e * 4;
  double c3[3];
  for (int j = 0; j < 3; ++j) {
    const double* x = xyz + j * n;
    c3[j] = (x[N[0]] + x[N[1]] + x[N[2]] + x[N[3]]) / 4.0;
  }
  double o[5];
  problem_source(q, c3[0], c3[1], c3[2], sc->t + sc->dt / 2.0, o);
  for (int c = 0; c < 5; ++c) Se[e * 5 + c] = o[c];
}

// 1/vol and cbrt(vol).
__global__ void k_node_factors(int64_t n, const double* __restrict__ vol,
                               double* __restrict__ ivol, double* __restrict__ cbrtv) {
  const int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (p >= n) return;
  ivol[p] = 1.0 / vol[p];
  cbrtv[p] = cbrt(vol[p]);
}

__global__ void k_reset_min(KScalars* s) { s->dtmin = __double_as_longlong(DBL_MAX); }

__global__ void k_aos_to_soa(int64_t n, int nc, const double* __restrict__ a,
                             double* __restrict__ s) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n * nc) return;
  int64_t p = i / nc;
  int c = static_cast<int>(i - p * nc);
  s[c * n + p] = a[i];
}
__global__ void k_soa_to_aos(int64_t n, int nc, const double* __restrict__ s,
                             double* __restrict__ a) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n * nc) return;
  int64_t p = i / nc;
  int c = static_cast<int>(i - p * nc);
  a[i] = s[c * n + p];
}

KBC kbc_of(KozCGDev* d) {
  return KBC{d->nbc,   d->bcnode, d->bcdir, d->bcsymp, d->dirmask,
             d->dirval, d->symn,  d->src,   d->xyz};
}

int refresh_dt(xg_ctx* c, KozCGDev* d) {
  k_reset_min<<<1, 1, 0, c->stream>>>(d->scal);
  XG_CHECK_LAUNCH(c);
  k_dt<<<blocks_for(d->n, kBlock), kBlock, 0, c->stream>>>(d->n, d->U, d->cbrtv, d->prm.gamma,
                                                            &d->scal->dtmin);
  XG_CHECK_LAUNCH(c);
  d->dt_valid = true;
  return XG_OK;
}

NodeArgs node_args(KozCGDev* d) {
  return NodeArgs{d->n,  d->ivol,         d->cbrtv,    d->scal,      kbc_of(d),
                  d->bcof, d->prm.fct,    d->prm.fctclip, d->prm.gamma, d->U,
                  d->R,  d->P,            &d->scal->dtmin};
}

BlockLists block_lists(const KozCGDev* d) {
  return BlockLists{d->bptr, d->bnode, d->bstart, reinterpret_cast<const uint32_t*>(d->bslot)};
}

// Node primitives and the element Galerkin (+ antidiffusive) pass on state U:
// in FP64 into the residual slot records, in FP32 added into the zeroed node
// records.
template <class F>
void galerkin(xg_ctx* c, KozCGDev* d, const double* U, int fct) {
  cudaStream_t s = c->stream;
  const int64_t n = d->n, ne = d->ne;
  const double *S = nullptr, *Se = nullptr;
  if (d->src.problem != XG_SRC_NONE) {
    k_src_nodes<<<blocks_for(n, kBlock), kBlock, 0, s>>>(n, d->src, d->scal, d->xyz, d->S);
    k_src_elems<<<blocks_for(ne, kBlock), kBlock, 0, s>>>(n, ne, d->src, d->scal, d->inpoel,
                                                          d->xyz, d->Se);
    S = d->S;
    Se = d->Se;
  }
  const int tb = node_block(c, n, kBlock);
  F* V = reinterpret_cast<F*>(d->V);
  if constexpr (sizeof(F) == 8) {
    k_node_prim<double><<<blocks_for(n, tb), tb, 0, s>>>(n, U, d->prm.gamma, V);
    k_elem_rhs64<<<blocks_for(ne, kEB), kEB, 0, s>>>(n, ne, d->inpoel, d->geo64, V, d->scal,
                                                     d->prm.gamma, d->prm.ctau, fct, S, Se,
                                                     d->E);
  } else {
    k_node_prim<float><<<blocks_for(n, tb), tb, 0, s>>>(n, U, d->prm.gamma, V);
    k_elem_rhs_aec32<<<blocks_for(ne, kFB), kFB, 0, s>>>(n, ne, d->inpoel, d->geo32, V,
                                                         d->scal, d->prm.gamma, d->prm.ctau, fct,
                                                         S, Se, block_lists(d), d->R32);
  }
}

// One KozCG step with the dt already in the device scalars, element
// arithmetic in F.
template <class F>
int step_impl(xg_ctx* c, KozCGDev* d) {
  cudaStream_t s = c->stream;
  const int64_t n = d->n, ne = d->ne;
  const int fct = d->prm.fct;
  const int tb = node_block(c, n, kBlock);
  const unsigned nb = blocks_for(n, tb);
  const NodeArgs q = node_args(d);
  // FP32: R with P [n][16], A [n][8] accumulate atomically from zero
  if (sizeof(F) == 4) {
    XG_CUDA(c, cudaMemsetAsync(d->R32, 0, n * kRP * 4, s));
    if (fct) XG_CUDA(c, cudaMemsetAsync(d->A32, 0, n * kAR * 4, s));
  }
  galerkin<F>(c, d, d->U, fct);
  XG_CHECK_LAUNCH(c);
  if constexpr (sizeof(F) == 4) {
    if (fct) {
      k_node_low32<<<nb, tb, 0, s>>>(q, d->R32, d->K32);
      k_node_limit<float><<<nb, tb, 0, s>>>(n, d->aoff, d->aw, d->anbr, d->K32, d->R, d->P,
                                            d->Q32);
      const int eb = node_block(c, ne, kBlock);
      k_elem_lim32<<<blocks_for(ne, eb), eb, 0, s>>>(n, ne, d->inpoel, d->geo32,
                                                     reinterpret_cast<float*>(d->V), d->Q32,
                                                     d->prm.ctau, d->prm.fctsys, d->A32);
    }
    k_node_update32<<<nb, tb, 0, s>>>(q, fct ? d->A32 : d->R32);
  } else {
    if (fct) {
      k_node_low64<<<nb, tb, 0, s>>>(q, d->soff, d->sw, d->sslot, d->E, d->K);
      k_node_limit<double><<<nb, tb, 0, s>>>(n, d->aoff, d->aw, d->anbr, d->K, d->R, d->P, d->Q);
      k_elem_lim64<<<blocks_for(ne, kEB), kEB, 0, s>>>(n, ne, d->inpoel, d->E, d->Q,
                                                       d->prm.fctsys, d->L);
      k_node_update64<true><<<nb, tb, 0, s>>>(q, d->soff, d->sw, d->sslot, d->L);
    } else {
      k_node_update64<false><<<nb, tb, 0, s>>>(q, d->soff, d->sw, d->sslot, d->E);
    }
  }
  XG_CHECK_LAUNCH(c);
  return XG_OK;
}

int step(xg_ctx* c, KozCGDev* d) {
  if (d->prm.precision == XG_FP32_FLUX) return step_impl<float>(c, d);
  return step_impl<double>(c, d);
}

// The residual of FP32 node records [n][16] to FP64 [5][n].
__global__ void k_rec_to_soa(int64_t n, const float* __restrict__ a, double* __restrict__ b) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n * 5) return;
  const int64_t c = i / n, p = i - c * n;
  b[i] = double(a[p * kRP + c]);
}

}  // namespace
}  // namespace xg

using namespace xg;

extern "C" {

int xg_kozcg_setup(xg_ctx* c, const xg_kozcg_params* prm, int64_t npoin, const double* coord,
                   const double* vol, int64_t nelem, const uint64_t* inpoel) {
  XG_HOST_TRY
  int rc = use(c);
  if (rc) return rc;
  if (!prm || npoin <= 0 || nelem <= 0 || !coord || !vol || !inpoel)
    return fail(c, XG_ERR_ARG, "kozcg_setup: bad mesh");
  if (npoin >= (int64_t(1) << 31) - 64) return fail(c, XG_ERR_ARG, "kozcg_setup: too many nodes");
  if (prm->fctsys & ~31) return fail(c, XG_ERR_ARG, "kozcg_setup: fctsys mask beyond 5 components");
  if (prm->precision != XG_FP64 && prm->precision != XG_FP32_FLUX)
    return fail(c, XG_ERR_ARG, "kozcg_setup: unknown precision");
  for (int64_t i = 0; i < nelem * 4; ++i)
    if (inpoel[i] >= static_cast<uint64_t>(npoin))
      return fail(c, XG_ERR_ARG, "kozcg_setup: element node id out of range");
  // Elements in the order of their smallest node id (stable counting sort),
  // so that consecutive elements share nearby nodes: the element passes then
  // read nearby node data, and the elements holding a run of nodes (the
  // slots one warp of a node pass reads) lie in a window of the slot
  // records about the mesh's node bandwidth wide, instead of across the
  // whole array.  Results do not depend on the element order beyond the
  // order of each node's sums, which stays fixed.
  std::vector<int32_t> ip(nelem * 4);
  {
    std::vector<int64_t> cnt(npoin + 1, 0);
    std::vector<int32_t> key(nelem);
    for (int64_t e = 0; e < nelem; ++e) {
      uint64_t m = inpoel[e * 4];
      for (int a = 1; a < 4; ++a) m = std::min(m, inpoel[e * 4 + a]);
      key[e] = static_cast<int32_t>(m);
      ++cnt[m + 1];
    }
    for (int64_t i = 0; i < npoin; ++i) cnt[i + 1] += cnt[i];
    for (int64_t e = 0; e < nelem; ++e) {
      const int64_t to = cnt[key[e]]++;
      for (int a = 0; a < 4; ++a) ip[to * 4 + a] = static_cast<int32_t>(inpoel[e * 4 + a]);
    }
  }
  // node adjacency for the allowed limits: the elements of each node
  // (counting sort), then each node's sorted distinct element neighbours,
  // laid out as SELL-32
  const int64_t nslice = (npoin + 31) / 32;
  const bool f64 = prm->precision == XG_FP64;
  if (f64 && nelem * 4 >= (int64_t(1) << 31))
    return fail(c, XG_ERR_ARG, "kozcg_setup: too many elements for FP64 slots");
  std::vector<int32_t> aoff(nslice + 1), aw(nslice), anbr;
  // FP64 node sums: per node its (element, local node) slots e * 4 + a in
  // ascending e, SELL-32 (slice offsets soff, widths sw, -1 padding)
  std::vector<int32_t> soff(nslice + 1), sw(nslice), sslot;
  {
    std::vector<int64_t> eptr(npoin + 1, 0);
    for (int64_t i = 0; i < nelem * 4; ++i) ++eptr[ip[i] + 1];
    for (int64_t i = 0; i < npoin; ++i) eptr[i + 1] += eptr[i];
    std::vector<int32_t> eln(nelem * 4), els(f64 ? nelem * 4 : 0);
    {
      std::vector<int64_t> fill(eptr.begin(), eptr.end() - 1);
      for (int64_t e = 0; e < nelem; ++e)
        for (int a = 0; a < 4; ++a) {
          const int64_t k = fill[ip[e * 4 + a]]++;
          eln[k] = static_cast<int32_t>(e);
          if (f64) els[k] = static_cast<int32_t>(e * 4 + a);
        }
    }
    if (f64) {
      int64_t tot = 0;
      for (int64_t sl = 0; sl < nslice; ++sl) {
        int64_t w = 0;
        for (int64_t i = sl * 32; i < std::min<int64_t>(npoin, sl * 32 + 32); ++i)
          w = std::max(w, eptr[i + 1] - eptr[i]);
        soff[sl] = static_cast<int32_t>(tot);
        sw[sl] = static_cast<int32_t>(w);
        tot += 32 * w;
        if (tot >= (int64_t(1) << 31)) return fail(c, XG_ERR_ARG, "kozcg_setup: slots too many");
      }
      soff[nslice] = static_cast<int32_t>(tot);
      sslot.assign(static_cast<size_t>(std::max<int64_t>(1, tot)), -1);
      for (int64_t i = 0; i < npoin; ++i) {
        const int64_t sl = i / 32, lane = i % 32;
        for (int64_t k = eptr[i]; k < eptr[i + 1]; ++k)
          sslot[soff[sl] + (k - eptr[i]) * 32 + lane] = els[k];
      }
    }
    std::vector<int64_t> nptr(npoin + 1, 0);
    std::vector<int32_t> nb;
    nb.reserve(static_cast<size_t>(npoin) * 16);
    std::vector<int32_t> tmp, met(npoin, -1);  // met: the last node a node was found beside
    for (int64_t i = 0; i < npoin; ++i) {
      tmp.clear();
      met[i] = static_cast<int32_t>(i);
      for (int64_t k = eptr[i]; k < eptr[i + 1]; ++k)
        for (int a = 0; a < 4; ++a) {
          const int32_t j = ip[int64_t(eln[k]) * 4 + a];
          if (met[j] != i) {
            met[j] = static_cast<int32_t>(i);
            tmp.push_back(j);
          }
        }
      std::sort(tmp.begin(), tmp.end());
      nb.insert(nb.end(), tmp.begin(), tmp.end());
      nptr[i + 1] = static_cast<int64_t>(nb.size());
    }
    int64_t tot = 0;
    for (int64_t sl = 0; sl < nslice; ++sl) {
      int64_t w = 0;
      for (int64_t i = sl * 32; i < std::min<int64_t>(npoin, sl * 32 + 32); ++i)
        w = std::max(w, nptr[i + 1] - nptr[i]);
      aoff[sl] = static_cast<int32_t>(tot);
      aw[sl] = static_cast<int32_t>(w);
      tot += 32 * w;
      if (tot >= (int64_t(1) << 31)) return fail(c, XG_ERR_ARG, "kozcg_setup: adjacency too large");
    }
    aoff[nslice] = static_cast<int32_t>(tot);
    anbr.assign(static_cast<size_t>(std::max<int64_t>(1, tot)), -1);
    for (int64_t i = 0; i < npoin; ++i) {
      const int64_t sl = i / 32, lane = i % 32;
      for (int64_t k = nptr[i]; k < nptr[i + 1]; ++k)
        anbr[aoff[sl] + (k - nptr[i]) * 32 + lane] = nb[k];
    }
  }
  // FP32: the distinct nodes of each block of kFB elements, most slots first
  // (the lanes that add a block's nodes together then loop alike), and their
  // slots in ascending order
  std::vector<int32_t> bptr, bnode;
  std::vector<uint16_t> bstart;
  std::vector<uint8_t> bslot;
  if (!f64) {
    const int64_t nblk = (nelem + kFB - 1) / kFB;
    bptr.assign(static_cast<size_t>(nblk + 1), 0);
    bslot.assign(static_cast<size_t>(nblk * 4 * kFB), 0);
    bnode.reserve(static_cast<size_t>(nelem));
    bstart.reserve(static_cast<size_t>(nelem));
    std::vector<int32_t> seen(npoin, -1);  // the last block that holds a node
    std::vector<uint8_t> idx(npoin);       // its place there, in order of appearance
    for (int64_t b = 0; b < nblk; ++b) {
      const int nq = static_cast<int>(std::min<int64_t>(4 * kFB, nelem * 4 - b * 4 * kFB));
      const int32_t* q = ip.data() + b * 4 * kFB;
      int32_t node[4 * kFB];
      int cnt[4 * kFB], of[4 * kFB], first[4 * kFB + 2] = {}, start[4 * kFB];
      int nu = 0;
      for (int k = 0; k < nq; ++k) {
        if (seen[q[k]] != b) {
          seen[q[k]] = static_cast<int32_t>(b);
          idx[q[k]] = static_cast<uint8_t>(nu);
          node[nu] = q[k];
          cnt[nu++] = 0;
        }
        ++cnt[idx[q[k]]];
      }
      for (int j = 0; j < nu; ++j) ++first[4 * kFB - cnt[j] + 1];
      for (int k = 0; k <= 4 * kFB; ++k) first[k + 1] += first[k];
      for (int j = 0; j < nu; ++j) of[j] = first[4 * kFB - cnt[j]]++;  // place, most slots first
      int32_t sorted[4 * kFB];
      int count[4 * kFB];
      for (int j = 0; j < nu; ++j) {
        sorted[of[j]] = node[j];
        count[of[j]] = cnt[j];
      }
      for (int j = 0, k = 0; j < nu; k += count[j++]) {
        start[j] = k;
        bnode.push_back(sorted[j]);
        bstart.push_back(static_cast<uint16_t>(k));
      }
      for (int k = 0; k < nq; ++k) {
        const int j = of[idx[q[k]]];
        bslot[b * 4 * kFB + start[j]++] = static_cast<uint8_t>(k);
      }
      if (bnode.size() >= (size_t(1) << 31))
        return fail(c, XG_ERR_ARG, "kozcg_setup: too many elements");
      bptr[b + 1] = static_cast<int32_t>(bnode.size());
    }
  }
  if (c->kozcg) {
    XG_CUDA(c, cudaStreamSynchronize(c->stream));
    destroy_kozcg(c->kozcg);
    c->kozcg = nullptr;
  }
  auto* d = new KozCGDev;
  c->kozcg = d;
  d->n = npoin;
  d->ne = nelem;
  d->prm = *prm;
  d->nslice = nslice;
  for (int pass = 0; pass < 2; ++pass) {
    Arena& A = d->arena;
    A.plan(d->inpoel, nelem * 4);
    A.plan(d->xyz, npoin * 3);
    A.plan(d->ivol, npoin);
    A.plan(d->cbrtv, npoin);
    A.plan(d->U, npoin * 5);
    A.plan(d->R, npoin * 5);
    A.plan(d->P, npoin * 10);
    A.plan(d->A, npoin * 5);
    A.plan(d->stage, npoin * 5);
    A.plan(d->V, f64 ? npoin * 8 : npoin * 4);  // [n][8] of the mode's precision
    A.plan(d->aoff, aoff.size());
    A.plan(d->aw, aw.size());
    A.plan(d->anbr, anbr.size());
    if (prm->precision == XG_FP32_FLUX) {
      A.plan(d->R32, npoin * 16);  // R and P records
      A.plan(d->A32, npoin * 8);
      A.plan(d->Q32, npoin * kC32);
      A.plan(d->K32, npoin * kC32);
      A.plan(d->geo32, nelem * kGeo);
      A.plan(d->bptr, bptr.size());
      A.plan(d->bnode, bnode.size());
      A.plan(d->bstart, bstart.size());
      A.plan(d->bslot, bslot.size());
    } else {
      A.plan(d->Q, npoin * kC64);
      A.plan(d->K, npoin * kC64);
      A.plan(d->geo64, nelem * kGeo);
      A.plan(d->E, nelem * 4 * kRecD2 * 2);
      if (prm->fct) A.plan(d->L, nelem * 4 * kLimD2 * 2);
      A.plan(d->soff, soff.size());
      A.plan(d->sw, sw.size());
      A.plan(d->sslot, sslot.size());
    }
    A.plan(d->bcof, npoin);
    A.plan(d->scal, 1);
    if (pass == 0) {
      cudaError_t e = A.reserve();
      if (e != cudaSuccess) {
        destroy_kozcg(d);
        c->kozcg = nullptr;
        return fail(c, XG_ERR_CUDA, std::string("kozcg_setup: ") + cudaGetErrorString(e));
      }
    }
  }
  cudaStream_t s = c->stream;
  auto up = [&](void* dst, const void* src, size_t bytes) { return upload(c, dst, src, bytes); };
  XG_CUDA(c, up(d->inpoel, ip.data(), ip.size() * 4));
  XG_CUDA(c, up(d->xyz, coord, npoin * 3 * 8));
  // through the staging buffer
  XG_CUDA(c, up(d->stage, vol, npoin * 8));
  k_node_factors<<<blocks_for(npoin, kBlock), kBlock, 0, s>>>(npoin, d->stage, d->ivol, d->cbrtv);
  XG_CHECK_LAUNCH(c);
  XG_CUDA(c, up(d->aoff, aoff.data(), aoff.size() * 4));
  XG_CUDA(c, up(d->aw, aw.data(), aw.size() * 4));
  XG_CUDA(c, up(d->anbr, anbr.data(), anbr.size() * 4));
  if (!f64) {
    XG_CUDA(c, up(d->bptr, bptr.data(), bptr.size() * 4));
    XG_CUDA(c, up(d->bnode, bnode.data(), bnode.size() * 4));
    XG_CUDA(c, up(d->bstart, bstart.data(), bstart.size() * 2));
    XG_CUDA(c, up(d->bslot, bslot.data(), bslot.size()));
  }
  if (f64) {
    XG_CUDA(c, up(d->soff, soff.data(), soff.size() * 4));
    XG_CUDA(c, up(d->sw, sw.data(), sw.size() * 4));
    XG_CUDA(c, up(d->sslot, sslot.data(), sslot.size() * 4));
  }
  XG_CUDA(c, cudaMemsetAsync(d->U, 0, npoin * 5 * 8, s));
  XG_CUDA(c, cudaMemsetAsync(d->bcof, 0xff, npoin * 4, s));  // -1
  if (f64)
    k_geo<double><<<blocks_for(nelem, kBlock), kBlock, 0, s>>>(npoin, nelem, d->inpoel, d->xyz,
                                                               d->geo64);
  else
    k_geo<float><<<blocks_for(nelem, kBlock), kBlock, 0, s>>>(npoin, nelem, d->inpoel, d->xyz,
                                                              d->geo32);
  XG_CHECK_LAUNCH(c);
  KScalars k0{};  // every member zero
  double big = DBL_MAX;
  std::memcpy(&k0.dtmin, &big, sizeof(double));
  XG_CUDA(c, cudaMemcpyAsync(d->scal, &k0, sizeof(k0), cudaMemcpyHostToDevice, s));
  XG_CUDA(c, cudaStreamSynchronize(s));
  return XG_OK;
  XG_HOST_CATCH(c)
}

int xg_kozcg_set_bc(xg_ctx* c, int64_t nsym, const uint64_t* symnodes, const double* symnorms,
                    int64_t ndir, const uint64_t* dirnodes, const int32_t* dirmask,
                    const double* dirvals) {
  XG_HOST_TRY
  int rc = use(c);
  if (rc) return rc;
  KozCGDev* d = c->kozcg;
  if (!d) return fail(c, XG_ERR_STATE, "kozcg_set_bc before kozcg_setup");
  if ((nsym && (!symnodes || !symnorms)) || (ndir && (!dirnodes || !dirmask || !dirvals)))
    return fail(c, XG_ERR_ARG, "kozcg_set_bc: null array");
  const int64_t n = d->n;
  std::vector<int64_t> ids;
  for (int64_t i = 0; i < nsym; ++i) {
    if (symnodes[i] >= uint64_t(n)) return fail(c, XG_ERR_ARG, "kozcg_set_bc: node id");
    ids.push_back(int64_t(symnodes[i]));
  }
  for (int64_t i = 0; i < ndir; ++i) {
    if (dirnodes[i] >= uint64_t(n)) return fail(c, XG_ERR_ARG, "kozcg_set_bc: node id");
    ids.push_back(int64_t(dirnodes[i]));
  }
  std::sort(ids.begin(), ids.end());
  ids.erase(std::unique(ids.begin(), ids.end()), ids.end());
  const int64_t nbc = static_cast<int64_t>(ids.size());
  auto pos = [&](uint64_t p) {
    return static_cast<int64_t>(std::lower_bound(ids.begin(), ids.end(), int64_t(p)) - ids.begin());
  };
  std::vector<int32_t> node(nbc), dir(nbc, -1), symp(nbc + 1, 0);
  for (int64_t i = 0; i < nbc; ++i) node[i] = static_cast<int32_t>(ids[i]);
  for (int64_t k = 0; k < ndir; ++k) dir[pos(dirnodes[k])] = static_cast<int32_t>(k);
  std::vector<int64_t> cnt(nbc, 0);
  for (int64_t k = 0; k < nsym; ++k) ++cnt[pos(symnodes[k])];
  for (int64_t i = 0; i < nbc; ++i) symp[i + 1] = symp[i] + static_cast<int32_t>(cnt[i]);
  std::vector<double> symn(std::max<int64_t>(1, nsym) * 3, 0.0);
  {
    std::vector<int32_t> fill(symp.begin(), symp.end() - 1);
    for (int64_t k = 0; k < nsym; ++k) {
      int32_t j = fill[pos(symnodes[k])]++;
      for (int a = 0; a < 3; ++a) symn[j * 3 + a] = symnorms[k * 3 + a];
    }
  }
  std::vector<int32_t> bcof(n, -1);
  for (int64_t i = 0; i < nbc; ++i) bcof[ids[i]] = static_cast<int32_t>(i);
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  d->bcarena.release();
  for (int pass = 0; pass < 2; ++pass) {
    Arena& A = d->bcarena;
    A.plan(d->bcnode, std::max<int64_t>(1, nbc));
    A.plan(d->bcdir, std::max<int64_t>(1, nbc));
    A.plan(d->bcsymp, nbc + 1);
    A.plan(d->symn, symn.size());
    A.plan(d->dirmask, std::max<int64_t>(1, ndir) * 5);
    A.plan(d->dirval, std::max<int64_t>(1, ndir) * 5);
    if (pass == 0) XG_CUDA(c, A.reserve());
  }
  auto up = [&](void* dst, const void* src, size_t bytes) { return upload(c, dst, src, bytes); };
  XG_CUDA(c, up(d->bcnode, node.data(), nbc * 4));
  XG_CUDA(c, up(d->bcdir, dir.data(), nbc * 4));
  XG_CUDA(c, up(d->bcsymp, symp.data(), (nbc + 1) * 4));
  XG_CUDA(c, up(d->symn, symn.data(), symn.size() * 8));
  XG_CUDA(c, up(d->dirmask, dirmask, ndir * 5 * 4));
  XG_CUDA(c, up(d->dirval, dirvals, ndir * 5 * 8));
  XG_CUDA(c, up(d->bcof, bcof.data(), n * 4));
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  d->nbc = nbc;
  d->dt_valid = false;
  return XG_OK;
  XG_HOST_CATCH(c)
}

int xg_kozcg_set_state(xg_ctx* c, const double* U, double t) {
  int rc = use(c);
  if (rc) return rc;
  KozCGDev* d = c->kozcg;
  if (!d) return fail(c, XG_ERR_STATE, "kozcg_set_state before kozcg_setup");
  if (!U) return fail(c, XG_ERR_ARG, "kozcg_set_state: null U");
  XG_CUDA(c, cudaMemcpyAsync(d->stage, U, d->n * 5 * 8, cudaMemcpyHostToDevice, c->stream));
  k_aos_to_soa<<<blocks_for(d->n * 5, kBlock), kBlock, 0, c->stream>>>(d->n, 5, d->stage, d->U);
  XG_CHECK_LAUNCH(c);
  d->t = t;
  rc = refresh_dt(c, d);
  if (rc) return rc;
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  return XG_OK;
}

int xg_kozcg_get_state(xg_ctx* c, double* U, double* t) {
  int rc = use(c);
  if (rc) return rc;
  KozCGDev* d = c->kozcg;
  if (!d) return fail(c, XG_ERR_STATE, "kozcg_get_state before kozcg_setup");
  if (U) {
    k_soa_to_aos<<<blocks_for(d->n * 5, kBlock), kBlock, 0, c->stream>>>(d->n, 5, d->U, d->stage);
    XG_CHECK_LAUNCH(c);
    XG_CUDA(c, cudaMemcpyAsync(U, d->stage, d->n * 5 * 8, cudaMemcpyDeviceToHost, c->stream));
  }
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  if (t) *t = d->t;
  return XG_OK;
}

int xg_kozcg_rhs(xg_ctx* c, const double* U, double dt, double* R) {
  int rc = use(c);
  if (rc) return rc;
  KozCGDev* d = c->kozcg;
  if (!d) return fail(c, XG_ERR_STATE, "kozcg_rhs before kozcg_setup");
  if (!U || !R) return fail(c, XG_ERR_ARG, "kozcg_rhs: null array");
  cudaStream_t s = c->stream;
  // use A as scratch for the caller's state so the device state is untouched
  XG_CUDA(c, cudaMemcpyAsync(d->stage, U, d->n * 5 * 8, cudaMemcpyHostToDevice, s));
  k_aos_to_soa<<<blocks_for(d->n * 5, kBlock), kBlock, 0, s>>>(d->n, 5, d->stage, d->A);
  XG_CHECK_LAUNCH(c);
  k_set_step<<<1, 1, 0, s>>>(d->scal, d->t, dt);  // the sources at the context's time
  XG_CHECK_LAUNCH(c);
  if (d->prm.precision == XG_FP32_FLUX) {
    XG_CUDA(c, cudaMemsetAsync(d->R32, 0, d->n * kRP * 4, s));
    galerkin<float>(c, d, d->A, 0);
    k_rec_to_soa<<<blocks_for(d->n * 5, kBlock), kBlock, 0, s>>>(d->n, d->R32, d->R);
  } else {
    galerkin<double>(c, d, d->A, 0);
    k_node_rhs64<<<blocks_for(d->n, kBlock), kBlock, 0, s>>>(d->n, d->soff, d->sw, d->sslot, d->E,
                                                             d->R);
  }
  XG_CHECK_LAUNCH(c);
  k_soa_to_aos<<<blocks_for(d->n * 5, kBlock), kBlock, 0, s>>>(d->n, 5, d->R, d->stage);
  XG_CHECK_LAUNCH(c);
  XG_CUDA(c, cudaMemcpyAsync(R, d->stage, d->n * 5 * 8, cudaMemcpyDeviceToHost, s));
  XG_CUDA(c, cudaStreamSynchronize(s));
  d->dt_valid = false;
  return XG_OK;
}

int xg_kozcg_dt(xg_ctx* c, double* dt) {
  int rc = use(c);
  if (rc) return rc;
  KozCGDev* d = c->kozcg;
  if (!d) return fail(c, XG_ERR_STATE, "kozcg_dt before kozcg_setup");
  if (!dt) return fail(c, XG_ERR_ARG, "kozcg_dt: null dt");
  if (!d->dt_valid) {
    rc = refresh_dt(c, d);
    if (rc) return rc;
  }
  KScalars h;
  XG_CUDA(c, cudaMemcpyAsync(&h, d->scal, sizeof(h), cudaMemcpyDeviceToHost, c->stream));
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  double m;
  std::memcpy(&m, &h.dtmin, sizeof(double));
  *dt = std::fabs(d->prm.const_dt) > std::numeric_limits<double>::epsilon() ? d->prm.const_dt
                                                                             : m * d->prm.cfl;
  return XG_OK;
}

int xg_kozcg_bc(xg_ctx* c) {
  int rc = use(c);
  if (rc) return rc;
  KozCGDev* d = c->kozcg;
  if (!d) return fail(c, XG_ERR_STATE, "kozcg_bc before kozcg_setup");
  if (d->nbc) {
    k_bc<<<blocks_for(d->nbc, kBlock), kBlock, 0, c->stream>>>(d->n, kbc_of(d), d->U, d->t);
    XG_CHECK_LAUNCH(c);
  }
  rc = refresh_dt(c, d);
  if (rc) return rc;
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  return XG_OK;
}

int xg_kozcg_run(xg_ctx* c, int64_t nstep, double* dts, float* ms) {
  int rc = use(c);
  if (rc) return rc;
  KozCGDev* d = c->kozcg;
  if (!d) return fail(c, XG_ERR_STATE, "kozcg_run before kozcg_setup");
  if (nstep < 0) return fail(c, XG_ERR_ARG, "kozcg_run: negative step count");
  if (nstep == 0) {
    if (ms) *ms = 0.f;
    return XG_OK;
  }
  if (!d->dt_valid) {
    rc = refresh_dt(c, d);
    if (rc) return rc;
  }
  if (d->dthist_cap < nstep) {
    XG_CUDA(c, cudaStreamSynchronize(c->stream));
    if (d->dthist) cudaFree(d->dthist);
    d->dthist = nullptr;
    XG_CUDA(c, cudaMalloc(&d->dthist, nstep * sizeof(double)));
    d->dthist_cap = nstep;
  }
  k_set_time<<<1, 1, 0, c->stream>>>(d->scal, d->t);
  XG_CHECK_LAUNCH(c);
  cudaEvent_t e0, e1;
  XG_CUDA(c, cudaEventCreate(&e0));
  XG_CUDA(c, cudaEventCreate(&e1));
  XG_CUDA(c, cudaEventRecord(e0, c->stream));
  for (int64_t k = 0; k < nstep; ++k) {
    k_step_begin<<<1, 1, 0, c->stream>>>(d->scal, d->prm.cfl, d->prm.const_dt, d->dthist, k);
    XG_CHECK_LAUNCH(c);
    rc = step(c, d);
    if (rc) return rc;
  }
  XG_CUDA(c, cudaEventRecord(e1, c->stream));
  XG_CUDA(c, cudaEventSynchronize(e1));
  float el = 0.f;
  XG_CUDA(c, cudaEventElapsedTime(&el, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (ms) *ms = el;
  std::vector<double> h(nstep);
  XG_CUDA(c, cudaMemcpy(h.data(), d->dthist, nstep * 8, cudaMemcpyDeviceToHost));
  for (double v : h) d->t += v;
  if (dts) std::memcpy(dts, h.data(), nstep * 8);
  d->dt_valid = true;
  KScalars s;
  XG_CUDA(c, cudaMemcpy(&s, d->scal, sizeof(s), cudaMemcpyDeviceToHost));
  if (s.blowup) return fail(c, XG_ERR_BLOWUP, "dt below machine epsilon");
  return XG_OK;
}

int xg_kozcg_step(xg_ctx* c, double dt) {
  int rc = use(c);
  if (rc) return rc;
  KozCGDev* d = c->kozcg;
  if (!d) return fail(c, XG_ERR_STATE, "kozcg_step before kozcg_setup");
  if (!(dt > 0.0) || !std::isfinite(dt)) return fail(c, XG_ERR_ARG, "kozcg_step: dt must be > 0");
  k_set_step<<<1, 1, 0, c->stream>>>(d->scal, d->t, dt);
  XG_CHECK_LAUNCH(c);
  rc = step(c, d);
  if (rc) return rc;
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  d->t += dt;
  d->dt_valid = true;  // the step's solve formed the next CFL minimum
  return XG_OK;
}

int xg_kozcg_set_source(xg_ctx* c, int problem, const double* prm) {
  int rc = use(c);
  if (rc) return rc;
  KozCGDev* d = c->kozcg;
  if (!d) return fail(c, XG_ERR_STATE, "kozcg_set_source before kozcg_setup");
  if (problem < XG_SRC_NONE || problem > XG_SRC_RAYLEIGH_TAYLOR)
    return fail(c, XG_ERR_ARG, "kozcg_set_source: unknown problem");
  if (problem != XG_SRC_NONE && problem != XG_SRC_TAYLOR_GREEN && !prm)
    return fail(c, XG_ERR_ARG, "kozcg_set_source: this problem needs its parameters");
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  if (problem != XG_SRC_NONE && !d->S) {
    XG_CUDA(c, cudaMalloc(&d->S, d->n * 5 * sizeof(double)));
    XG_CUDA(c, cudaMalloc(&d->Se, std::max<int64_t>(1, d->ne) * 5 * sizeof(double)));
  }
  d->src.problem = problem;
  for (int k = 0; k < 8; ++k) d->src.p[k] = prm ? prm[k] : 0.0;
  d->src.gamma = d->prm.gamma;
  return XG_OK;
}

}  // extern "C"
