// Sparse matrix and preconditioned conjugate gradients on one GB300.
//
// Reference path (paths relative to the reference project root):
//   tk::CSR                         src/LinearSolver/CSR.{hpp,cpp}
//   CSR::mult                       src/LinearSolver/CSR.cpp:154-172
//   CSR::dirichlet                  src/LinearSolver/CSR.cpp:106-152
//   ConjugateGradients::init/apply/r/setup/next/qAp/q/pq/rz/x
//                                   src/LinearSolver/ConjugateGradients.cpp:105-823
//
// Layout: the matrix is stored as SELL-32 (slices of 32 rows, each padded to
// the slice's longest row; entry k of row i at off[s] + k*32 + lane) with
// int32 columns and FP64 values.  Dirichlet elimination never rewrites the
// host matrix: a device pass builds the working values from the original
// ones and the Dirichlet mask, which is what the reference's sequential
// elimination produces (rows and columns of Dirichlet nodes zeroed, 1 on
// their diagonal), and the right-hand side correction sum_i a_ji * val_i is
// summed per row in the reference's order (decreasing node id).
//
// One PCG iteration (the reference's FP64 algorithm) runs inside k_cg_loop,
// one cooperative launch for the whole solve, where the rows fit the SMs'
// shared memory (924,160 rows on 152 of them) and no factor is applied.  Otherwise it
// is three kernels:
//   k_cg_p: p = z + beta p (beta = rho/rho0)
//   k_cg_a: q = A p, partial (p, q)
//   k_cg_b: alpha = rho/(p,q); r -= alpha q; x += alpha p; z = r/d (Jacobi,
//           as r times the stored inverse diagonal);
//           partial (r,z), (r,r); convergence test
// plus, for the factored preconditioner (pc 2, no reference counterpart),
// z = -S (I+N)(I+N)^T S r in two passes over the lower and upper triangles.
// GB300 runs FP64 arithmetic at a small fraction of its FP32 rate, so the
// FP64 kernels keep FP64 operations per row to what the algorithm needs
// (p is formed once per row, scalar divisions once per block).
// Kernels loop over rows with a grid of one wave of resident blocks, so a
// reduction has one partial per block; the last block to finish (an atomic
// ticket, no spinning) adds them in block order, so every reduction is
// deterministic.  Kernels return at once when the solve is done, so the host
// launches iterations in batches and reads the done flag once per batch.
//
// Mixed precision (xg_cg_solve_mixed): the same iteration in FP32 on an FP32
// copy of the working matrix, its columns stored as 16-bit offsets from the
// row (when every |j - i| < 32768) and the factor values in FP16, with FP64
// dot products and reliable updates: the FP32 correction e = sum alpha p' is
// folded into the FP64 x and the FP32 residual replaced by the true FP64
// residual b - A x whenever the recursive residual has fallen by the factor
// `inner_tol` since the last replacement.  The search direction is kept
// across replacements, so the FP32 iteration follows the FP64 one instead of
// restarting.
//
// Whole solves run in one launch: k_cg_cluster (FP64, systems that fit the
// shared memory of 16 SMs), k_cg_loop (FP64, up to 924,160 rows) and
// k_mixed_loop (the FP32 iterations up to the next residual replacement); the
// FP64 factored solve and larger FP64 systems take a launch per pass.

#include <cuda_fp16.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <limits>
#include <vector>

#include "xg_internal.hpp"

namespace xg {

namespace {
constexpr int kSlice = 32;
constexpr int32_t kPad = -1;
constexpr int16_t kPad16 = std::numeric_limits<int16_t>::min();
constexpr int kBlock = 256;
constexpr int kBatch = 16;
constexpr int kLoopThreads = 1024;  // the whole-solve kernel k_cg_loop: one block per SM
constexpr int kLoopRound = 8;       // its entries in flight per row

struct CGScalars {
  double rho, rho0, pq, alpha, rr, normb, tol, delta, rlast;
  double pad0;
  int64_t it, maxit;
  int32_t done, finished, converged, pc;
  int32_t guard, pad1;  // 0: |(p,q)| < DBL_EPSILON ends the solve; 1: underflow only
  unsigned int ticket[4];
  int32_t err, pad2;  // k_cg_loop: a wait for the other blocks ran out
};


}  // namespace

struct CGDev {
  Arena arena;
  int64_t n = 0, nslice = 0, nent = 0, maxgrid = 0;
  int wmax = 0;  // the widest slice
  int32_t *soff = nullptr, *swidth = nullptr, *col = nullptr;
  int16_t* col16 = nullptr;            // column - row, kPad16 for padding
  double* a0 = nullptr;                // original values (SELL order)
  double* a = nullptr;                 // working values (after Dirichlet elimination)
  float* a32 = nullptr;
  float* rs32 = nullptr;               // per row: exact (FP64) working row sum, in FP32
  int32_t* diagpos = nullptr;          // SELL index of each row's diagonal
  uint8_t* bcmask = nullptr;
  double* bcval = nullptr;
  double *x = nullptr, *b = nullptr, *r = nullptr, *q = nullptr, *z = nullptr, *d = nullptr;
  double* p[2] = {nullptr, nullptr};
  float *r32 = nullptr, *q32 = nullptr, *z32 = nullptr, *d32 = nullptr;
  double* e64 = nullptr;  // the mixed solve's correction sum alpha p', accumulated in FP64
  float* p32 = nullptr;
  float2 *zp32 = nullptr, *vt32 = nullptr;  // records of the mixed iteration: (z, p), (S r, S q)
  double* partial = nullptr;  // 3 * maxgrid
  CGScalars* scal = nullptr;
  double* lpart = nullptr;         // k_cg_loop: [3 barriers of an iteration][2 sums][SMs]
  unsigned int* larrive = nullptr;  // and its arrival count
  bool apply = false;
  bool ready = false;
  bool use16 = false;  // every |j - i| fits a 16-bit offset
  int pc = 1;
  int64_t last_it = 0;
  double last_normr = 0, last_normb = 0;
  int last_conv = 0;
  // factored approximate inverse M^-1 = -S (I+N)(I+N)^T S (pc 2): lower and
  // upper triangles of the matrix graph as SELL-32, the factor values (FP32,
  // and FP16 for the mixed solver), the row scales s = 1/sqrt|a_ii| and the
  // normalised couplings e_ij = a_ij s_i s_j
  int64_t nentL = 0, nentU = 0;
  int32_t *soffL = nullptr, *swL = nullptr, *colL = nullptr, *posL = nullptr, *tposU = nullptr;
  int32_t *soffU = nullptr, *swU = nullptr, *colU = nullptr;
  int16_t *colL16 = nullptr, *colU16 = nullptr;
  float *nvL = nullptr, *nvU = nullptr, *srow = nullptr, *msrow = nullptr;
  float *eL = nullptr, *eU = nullptr;
  __half *hvL = nullptr, *hvU = nullptr;
  float* eF = nullptr;  // e_ij in the full layout (0 on the diagonal and at Dirichlet nodes)
  double *v = nullptr, *u = nullptr, *t = nullptr;  // S r, (I+N)^T S r; t: xg_cg_precondition
  float *v32 = nullptr, *u32 = nullptr;
  bool geom_set = false;
  bool factor_set = false;
  uint64_t bc_key = 0;  // hash of the Dirichlet mask the geometry was built for
  int guard = 0;        // breakdown guard of the FP64 solver (xg_cg_set_guard)
  int64_t launch_its = 0;  // iterations per launch (xg_cg_set_launch_limit), 0: the kernels' own
  xg_lpc* factor_model = nullptr;  // network emitting N, or null: N = factor_c * e
  double factor_c = 1.0;
};

void destroy_cg(CGDev* d) { delete d; }
size_t bytes_cg(const CGDev* d) { return d ? d->arena.bytes() : 0; }

namespace {

// ---------------------------------------------------------------- reductions

// Sum of one value per thread into partial[k * gridDim.x + blockIdx.x];
// returns true in the block that completes last (its threads then see every
// partial).  The warp sums run in A (FP32 for the FP32 solver, whose values
// are FP32: FP64 shuffles and adds per thread load GB300's narrow FP64
// pipe); the warp totals are summed in FP64.
template <int K, class A>
__device__ __forceinline__ bool block_partials(const A (&v)[K], double* partial,
                                               unsigned int* ticket) {
  __shared__ double sm[K][32];
  __shared__ bool last;
  A s[K];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    s[k] = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], o);
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0)
#pragma unroll
    for (int k = 0; k < K; ++k) sm[k][wid] = double(s[k]);
  __syncthreads();
  if (threadIdx.x == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    for (int k = 0; k < K; ++k) {
      double t = 0.0;
      for (int w = 0; w < nw; ++w) t += sm[k][w];
      partial[k * gridDim.x + blockIdx.x] = t;
    }
    __threadfence();
    unsigned int prev = atomicAdd(ticket, 1u);
    last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  return last;
}

// In the last block: deterministic sum of the partials of component k, four
// independent lane-strided chains, then a fixed-order tree.
__device__ double sum_partials(const double* partial, int k) {
  __shared__ double red[kBlock];
  __threadfence();
  const int64_t nb = gridDim.x;
  const double* base = partial + k * nb;
  double t0 = 0.0, t1 = 0.0, t2 = 0.0, t3 = 0.0;
  int64_t i = threadIdx.x;
  for (; i + 3 * kBlock < nb; i += 4 * kBlock) {
    t0 += __ldcg(base + i);
    t1 += __ldcg(base + i + kBlock);
    t2 += __ldcg(base + i + 2 * kBlock);
    t3 += __ldcg(base + i + 3 * kBlock);
  }
  for (; i < nb; i += kBlock) t0 += __ldcg(base + i);
  red[threadIdx.x] = (t0 + t1) + (t2 + t3);
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
    __syncthreads();
  }
  double r = red[0];
  __syncthreads();
  return r;
}

// ---------------------------------------------------------------- row access

// Column of SELL entry e of row i (or -1 for padding), from int32 columns or
// 16-bit offsets.  The int32 columns and FP64 values (the FP64 solver's
// matrix stream, larger than L2) are read with the evict-first hint so that
// the gathered vectors stay in L2; the FP32 solver's narrower stream is read
// through the non-coherent cache (measured faster for it).
struct Cols32 {
  using E = int32_t;
  const int32_t* c;
  __device__ __forceinline__ static int32_t of(int32_t v, int32_t) { return v; }
  __device__ __forceinline__ int32_t at(int32_t e, int32_t) const { return __ldcs(c + e); }
};
struct Cols16 {
  using E = int16_t;
  const int16_t* c;
  __device__ __forceinline__ static int32_t of(int16_t v, int32_t i) {
    return v == kPad16 ? -1 : i + int32_t(v);
  }
  __device__ __forceinline__ int32_t at(int32_t e, int32_t i) const {
    const int16_t dlt = __ldg(c + e);
    return dlt == kPad16 ? -1 : i + int32_t(dlt);
  }
};

__device__ __forceinline__ float ldv(const __half* p) { return __half2float(p[0]); }
__device__ __forceinline__ float ldv(const float* p) { return __ldg(p); }
__device__ __forceinline__ double ldv(const double* p) { return __ldcs(p); }

// sum_k val[e_k] * g(col[e_k]) over row i of a SELL-32 layout, in entry
// order, issued in groups of U entries so that U column / value loads and
// then U gathers are in flight at once (padding reads the row's own entry
// with weight 0).
template <int U, class T, class CI, class V, class G>
__device__ __forceinline__ T sell_row(CI ci, const V* __restrict__ val, int32_t off, int w,
                                      int lane, int32_t i, G g) {
  T s = T(0);
  int k = 0;
  for (; k + U <= w; k += U) {
    int32_t cc[U];
    T vv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int32_t e = off + (k + u) * kSlice + lane;
      const int32_t c = ci.at(e, i);
      vv[u] = c < 0 ? T(0) : T(ldv(val + e));
      cc[u] = c < 0 ? i : c;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) s += vv[u] * g(cc[u]);
  }
  for (; k < w; ++k) {
    const int32_t e = off + k * kSlice + lane;
    const int32_t c = ci.at(e, i);
    if (c >= 0) s += T(ldv(val + e)) * g(c);
  }
  return s;
}

// The same sum with each round fully unrolled to the exact number of entries
// left (at most XM): a row of w <= XM entries is one round, its column /
// value loads and then its gathers all in flight at once, with no predicated
// or sequential tail (the slice width is uniform across the warp, so the
// dispatch does not diverge).  Wider rows take rounds of XM.  XM bounds the
// registers of the kernel: 16 for whole rows (15 entries on a tetrahedral
// mesh of a cube), 8 for the strict triangles (7).

template <int W, class T, class CI, class V, class G>
__device__ __forceinline__ T sell_fixed(CI ci, const V* __restrict__ val, int32_t off, int lane,
                                        int32_t i, G g, T s) {
  int32_t cc[W];
  T vv[W];
#pragma unroll
  for (int u = 0; u < W; ++u) {
    const int32_t e = off + u * kSlice + lane;
    const int32_t c = ci.at(e, i);
    vv[u] = c < 0 ? T(0) : T(ldv(val + e));
    cc[u] = c < 0 ? i : c;
  }
#pragma unroll
  for (int u = 0; u < W; ++u) s += vv[u] * g(cc[u]);
  return s;
}

template <int W, int XM, class T, class CI, class V, class G>
__device__ __forceinline__ T sell_tail(int r, CI ci, const V* __restrict__ val, int32_t off,
                                       int lane, int32_t i, G g, T s) {
  if constexpr (W <= XM) {
    if (r == W) return sell_fixed<W, T>(ci, val, off, lane, i, g, s);
    return sell_tail<W + 1, XM, T>(r, ci, val, off, lane, i, g, s);
  } else {
    return s;
  }
}

template <class T, int XM = 16, class CI, class V, class G>
__device__ __forceinline__ T sell_row_x(CI ci, const V* __restrict__ val, int32_t off, int w,
                                        int lane, int32_t i, G g) {
  T s = T(0);
  int k = 0;
  for (; w - k > XM; k += XM) s = sell_fixed<XM, T>(ci, val, off + k * kSlice, lane, i, g, s);
  if (w > k) s = sell_tail<1, XM, T>(w - k, ci, val, off + k * kSlice, lane, i, g, s);
  return s;
}

// One wave of resident blocks of kernel K for n rows (blocks per SM: the same on
// every sm_103a device).
template <auto K>
unsigned pgrid(const xg_ctx* c, int64_t n) {
  static const int per_sm = [] {
    int v = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, K, kBlock, 0) != cudaSuccess) v = 1;
    return v < 1 ? 1 : v;
  }();
  const int64_t want = (n + kBlock - 1) / kBlock;
  return static_cast<unsigned>(
      std::max<int64_t>(1, std::min<int64_t>(want, int64_t(per_sm) * c->nsm)));
}

#define XG_ROWS(i, n) \
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < (n); \
       i += int64_t(gridDim.x) * blockDim.x)

// ---------------------------------------------------------------- launches

// The iteration kernels are launched as programmatic dependents of the
// kernel before them in the stream: their blocks may be scheduled while that
// kernel drains (its blocks trigger after their row loop, before the
// reduction tail) and wait in griddep_wait() until it has completed and its
// writes are visible.  Every kernel launched with launch_dep() calls
// griddep_wait() before it reads anything.
__device__ __forceinline__ void griddep_wait() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
}
__device__ __forceinline__ void griddep_trigger() {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

template <class... P, class... A>
void launch_dep_k(void (*k)(P...), unsigned grid, cudaStream_t s, A&&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(kBlock);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  (void)cudaLaunchKernelEx(&cfg, k, std::forward<A>(args)...);  // errors: cudaGetLastError
}

// Kernel K over n rows, one wave of resident blocks, as a dependent launch.
template <auto K, class... A>
void launch_dep(const xg_ctx* c, int64_t n, A&&... args) {
  launch_dep_k(K, pgrid<K>(c, n), c->stream, std::forward<A>(args)...);
}

// ---------------------------------------------------------------- kernels

// CSR::mult on the original values: y = A x.
__global__ void __launch_bounds__(kBlock) k_spmv(int64_t n, const int32_t* __restrict__ soff,
                                                 const int32_t* __restrict__ sw,
                                                 const int32_t* __restrict__ col,
                                                 const double* __restrict__ a,
                                                 const double* __restrict__ x,
                                                 double* __restrict__ y) {
  XG_ROWS(i, n) {
    const int lane = int(i & 31);
    y[i] = sell_row_x<double>(Cols32{col}, a, soff[i >> 5], sw[i >> 5], lane, int32_t(i),
                               [&](int32_t c) { return __ldg(x + c); });
  }
}

// Working values from the original ones and the Dirichlet mask; the
// right-hand-side correction of every non-Dirichlet row (sum over its
// Dirichlet columns in decreasing column order, CSR.cpp:130-138 as driven by
// ConjugateGradients.cpp:475-485); Dirichlet rows of b take their values
// (ConjugateGradients.cpp:542-552); Neumann contributions are added first
// (ConjugateGradients.cpp:472-473).
__global__ void k_apply_bc(int64_t n, const int32_t* __restrict__ soff,
                           const int32_t* __restrict__ sw, const int32_t* __restrict__ col,
                           const double* __restrict__ a0, double* __restrict__ a,
                           float* __restrict__ a32, const uint8_t* __restrict__ mask,
                           const double* __restrict__ val, const double* __restrict__ neu,
                           double* __restrict__ b) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const int lane = int(i & 31);
  const int32_t off = soff[i >> 5], w = sw[i >> 5];
  const bool rowbc = mask[i] != 0;
  double corr = 0.0;
  for (int k = w - 1; k >= 0; --k) {
    const int32_t e = off + k * kSlice + lane;
    const int32_t c = col[e];
    if (c < 0) continue;
    double v = a0[e];
    double nv;
    if (rowbc) {
      nv = (c == i) ? 1.0 : 0.0;
    } else if (mask[c]) {
      corr += v * val[c];
      nv = 0.0;
    } else {
      nv = v;
    }
    a[e] = nv;
    a32[e] = float(nv);
  }
  double bi = b[i] + (neu ? neu[i] : 0.0);
  bi -= corr;
  if (rowbc) bi = val[i];
  b[i] = bi;
}

// rs_i = sum_j a_ij of the working matrix (FP64), stored in FP32.
__global__ void k_row_sums(int64_t n, const int32_t* __restrict__ soff,
                           const int32_t* __restrict__ sw, const int32_t* __restrict__ col,
                           const double* __restrict__ a, float* __restrict__ rs) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const int lane = int(i & 31);
  const int32_t off = soff[i >> 5], w = sw[i >> 5];
  double sum = 0.0;
  for (int k = 0; k < w; ++k) {
    const int32_t e = off + k * kSlice + lane;
    if (col[e] >= 0) sum += a[e];
  }
  rs[i] = float(sum);
}

__global__ void k_copy_values(int64_t nent, const double* __restrict__ a0, double* __restrict__ a,
                              float* __restrict__ a32) {
  int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (e >= nent) return;
  a[e] = a0[e];
  a32[e] = float(a0[e]);
}

// ConjugateGradients::setup + pc + initres (ConjugateGradients.cpp:105-319):
// r = b - A x, d = 1/diag(A) (Jacobi) or 1 (none, factor), z = r d, p = r,
// partials of (b,b) and (r,z).
__global__ void __launch_bounds__(kBlock) k_setup(int64_t n, const int32_t* __restrict__ soff,
                                                   const int32_t* __restrict__ sw,
                                                   const int32_t* __restrict__ col,
                                                   const double* __restrict__ a,
                                                   const int32_t* __restrict__ diagpos,
                                                   const double* __restrict__ x,
                                                   const double* __restrict__ b,
                                                   double* __restrict__ r, double* __restrict__ d,
                                                   double* __restrict__ z, double* __restrict__ p,
                                                   float* __restrict__ d32, double* partial,
                                                   CGScalars* sc) {
  double v[2] = {0.0, 0.0};
  const int pc = sc->pc;
  XG_ROWS(i, n) {
    const int lane = int(i & 31);
    const double s = sell_row_x<double>(Cols32{col}, a, soff[i >> 5], sw[i >> 5], lane,
                                         int32_t(i), [&](int32_t c) { return x[c]; });
    const double ri = b[i] - s;
    // the inverse Jacobi diagonal: one multiply per row and iteration in
    // place of an FP64 division (the slow FP64 pipe of this GPU)
    const double di = pc == 1 ? 1.0 / a[diagpos[i]] : 1.0;
    r[i] = ri;
    d[i] = di;
    d32[i] = float(di);
    const double zi = ri * di;
    z[i] = zi;
    p[i] = ri;
    v[0] += b[i] * b[i];
    v[1] += ri * zi;
  }
  if (block_partials<2>(v, partial, &sc->ticket[0])) {
    double bb = sum_partials(partial, 0);
    double rz = sum_partials(partial, 1);
    if (threadIdx.x == 0) {
      sc->normb = sqrt(bb);
      sc->rho = rz;
      sc->it = 0;
      sc->done = 0;
      sc->finished = 0;
      sc->converged = 0;
      sc->ticket[0] = 0;
    }
  }
}

// next + qAp + q (ConjugateGradients.cpp:584-669): p' = z + beta p,
// q = A p', partial (p', q); the last block sets alpha = rho / (p', q).
// T is the vector type, V the matrix value type, CI the column encoding.
//
// beta = rho/rho0 (0 in the first iteration), formed once per block: an FP64
// division per thread would load GB300's narrow FP64 pipe.
template <class T>
__device__ __forceinline__ T block_beta(const CGScalars* sc) {
  __shared__ T beta_s;
  if (threadIdx.x == 0) beta_s = sc->it == 0 ? T(0) : T(sc->rho / sc->rho0);
  __syncthreads();
  return beta_s;
}

// p = z + beta p in place (the FP64 solver; its SpMV then gathers p alone,
// with half the FP64 operations of forming p per gathered entry).
template <class T>
__global__ void __launch_bounds__(kBlock) k_cg_p(int64_t n, const T* __restrict__ z,
                                                  T* __restrict__ p, const CGScalars* sc) {
  griddep_wait();
  if (sc->done) return;
  const T beta = block_beta<T>(sc);
  XG_ROWS(i, n) p[i] = z[i] + beta * p[i];
  griddep_trigger();
}

// q = A p, (p, q).
template <class T, class V, class CI>
__global__ void __launch_bounds__(kBlock) k_cg_a(int64_t n, const int32_t* __restrict__ soff,
                                                  const int32_t* __restrict__ sw, CI ci,
                                                  const V* __restrict__ a,
                                                  const T* __restrict__ p, T* __restrict__ q,
                                                  double* partial, CGScalars* sc) {
  griddep_wait();
  if (sc->done) return;
  T dot = T(0);
  XG_ROWS(i, n) {
    const T s = sell_row_x<T>(ci, a, soff[i >> 5], sw[i >> 5], int(i & 31), int32_t(i),
                               [&](int32_t c) { return __ldg(p + c); });
    q[i] = s;
    dot += p[i] * s;
  }
  griddep_trigger();
  T v[1] = {dot};
  if (block_partials<1>(v, partial, &sc->ticket[1])) {
    double pq = sum_partials(partial, 0);
    if (threadIdx.x == 0) {
      sc->rho0 = sc->rho;
      sc->pq = pq;
      // the reference's breakdown guard is an absolute epsilon
      // (ConjugateGradients.cpp:681-690); with guard 1, underflow only
      const double eps = sc->guard == 0 ? DBL_EPSILON : DBL_MIN;
      if (fabs(pq) < eps) {
        sc->finished = 1;
        sc->alpha = 0.0;
      } else {
        sc->alpha = sc->rho / pq;
      }
      sc->ticket[1] = 0;
    }
  }
}

// The end of an iteration, in the last block: (r,r), the count and the
// stopping test: ||r|| < tol ||b||, or maxit iterations
// (ConjugateGradients.cpp:772-823).
__device__ __forceinline__ void end_iteration(double rr, CGScalars* sc) {
  sc->rr = rr;
  sc->it += 1;
  const double nr = sqrt(rr);
  const double nb = sc->normb > 1.0e-14 ? sc->normb : 1.0;
  if (sc->finished || nr < sc->tol * nb || sc->it >= sc->maxit) {
    sc->done = 1;
    sc->converged = nr > sc->tol * nb ? 0 : 1;
  }
}

// pq + rz + x (ConjugateGradients.cpp:671-823), fused: r -= alpha q,
// x += alpha p; Jacobi z = r d (d the inverse diagonal), rho = (r, z), (r, r)
// and the stopping test, or (FACTOR) v = S r for the factor passes that follow.
template <class T, bool FACTOR>
__global__ void __launch_bounds__(kBlock) k_cg_b(int64_t n, const T* __restrict__ q,
                                                  const T* __restrict__ d,
                                                  const T* __restrict__ p,
                                                  const float* __restrict__ srow,
                                                  T* __restrict__ r, T* __restrict__ z,
                                                  T* __restrict__ vs, T* __restrict__ x,
                                                  double* partial, CGScalars* sc) {
  griddep_wait();
  if (sc->done) return;
  const T alpha = T(sc->alpha);
  if (FACTOR) {
    // no reduction here: (r,z), (r,r) and the stopping test close the
    // iteration in k_pc_lower
    XG_ROWS(i, n) {
      const T ri = r[i] - alpha * q[i];
      r[i] = ri;
      x[i] += alpha * p[i];
      vs[i] = T(srow[i]) * ri;
    }
    griddep_trigger();
    return;
  }
  T rz = T(0), rr = T(0);  // per thread in T, widened in block_partials
  XG_ROWS(i, n) {
    const T ri = r[i] - alpha * q[i];
    r[i] = ri;
    x[i] += alpha * p[i];
    const T zi = ri * d[i];
    z[i] = zi;
    rz += ri * zi;
    rr += ri * ri;
  }
  griddep_trigger();
  const T v[2] = {rz, rr};
  if (block_partials<2>(v, partial, &sc->ticket[2])) {
    double rz = sum_partials(partial, 0);
    double rr = sum_partials(partial, 1);
    if (threadIdx.x == 0) {
      sc->rho = rz;
      end_iteration(rr, sc);
      sc->ticket[2] = 0;
    }
  }
}

// ---- factored approximate inverse (pc 2)

// u = (I+N)^T v: u_i = v_i + sum_{j>i} N_ji v_j (upper layout of N).
template <class T, class V, class CI>
__global__ void __launch_bounds__(kBlock) k_pc_upper(int64_t n, const int32_t* __restrict__ soffU,
                                                      const int32_t* __restrict__ swU, CI ci,
                                                      const V* __restrict__ nvU,
                                                      const T* __restrict__ vs,
                                                      T* __restrict__ u,
                                                      const CGScalars* __restrict__ sc) {
  griddep_wait();
  if (sc->done) return;
  XG_ROWS(i, n) {
    const int lane = int(i & 31);
    u[i] = vs[i] + sell_row_x<T, 8>(ci, nvU, soffU[i >> 5], swU[i >> 5], lane, int32_t(i),
                                  [&](int32_t c) { return __ldg(vs + c); });
  }
}

// z = -S (I+N) u (Dirichlet rows: z = r), partial (r,z); the last block
// stores rho = (r,z).  MODE 0 applies the preconditioner only; MODE 1 also
// closes a CG iteration: partial (r,r), the count and the stopping test.
template <class T, class V, class CI, int MODE>
__global__ void __launch_bounds__(kBlock, sizeof(T) == 4 ? 6 : 1) k_pc_lower(int64_t n, const int32_t* __restrict__ soffL,
                                                      const int32_t* __restrict__ swL, CI ci,
                                                      const V* __restrict__ nvL,
                                                      const float* __restrict__ srow,
                                                      const uint8_t* __restrict__ mask,
                                                      const T* __restrict__ u,
                                                      const T* __restrict__ r,
                                                      T* __restrict__ z, double* partial,
                                                      CGScalars* sc) {
  griddep_wait();
  if (sc->done) return;
  T rz = T(0), rr = T(0);  // per thread in T (FP32 for the mixed solver), widened once
  XG_ROWS(i, n) {
    const int lane = int(i & 31);
    const T acc = u[i] + sell_row_x<T, 8>(ci, nvL, soffL[i >> 5], swL[i >> 5], lane, int32_t(i),
                                        [&](int32_t c) { return __ldg(u + c); });
    const T ri = r[i];
    const T zi = mask[i] ? ri : -T(srow[i]) * acc;
    z[i] = zi;
    rz += ri * zi;
    if (MODE > 0) rr += ri * ri;
  }
  griddep_trigger();
  T v[2] = {rz, rr};
  if (MODE == 0) {
    T w[1] = {v[0]};
    if (block_partials<1>(w, partial, &sc->ticket[3])) {
      double rz = sum_partials(partial, 0);
      if (threadIdx.x == 0) {
        sc->rho = rz;
        sc->ticket[3] = 0;
      }
    }
  } else if (block_partials<2>(v, partial, &sc->ticket[3])) {
    double rz = sum_partials(partial, 0);
    double rr = sum_partials(partial, 1);
    if (threadIdx.x == 0) {
      sc->rho = rz;
      end_iteration(rr, sc);
      sc->ticket[3] = 0;
    }
  }
}

// ---- the FP64 iteration as one kernel

// Polls of the arrival count before a wait gives up (about a second).
constexpr int kLoopSpin = 1 << 20;

// The blocks' meeting points in k_cg_loop.
struct LoopSync {
  double* part;          // [3][2][blocks]
  unsigned int* arrive;  // arrivals since the launch
  unsigned int target;   // arrivals when every block has reached this barrier
  int turn;              // barriers so far, modulo 3
};

// The second half of a barrier: warp k < K (at least warp 0) comes with the
// block's sum of value k in lane 0 of `s`.
template <int K, class F>
__device__ __forceinline__ bool grid_meet(double s, LoopSync& sync, CGScalars* sc, int* okay,
                                          F fin) {
  constexpr int KW = K > 0 ? K : 1;  // polling warps
  const int nb = gridDim.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  sync.target += unsigned(nb) * KW;
  if (wid < KW) {
    double* part = sync.part + (sync.turn * 2 + wid) * nb;
    if (K > 0 && lane == 0) part[blockIdx.x] = s;
    if (lane == 0) {
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(sync.arrive) : "memory");
      unsigned int seen = 0;
      int spin = 0;
      do {
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];"
                     : "=r"(seen)
                     : "l"(sync.arrive)
                     : "memory");
      } while (int(seen - sync.target) < 0 && ++spin < kLoopSpin);
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      if (spin >= kLoopSpin) {
        *okay = 0;
        atomicExch(&sc->err, 1);
      }
    }
    __syncwarp();
    if (K > 0) {
      // up to 256 blocks' sums in one round of loads
      double sum = 0.0, at[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) at[j] = lane + 32 * j < nb ? __ldcg(part + lane + 32 * j) : 0.0;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (32 * j < nb) sum += at[j];
      for (int b = lane + 256; b < nb; b += 32) sum += __ldcg(part + b);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) fin(wid, sum);
    }
  }
  sync.turn = sync.turn == 2 ? 0 : sync.turn + 1;
  __syncthreads();
  return *okay != 0;
}

// Barrier of all blocks of k_cg_loop that also sums K values per thread over
// the grid (K = 0: the barrier alone; the threads from `active` on hold 0);
// lane 0 of warp k calls fin(k, sum) with the total of value k before the
// block goes on.  Everything the grid wrote
// before the barrier is visible after it.
//
// An FP64 instruction holds its SM quarter's FP64 unit for 64 cycles on
// GB300, whatever the number of lanes, so the block's sums are formed with as
// few warp instructions as a tree allows: through shared memory, one warp of
// each quarter adds a quarter of the rows, then one warp per value the rest
// (11 in sequence; shuffles in each of 32 warps would take 40 per quarter).
// Each value's warp leaves the block's sum in global memory and counts
// itself in; one counter polled by lane 0 meets in 1.3 us on 152 SMs, where
// every block polling every block's slot took 4.7 us.  The warp then adds all
// blocks' sums in block order, so every block holds the same bits.  The sums
// alternate between three arrays: a block passes a barrier only after every
// block has arrived, so it may be one barrier ahead of the slowest reader
// and never overwrites what is still to be read.  False in every thread of the
// block when a wait ran out.
template <int K, class F>
__device__ __forceinline__ bool grid_sum(const double (&v)[K > 0 ? K : 1], int active,
                                         LoopSync& sync, CGScalars* sc, F fin) {
  constexpr int KW = K > 0 ? K : 1;          // values, at least one
  constexpr int NW = kLoopThreads / 32 / 4;  // rows of each quarter's warp
  __shared__ double rows[KW][kLoopThreads];
  __shared__ double quarter[KW][4][32];
  __shared__ int okay;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) okay = 1;
  if (K > 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) rows[k][threadIdx.x] = v[k];
    __syncthreads();
    if (wid < 4 * K) {
      const int k = wid >> 2, qd = wid & 3;
      double s = 0.0;
#pragma unroll
      for (int j = 0; j < NW; ++j)
        if (32 * (qd + 4 * j) < active) s += rows[k][lane + 32 * (qd + 4 * j)];
      quarter[k][qd][lane] = s;
    }
  }
  __syncthreads();
  double s = 0.0;
  if (K > 0 && wid < KW) {
    s = (quarter[wid][0][lane] + quarter[wid][1][lane]) +
        (quarter[wid][2][lane] + quarter[wid][3][lane]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  return grid_meet<K>(s, sync, sc, &okay, fin);
}

// The barrier with sums of FP32 values: summed over each warp in FP32, the
// warps' sums and the blocks' in FP64 (as block_partials sums them).
template <int NT, int K, class F>
__device__ __forceinline__ bool grid_sum32(const float (&v)[K], LoopSync& sync, CGScalars* sc,
                                           F fin) {
  __shared__ float warps[K][32];
  __shared__ int okay;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (threadIdx.x == 0) okay = 1;
#pragma unroll
  for (int k = 0; k < K; ++k) {
    float t = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) warps[k][wid] = t;
  }
  __syncthreads();
  double s = 0.0;
  if (wid < K) {
    s = lane < NT / 32 ? double(warps[wid][lane]) : 0.0;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  }
  return grid_meet<K>(s, sync, sc, &okay, fin);
}

// Up to maxits whole iterations of the FP64 PCG without a factor
// (ConjugateGradients::next/qAp/q/pq/rz/x, ConjugateGradients.cpp:584-823; the
// same operations in the same order per row as k_cg_p, k_cg_a and k_cg_b) in
// one cooperative launch, one block per SM, each block holding a contiguous
// run of `per` rows with its residual, q (then z), direction and inverse
// diagonal in shared memory; only the direction (gathered by other rows), x
// and the matrix are in global memory.
//
// The bounds are the FP64 pipe (22 operations a row: 11 us an iteration at 65^3,
// 38 at 97^3, where it is 70 % busy) and three grid barriers (grid_sum), for
// the drains, gaps and reduction tails of three launches: 38 -> 21 us an
// iteration at 65^3, 65 -> 48 at 97^3, 17 -> 10 at 17^3.  1024 threads with
// rounds of 8 entries and 512 with rounds of 16 are within 3 % of each other.
template <class CI>
__global__ void __launch_bounds__(kLoopThreads, 1)
    k_cg_loop(int64_t n, int per, int64_t maxits, const int32_t* __restrict__ soff,
              const int32_t* __restrict__ sw, CI ci, const double* __restrict__ a,
              const double* __restrict__ d, double* r, double* z, double* p, double* x,
              double* lpart, unsigned int* larrive, CGScalars* sc) {
  extern __shared__ double loop_smem[];
  __shared__ double sh_scale, sh_rho, sh_rho0, sh_rr, sh_pq;  // scale: alpha, then beta
  __shared__ int sh_fin, sh_end;
  if (sc->done) return;
  double* sr = loop_smem;
  double* sq = sr + per;  // q, then z
  double* sp = sq + per;
  double* sd = sp + per;
  const int64_t r0 = int64_t(blockIdx.x) * per;
  const int rows = static_cast<int>(n - r0 < per ? n - r0 : per);
  for (int t = threadIdx.x; t < rows; t += kLoopThreads) {
    sr[t] = r[r0 + t];
    sq[t] = z[r0 + t];
    sp[t] = p[r0 + t];
    sd[t] = d[r0 + t];
  }
  int64_t it = sc->it;
  const int64_t maxit = sc->maxit;
  const double nb = sc->normb > 1.0e-14 ? sc->normb : 1.0;
  const double lim = sc->tol * nb;
  const double eps = sc->guard == 0 ? DBL_EPSILON : DBL_MIN;
  if (threadIdx.x == 0) {
    sh_rho = sc->rho;
    sh_rho0 = sc->rho0;
    sh_rr = sc->rr;
    sh_pq = sc->pq;
    sh_fin = sc->finished;
    sh_end = 0;
    sh_scale = it == 0 ? 0.0 : sc->rho / sc->rho0;
  }
  __syncthreads();
  LoopSync sync{lpart, larrive, 0u, 0};
  double alpha = sc->alpha;
  const double none[1] = {0.0};
  for (int64_t step = 0; step < maxits && !sh_end; ++step) {
    // p = z + beta p
    const double beta = sh_scale;
    for (int t = threadIdx.x; t < rows; t += kLoopThreads) {
      const double pi = sq[t] + beta * sp[t];
      sp[t] = pi;
      p[r0 + t] = pi;
    }
    if (!grid_sum<0>(none, 0, sync, sc, [](int, double) {})) return;
    // q = A p, (p, q)
    double dot[1] = {0.0};
    for (int t = threadIdx.x; t < rows; t += kLoopThreads) {
      const int64_t i = r0 + t;
      const double s =
          sell_row_x<double, kLoopRound>(ci, a, soff[i >> 5], sw[i >> 5], int(i & 31), int32_t(i),
                                         [&](int32_t c) { return p[c]; });
      sq[t] = s;
      dot[0] += sp[t] * s;
    }
    if (!grid_sum<1>(dot, rows, sync, sc, [&](int, double pq) {
          sh_pq = pq;
          sh_fin = fabs(pq) < eps;
          sh_scale = sh_fin ? 0.0 : sh_rho / pq;
        }))
      return;
    alpha = sh_scale;
    // r -= alpha q, x += alpha p, z = r d, (r, z), (r, r)
    double v[2] = {0.0, 0.0};
    for (int t = threadIdx.x; t < rows; t += kLoopThreads) {
      const double ri = sr[t] - alpha * sq[t];
      sr[t] = ri;
      x[r0 + t] += alpha * sp[t];
      const double zi = ri * sd[t];
      sq[t] = zi;
      v[0] += ri * zi;
      v[1] += ri * ri;
    }
    it += 1;
    if (!grid_sum<2>(v, rows, sync, sc, [&](int k, double sum) {
          if (k == 0) {
            sh_rho0 = sh_rho;
            sh_rho = sum;
            sh_scale = sum / sh_rho0;
          } else {  // the stopping test (ConjugateGradients.cpp:772-823)
            sh_rr = sum;
            const double nr = sqrt(sum);
            sh_end = sh_fin || nr < lim || it >= maxit ? (nr > lim ? 1 : 2) : 0;
          }
        }))
      return;
  }
  for (int t = threadIdx.x; t < rows; t += kLoopThreads) {
    r[r0 + t] = sr[t];
    z[r0 + t] = sq[t];
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc->rho = sh_rho;
    sc->rho0 = sh_rho0;
    sc->rr = sh_rr;
    sc->pq = sh_pq;
    sc->alpha = alpha;
    sc->it = it;
    sc->finished = sh_fin;
    sc->converged = sh_end == 2;
    sc->done = sh_end != 0;
  }
}

// ---- the mixed solve's FP32 iteration as one kernel

__device__ __forceinline__ unsigned smem_at(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
// `bytes` (a multiple of 16) from global to shared memory (16-byte boundaries
// both), asynchronously, counted at the barrier `mb`.  The bytes are read once
// a pass and leave L2 first: at 129^3 the vectors then stay there (A's pass
// 46 -> 40 us, the lower triangle's 23.5 -> 21.5).
__device__ __forceinline__ void bulk_copy(void* dst, const void* src, unsigned bytes,
                                          uint64_t* mb) {
  uint64_t once;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(once));
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint "
      "[%0], [%1], %2, [%3], %4;"
      :
      : "r"(smem_at(dst)), "l"(src), "r"(bytes), "r"(smem_at(mb)), "l"(once)
      : "memory");
}
// `bytes` will arrive at the barrier `mb` in its current phase.
__device__ __forceinline__ void bulk_expect(uint64_t* mb, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
               :
               : "r"(smem_at(mb)), "r"(bytes)
               : "memory");
}
// Waits for the phase `parity` of the barrier; false when it does not come
// within about a second (a try is suspended for a microsecond at most).
__device__ __forceinline__ bool bulk_wait(uint64_t* mb, unsigned parity) {
  for (int k = 0; k < kLoopSpin; ++k) {
    unsigned ok;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_at(mb)), "r"(parity), "r"(1000u)
        : "memory");
    if (ok) return true;
  }
  return false;
}

// Threads of k_mixed_loop, one block per SM, and its gathers in flight per
// row.  Whole rows of 15 entries in one round need 80 registers (768 threads):
// 153 us an iteration at 129^3 against 132 for 1024 threads and rounds of 8,
// both with copies of 16 bytes a lane.
constexpr int kMixThreads = 1024;
constexpr int kMixRound = 8;

// A warp's walk over the slices first, first + step, ... < end of a SELL-32
// layout: columns and values of the next slice (up to XM entries a row) are
// copied into the warp's stage in shared memory while the gathers of the
// current one are under way, and the next slice's place is read one slice
// earlier still.  Columns, values and gathers one after another would cost a
// slice two memory latencies, and the matrix is the larger part of the bytes.
// The copies are bulk copies, two a slice: as 16-byte asynchronous copies of
// every lane they held the load path (129^3: 132 us an iteration, 120 so).
//
// A warp's copies, in one word that its walks share: the phase of its barrier, a
// copy under way, a copy that did not arrive.  After a lost copy the warp issues
// no other and reads no stage; the kernel ends with an error, having waited for
// that copy once more.
constexpr unsigned kWalkPhase = 1, kWalkPending = 2, kWalkLost = 4;
template <class CI, class V, int XM>
struct SliceWalk {
  using E = typename CI::E;
  static constexpr int kBytes = XM * kSlice * int(sizeof(E) + sizeof(V));
  const int32_t *soff, *sw;
  CI ci;
  const V* val;
  char* stage;
  int32_t s, end;
  int32_t off, w, offn, wn;  // the slice in the stage, the next one
  const int4* places;        // the warp's first two slices, in shared memory
  uint64_t* mb;              // the warp's barrier
  int* bad;                  // set when a copy did not arrive
  static constexpr int step = kMixThreads / 32;

  // (one lane) the slice's columns and values into the stage
  __device__ __forceinline__ void copy(unsigned& st) {
    const unsigned we = w < XM ? w : XM;
    if (!we) return;
    st |= kWalkPending;
    if (threadIdx.x & 31) return;
    bulk_expect(mb, we * unsigned(kSlice * (sizeof(E) + sizeof(V))));
    bulk_copy(stage, val + off, we * unsigned(kSlice * sizeof(V)), mb);
    bulk_copy(stage + XM * kSlice * sizeof(V), ci.c + off, we * unsigned(kSlice * sizeof(E)), mb);
  }
  // the places of the warp's first two slices
  __device__ __forceinline__ int4 first_two(int32_t first) const {
    int4 f = make_int4(0, 0, 0, 0);
    if (first < end) {
      f.x = __ldg(soff + first);
      f.y = __ldg(sw + first);
    }
    if (first + step < end) {
      f.z = __ldg(soff + first + step);
      f.w = __ldg(sw + first + step);
    }
    return f;
  }
  // the first slice into the stage
  __device__ __forceinline__ void start(int32_t first, unsigned& st) {
    s = st & kWalkLost ? end : first;
    asm volatile("" : "+r"(s));  // keeps a pass's addresses out of the others' registers
    if (s >= end) return;
    const int4 f = places[threadIdx.x >> 5];
    off = f.x;
    w = f.y;
    offn = f.z;
    wn = f.w;
    __syncwarp();
    copy(st);
  }
  // the stage has been read: the next slice into it
  __device__ __forceinline__ void advance(unsigned& st) {
    __syncwarp();
    s += step;
    if (s < end) {
      off = offn;
      w = wn;
      copy(st);
      if (s + step < end) {
        offn = __ldg(soff + s + step);
        wn = __ldg(sw + s + step);
      }
    }
  }
  // entries k .. k + W - 1 of row i added to t; next() once the stage is read
  template <int W, class G, class N>
  __device__ __forceinline__ float fixed(int k, float t, int32_t i, G g, N next) {
    int32_t cc[W];
    float vv[W];
    const int o = k * kSlice + (threadIdx.x & 31);
    const V* sval = reinterpret_cast<const V*>(stage) + o;
    const E* scol = reinterpret_cast<const E*>(stage + XM * kSlice * sizeof(V)) + o;
#pragma unroll
    for (int u = 0; u < W; ++u) {
      const int32_t c = CI::of(scol[u * kSlice], i);
      vv[u] = c < 0 ? 0.0f : float(sval[u * kSlice]);
      cc[u] = c < 0 ? i : c;
    }
    next();
#pragma unroll
    for (int u = 0; u < W; ++u) t += vv[u] * g(cc[u]);
    return t;
  }
  template <int W, class G, class N>
  __device__ __forceinline__ float pick(int r, int k, float t, int32_t i, G g, N next) {
    if constexpr (W <= kMixRound) {
      if (r == W) return fixed<W>(k, t, i, g, next);
      return pick<W + 1>(r, k, t, i, g, next);
    } else {
      next();
      return t;
    }
  }
  // sum_k val[e_k] g(col[e_k]) over row i of the current slice, in entry
  // order, in rounds of at most kMixRound entries whose gathers are in flight
  // together; moves on to the next slice and calls `own` before the gathers
  // of the last staged round (loads of the next slice's own row go there).
  // The entries beyond XM of a wide slice are read one by one.
  template <class G, class O>
  __device__ __forceinline__ float row(int32_t i, G g, O own, unsigned& st) {
    const int32_t o = off;
    int32_t r = w;
    if (r > 0) {
      if (__all_sync(0xffffffffu, bulk_wait(mb, st & kWalkPhase))) {
        st = (st ^ kWalkPhase) & ~kWalkPending;
      } else {  // no entry is read, and the walk ends
        *bad = 1;
        st |= kWalkLost;
        r = 0;
        s = end;
      }
    }
    const int32_t rs = r < XM ? r : XM;
    float t = 0.0f;
    int k = 0;
    for (; rs - k > kMixRound; k += kMixRound) t = fixed<kMixRound>(k, t, i, g, [] {});
    t = pick<1>(rs - k, k, t, i, g, [&] {
      advance(st);
      own();
    });
    for (k = XM; k < r; ++k) {
      const int32_t e = o + k * kSlice + int(threadIdx.x & 31);
      const int32_t c = ci.at(e, i);
      if (c >= 0) t += float(ldv(val + e)) * g(c);
    }
    return t;
  }
};

template <class CI>
struct MixArgs {
  int64_t n, maxits;
  const int32_t *soff, *sw, *soffU, *swU, *soffL, *swL;
  CI ci, cu, cl;
  const float* a;
  const __half *nvU, *nvL;
  const float *rs, *msrow, *d;  // msrow: S, negative at Dirichlet nodes
  float *z, *p, *q, *r, *v, *u;
  float2 *zp, *vt;
  double* e;
  double* lpart;
  unsigned int* larrive;
  CGScalars* sc;
};

constexpr int kMixFull = 16, kMixTri = 8;  // staged entries per row: whole rows, triangles

// Up to maxits iterations of the mixed solve's FP32 PCG in one cooperative
// launch, one block per SM, each with a contiguous run of slices.  FACTOR:
// q = A p' and (p', q); the update with u = (I+N)^T S r'; z = -S (I+N) u
// (Dirichlet rows: z = r), (r, z), (r, r) and the stopping test.  Jacobi: the
// last two are one pass over the block's own rows.
//
// What a pass gathers is one record per row, 8 bytes, so an entry costs one
// address and one load: (z, p) for p' = z + beta p, formed per gathered
// entry, and with v = S r, t = S q the pair (v, t) for v' = v - alpha t, the
// neighbours' new scaled residuals (in the factored iteration the residual is
// kept as v; r = v / S where its norm is taken).  (p', q) is summed per thread
// in FP32 and widened once, and each row formed as
// sum_j a_ij (p'_j - p'_i) + rs_i p'_i (rs: the row's exact sum, zero for an
// interior row of the pressure Laplacian): on a smooth p' the terms
// a_ij p'_j of the plain sum cancel to a result about 1/kappa(A) of their
// size, which FP32 cannot hold, while the differences p'_j - p'_i are formed
// exactly and nothing large cancels.  The correction e += alpha p' is summed
// in FP64 (FP32 rounding noise in it would be amplified by A's largest
// eigenvalues into the residual the outer loop replaces).
//
// The bound is memory: 6 bytes an entry of A, 4 of each triangle and some 90
// of vectors a row, 0.5 GB an iteration at 129^3; A's pass runs at 7.4 TB/s
// there (part of the vectors stays in L2), the triangles' at 5, and the three
// barriers with their sums take 2 to 5 us each.  The whole solve's time over its
// iterations, a launch per pass against this: 145 / 104 us at 129^3, 35.5 / 27.9
// at 65^3, 27.1 / 24.3 at 17^3.
template <class CI, bool FACTOR>
__global__ void __launch_bounds__(kMixThreads, 1)
    k_mixed_loop(const __grid_constant__ MixArgs<CI> A) {
  extern __shared__ __align__(16) char mix_smem[];
  __shared__ double sh_beta, sh_rho, sh_rho0, sh_rr, sh_pq, sh_lim, sh_alpha;
  __shared__ int64_t sh_maxit;
  __shared__ int sh_fin, sh_end, sh_bad;
  __shared__ uint64_t sh_mb[kMixThreads / 32];
  __shared__ int4 sh_places[3][kMixThreads / 32];
  CGScalars* sc = A.sc;
  if (sc->done) return;
  using WalkA = SliceWalk<CI, float, kMixFull>;
  using WalkT = SliceWalk<CI, __half, kMixTri>;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  char* stage = mix_smem + wid * WalkA::kBytes;
  const int32_t ns = int32_t((A.n + kSlice - 1) / kSlice);
  const int32_t s0 = int32_t(int64_t(ns) * blockIdx.x / gridDim.x);
  const int32_t s1 = int32_t(int64_t(ns) * (blockIdx.x + 1) / gridDim.x);
  const int32_t last = int32_t(A.n - 1);
  const int64_t r0 = int64_t(s0) * kSlice, r1 = min(int64_t(s1) * kSlice, A.n);
  int64_t it = sc->it;
  if (threadIdx.x == 0) {
    const double nb = sc->normb > 1.0e-14 ? sc->normb : 1.0;
    // a residual replacement is due when ||r|| < max(tol ||b||, delta * rlast)
    // (rlast: the last true residual norm), or at maxit iterations
    sh_lim = fmax(sc->tol * nb, sc->delta * sc->rlast);
    sh_maxit = sc->maxit;
    sh_alpha = sc->alpha;
    sh_rho = sc->rho;
    sh_rho0 = sc->rho0;
    sh_rr = sc->rr;
    sh_pq = sc->pq;
    sh_fin = sc->finished;
    sh_end = 0;
    sh_bad = 0;
    sh_beta = it == 0 ? 0.0 : sc->rho / sc->rho0;
  }
  for (int64_t i = r0 + threadIdx.x; i < r1; i += kMixThreads)
    A.zp[i] = make_float2(A.z[i], A.p[i]);
  unsigned st = 0;  // the warp's copies
  uint64_t* mb = &sh_mb[wid];
  WalkA wa{A.soff, A.sw, A.ci, A.a, stage, 0, s1, 0, 0, 0, 0, sh_places[0], mb, &sh_bad};
  WalkT wu{A.soffU, A.swU, A.cu, A.nvU, stage, 0, s1, 0, 0, 0, 0, sh_places[1], mb, &sh_bad};
  WalkT wl{A.soffL, A.swL, A.cl, A.nvL, stage, 0, s1, 0, 0, 0, 0, sh_places[2], mb, &sh_bad};
  if (lane == 0)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_at(mb)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  __syncwarp();
  if (lane == 0) {
    sh_places[0][wid] = wa.first_two(s0 + wid);
    if (FACTOR) {
      sh_places[1][wid] = wu.first_two(s0 + wid);
      sh_places[2][wid] = wl.first_two(s0 + wid);
    }
  }
  __syncwarp();
  wa.start(s0 + wid, st);
  LoopSync sync{A.lpart, A.larrive, 0u, 0};
  const double none[1] = {0.0};
  bool ok = grid_sum<0>(none, 0, sync, sc, [](int, double) {});
  float alpha = 0.0f;
  for (int64_t step = 0; ok && step < A.maxits && !sh_end; ++step) {
    {  // q = A p', (p', q); the last iteration's alpha p into e
      const float beta = float(sh_beta);
      float dot[1] = {0.0f};
      float2 zp = make_float2(0.0f, 0.0f);
      float rs = 0.0f, vi = 0.0f, si = 0.0f;
      double ei = 0.0;
      auto own = [&] {
        if (wa.s < s1) {
          const int32_t j = min(wa.s * kSlice + lane, last);
          zp = A.zp[j];
          rs = __ldg(A.rs + j);
          ei = A.e[j];
          if (FACTOR) {
            vi = A.v[j];
            si = __ldg(A.msrow + j);
          }
        }
      };
      own();
      while (wa.s < s1) {
        const int32_t k = wa.s * kSlice + lane, row = min(k, last);
        const float p = zp.x + beta * zp.y, rp = rs * p, v = vi, sr = si;
        if (k <= last) A.e[row] = ei + double(alpha) * double(zp.y);
        const float q = wa.row(
                            row,
                            [&](int32_t c) {
                              const float2 g = A.zp[c];
                              return (g.x + beta * g.y) - p;
                            },
                            own, st) +
                        rp;
        if (k <= last) {
          A.p[row] = p;
          if (FACTOR)
            A.vt[row] = make_float2(v, fabsf(sr) * q);
          else
            A.q[row] = q;
          dot[0] += p * q;
        }
      }
      if (FACTOR) wu.start(s0 + wid, st);
      ok = grid_sum32<kMixThreads, 1>(dot, sync, sc, [&](int, double pq) {
        sh_pq = pq;
        sh_rho0 = sh_rho;
        sh_fin = fabs(pq) < DBL_MIN;
        sh_alpha = sh_fin ? 0.0 : sh_rho / pq;
      });
      ok = __syncthreads_and(ok && !sh_bad);
      if (!ok) break;
    }
    alpha = float(sh_alpha);
    float v[2] = {0.0f, 0.0f};
    if (FACTOR) {
      {  // v' = v - alpha t, u = (I+N)^T v'
        float2 vt = make_float2(0.0f, 0.0f);
        auto own = [&] {
          if (wu.s < s1) {
            const int32_t j = min(wu.s * kSlice + lane, last);
            vt = A.vt[j];
          }
        };
        own();
        while (wu.s < s1) {
          const int32_t k = wu.s * kSlice + lane, row = min(k, last);
          const float vi = vt.x - alpha * vt.y;
          if (k <= last) A.v[row] = vi;
          const float t = wu.row(
              row,
              [&](int32_t c) {
                const float2 g = A.vt[c];
                return g.x - alpha * g.y;
              },
              own, st);
          if (k <= last) A.u[row] = vi + t;
        }
      }
      wl.start(s0 + wid, st);
      ok = grid_sum<0>(none, 0, sync, sc, [](int, double) {});
      ok = __syncthreads_and(ok && !sh_bad);
      if (!ok) break;
      {  // z = -S (I+N) u
        float vi = 0.0f, ui = 0.0f, si = 1.0f, pi = 0.0f;
        auto own = [&] {
          if (wl.s < s1) {
            const int32_t j = min(wl.s * kSlice + lane, last);
            ui = A.u[j];
            vi = A.v[j];
            pi = A.p[j];
            si = __ldg(A.msrow + j);
          }
        };
        own();
        while (wl.s < s1) {
          const int32_t k = wl.s * kSlice + lane, row = min(k, last);
          const float u = ui, p = pi, sr = si, r = vi * __frcp_rn(fabsf(sr));
          const float acc = u + wl.row(row, [&](int32_t c) { return A.u[c]; }, own, st);
          const float zi = sr < 0.0f ? r : -sr * acc;
          if (k <= last) {
            A.zp[row] = make_float2(zi, p);
            v[0] += r * zi;
            v[1] += r * r;
          }
        }
      }
    } else {
      for (int64_t i = r0 + threadIdx.x; i < r1; i += kMixThreads) {
        const float r = A.r[i] - alpha * A.q[i], p = A.p[i];
        A.r[i] = r;
        const float zi = r * __ldg(A.d + i);
        A.zp[i] = make_float2(zi, p);
        v[0] += r * zi;
        v[1] += r * r;
      }
    }
    wa.start(s0 + wid, st);
    it += 1;
    ok = grid_sum32<kMixThreads, 2>(v, sync, sc, [&](int k, double sum) {
      if (k == 0) {
        sh_rho = sum;
        sh_beta = sum / sh_rho0;
      } else {
        sh_rr = sum;
        sh_end = sh_fin || sqrt(sum) < sh_lim || it >= sh_maxit;
      }
    });
    ok = __syncthreads_and(ok && !sh_bad);
  }
  // the next pass's first slice may be on its way
  if (st & kWalkPending) (void)bulk_wait(&sh_mb[wid], st & kWalkPhase);
  if (!ok) {  // a wait ran out
    if (threadIdx.x == 0) atomicExch(&sc->err, 1);
    return;
  }
  for (int64_t i = r0 + threadIdx.x; i < r1; i += kMixThreads) {
    A.z[i] = A.zp[i].x;
    A.e[i] += double(alpha) * double(A.p[i]);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    sc->rho = sh_rho;
    sc->rho0 = sh_rho0;
    sc->rr = sh_rr;
    sc->pq = sh_pq;
    sc->alpha = sh_alpha;
    sc->it = it;
    sc->finished = sh_fin;
    sc->done = sh_end;
  }
}

// ---- the FP64 iteration of a small system in one thread-block cluster
//
// A system of a few thousand rows is barriers: k_cg_loop's cost 1.3 us each
// through L2, 10 us an iteration at 17^3.  One cluster of 16 SMs meets by the
// hardware barrier and holds everything, matrix included, in its blocks'
// shared memory, gathering the direction from its owner's (distributed shared
// memory).  The FP64 work runs on 16 SMs instead of all, 22 operations a row
// and iteration: 6.6 against 11.1 us an iteration at 17^3, 9.4 against 11.2 at
// 21^3, 10.2 against 12.7 at 24^3, about where the shared memory ends (15
// entries a row; k_cg_loop takes what is larger or does not fit).
constexpr int kClusterSize = 16;
constexpr int kClusterThreads = 512;
constexpr int64_t kClusterRows = 16384;

__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::
                   : "memory");
}
// The address of this block's shared-memory location p in block `rank`.
__device__ __forceinline__ uint32_t cluster_addr(const void* p, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;"
               : "=r"(a)
               : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(rank));
  return a;
}
__device__ __forceinline__ double ld_cluster(uint32_t a) {
  double v;
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_cluster(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}

// As grid_sum over the cluster's blocks: lane 0 of warp k calls fin(k, sum).
// box: [3][2][kClusterSize] in shared memory, turn: barriers with sums so far,
// modulo 3 (a block may be one barrier ahead of the slowest reader).
template <int K, class F>
__device__ __forceinline__ void cluster_sum(const double (&v)[K], int active, double* box,
                                            int& turn, F fin) {
  constexpr int NW = kClusterThreads / 32 / 4;
  __shared__ double rows[K][kClusterThreads];
  __shared__ double quarter[K][4][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < K; ++k) rows[k][threadIdx.x] = v[k];
  __syncthreads();
  if (wid < 4 * K) {
    const int k = wid >> 2, qd = wid & 3;
    double s = 0.0;
#pragma unroll
    for (int j = 0; j < NW; ++j)
      if (32 * (qd + 4 * j) < active) s += rows[k][lane + 32 * (qd + 4 * j)];
    quarter[k][qd][lane] = s;
  }
  __syncthreads();
  double* b = box + turn * 2 * kClusterSize;
  if (wid < K) {
    double s = (quarter[wid][0][lane] + quarter[wid][1][lane]) +
               (quarter[wid][2][lane] + quarter[wid][3][lane]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane < kClusterSize)
      st_cluster(cluster_addr(b + wid * kClusterSize + blockIdx.x, lane), s);
  }
  cluster_sync();
  if (wid < K) {
    double s = lane < kClusterSize ? b[wid * kClusterSize + lane] : 0.0;
#pragma unroll
    for (int o = kClusterSize / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) fin(wid, s);
  }
  turn = turn == 2 ? 0 : turn + 1;
  __syncthreads();
}

// The whole solve of a small system: as k_cg_loop, one cluster of kClusterSize
// blocks (the grid), `per` rows each (whole slices), `ents` matrix entries at
// most in a block.
__global__ void __launch_bounds__(kClusterThreads, 1)
    k_cg_cluster(int64_t n, int per, int ents, int64_t maxits, const int32_t* __restrict__ soff,
                 const int32_t* __restrict__ sw, const int32_t* __restrict__ col,
                 const double* __restrict__ a, const double* __restrict__ d, double* r, double* z,
                 double* p, double* x, CGScalars* sc) {
  extern __shared__ double loop_smem[];
  __shared__ double box[3 * 2 * kClusterSize];
  __shared__ double sh_scale, sh_rho, sh_rho0, sh_rr, sh_pq;
  __shared__ int sh_fin, sh_end;
  double* sr = loop_smem;
  double* sq = sr + per;  // q, then z
  double* sp = sq + per;
  double* sd = sp + per;
  double* sx = sd + per;
  double* sa = sx + per;                                   // matrix values
  uint32_t* sc_at = reinterpret_cast<uint32_t*>(sa + ents);  // where each column's p lies
  const bool already = sc->done != 0;  // the same in every block
  const int64_t r0 = int64_t(blockIdx.x) * per;
  const int rows = already || r0 >= n ? 0 : static_cast<int>(n - r0 < per ? n - r0 : per);
  const int32_t e0 = rows ? soff[r0 >> 5] : 0;
  const int32_t e1 = rows ? soff[(r0 + rows + kSlice - 1) >> 5] : 0;
  for (int t = threadIdx.x; t < rows; t += kClusterThreads) {
    sr[t] = r[r0 + t];
    sq[t] = z[r0 + t];
    sp[t] = p[r0 + t];
    sd[t] = d[r0 + t];
    sx[t] = x[r0 + t];
  }
  for (int t = threadIdx.x; t < e1 - e0; t += kClusterThreads) {
    // padding reads the block's first p with weight 0
    const int32_t c = col[e0 + t];
    const int rank = c < 0 ? int(blockIdx.x) : c / per;
    sa[t] = c < 0 ? 0.0 : a[e0 + t];
    sc_at[t] = cluster_addr(sp, rank) + (c < 0 ? 0 : (c - rank * per) * 8);
  }
  int64_t it = sc->it;
  const int64_t maxit = sc->maxit;
  const double nb = sc->normb > 1.0e-14 ? sc->normb : 1.0;
  const double lim = sc->tol * nb;
  const double eps = sc->guard == 0 ? DBL_EPSILON : DBL_MIN;
  if (threadIdx.x == 0) {
    sh_rho = sc->rho;
    sh_rho0 = sc->rho0;
    sh_rr = sc->rr;
    sh_pq = sc->pq;
    sh_fin = sc->finished;
    sh_end = already ? 1 : 0;
    sh_scale = it == 0 ? 0.0 : sc->rho / sc->rho0;
  }
  double alpha = sc->alpha;
  // every block runs before another's shared memory is touched, and the loads
  // of the scalars are done before block 0 writes them back
  cluster_sync();
  int turn = 0;
  for (int64_t step = 0; step < maxits && !sh_end; ++step) {
    const double beta = sh_scale;
    for (int t = threadIdx.x; t < rows; t += kClusterThreads) sp[t] = sq[t] + beta * sp[t];
    cluster_sync();
    double dot[1] = {0.0};
    for (int t = threadIdx.x; t < rows; t += kClusterThreads) {
      const int64_t sl = (r0 + t) >> 5;
      const int w = sw[sl], o = soff[sl] - e0 + (t & 31);
      double s = 0.0;
      for (int k0 = 0; k0 < w; k0 += kLoopRound) {
        double v[kLoopRound], g[kLoopRound];
#pragma unroll
        for (int u = 0; u < kLoopRound; ++u) {
          const bool in = k0 + u < w;
          const int e = o + (k0 + u) * kSlice;
          v[u] = in ? sa[e] : 0.0;
          g[u] = in ? ld_cluster(sc_at[e]) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kLoopRound; ++u)
          if (k0 + u < w) s += v[u] * g[u];
      }
      sq[t] = s;
      dot[0] += sp[t] * s;
    }
    cluster_sum<1>(dot, rows, box, turn, [&](int, double pq) {
      sh_pq = pq;
      sh_fin = fabs(pq) < eps;
      sh_scale = sh_fin ? 0.0 : sh_rho / pq;
    });
    alpha = sh_scale;
    double v[2] = {0.0, 0.0};
    for (int t = threadIdx.x; t < rows; t += kClusterThreads) {
      const double ri = sr[t] - alpha * sq[t];
      sr[t] = ri;
      sx[t] += alpha * sp[t];
      const double zi = ri * sd[t];
      sq[t] = zi;
      v[0] += ri * zi;
      v[1] += ri * ri;
    }
    it += 1;
    cluster_sum<2>(v, rows, box, turn, [&](int k, double sum) {
      if (k == 0) {
        sh_rho0 = sh_rho;
        sh_rho = sum;
        sh_scale = sum / sh_rho0;
      } else {  // the stopping test (ConjugateGradients.cpp:772-823)
        sh_rr = sum;
        const double nr = sqrt(sum);
        sh_end = sh_fin || nr < lim || it >= maxit ? (nr > lim ? 1 : 2) : 0;
      }
    });
  }
  if (!already) {
    for (int t = threadIdx.x; t < rows; t += kClusterThreads) {
      r[r0 + t] = sr[t];
      z[r0 + t] = sq[t];
      p[r0 + t] = sp[t];
      x[r0 + t] = sx[t];
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      sc->rho = sh_rho;
      sc->rho0 = sh_rho0;
      sc->rr = sh_rr;
      sc->pq = sh_pq;
      sc->alpha = alpha;
      sc->it = it;
      sc->finished = sh_fin;
      sc->converged = sh_end == 2;
      sc->done = sh_end != 0;
    }
  }
  cluster_sync();  // no block leaves while another may read its shared memory
}

// v = S r
template <class T>
__global__ void k_scale(int64_t n, const float* __restrict__ srow, const T* __restrict__ r,
                        T* __restrict__ v) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i < n) v[i] = T(srow[i]) * r[i];
}

// ---- mixed precision: residual replacement

// r = b - A x in FP64 (true residual), r32 = r; Jacobi: z32 = r32 d32 and
// rho = (r32, z32); factor (srow given): v32 = S r32.  Partial (r,r) -> rr.
// FIRST starts the FP32 iteration (it = 0, so beta = 0); otherwise it
// continues with the kept search direction.
__global__ void __launch_bounds__(kBlock) k_outer_res(int64_t n, const int32_t* __restrict__ soff,
                                                       const int32_t* __restrict__ sw,
                                                       const int32_t* __restrict__ col,
                                                       const double* __restrict__ a,
                                                       const double* __restrict__ x,
                                                       const double* __restrict__ b,
                                                       const float* __restrict__ d32,
                                                       const float* __restrict__ srow,
                                                       float* __restrict__ r32,
                                                       float* __restrict__ z32,
                                                       float* __restrict__ v32, int first,
                                                       double* partial, CGScalars* sc) {
  double v[2] = {0.0, 0.0};
  XG_ROWS(i, n) {
    const int lane = int(i & 31);
    const double s = sell_row_x<double>(Cols32{col}, a, soff[i >> 5], sw[i >> 5], lane,
                                         int32_t(i), [&](int32_t c) { return __ldg(x + c); });
    const double ri = b[i] - s;
    const float rf = float(ri);
    r32[i] = rf;
    if (srow) {
      v32[i] = srow[i] * rf;
    } else {
      const float zf = rf * d32[i];
      z32[i] = zf;
      v[1] += double(rf) * double(zf);
    }
    v[0] += ri * ri;
  }
  if (block_partials<2>(v, partial, &sc->ticket[0])) {
    double rr = sum_partials(partial, 0);
    double rz = sum_partials(partial, 1);
    if (threadIdx.x == 0) {
      sc->rr = rr;
      if (!srow) sc->rho = rz;
      if (first) sc->it = 0;
      sc->done = 0;
      sc->finished = 0;
      sc->ticket[0] = 0;
    }
  }
}

// x += e, e = 0
__global__ void k_add_correction(int64_t n, double* __restrict__ e, double* __restrict__ x) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i < n) {
    x[i] += e[i];
    e[i] = 0.0;
  }
}

__global__ void k_jacobi_apply(int64_t n, const double* __restrict__ r, const double* __restrict__ d,
                               double* __restrict__ z) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i < n) z[i] = r[i] * d[i];
}

// ---- factor construction

// Row scales s_i = 1/sqrt|a_ii| of the working matrix; msrow: the same with the
// sign set at Dirichlet nodes.
__global__ void k_factor_geom(int64_t n, const double* __restrict__ a,
                              const int32_t* __restrict__ diagpos, float* __restrict__ srow,
                              const uint8_t* __restrict__ mask,
                              float* __restrict__ msrow) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  srow[i] = float(1.0 / sqrt(fabs(a[diagpos[i]])));
  msrow[i] = mask[i] ? -srow[i] : srow[i];
}
// e_ij = a_ij s_i s_j (0 when i or j is a Dirichlet node) in the lower and
// upper layouts.
__global__ void k_factor_e(int64_t n, const int32_t* __restrict__ soffL,
                           const int32_t* __restrict__ swL, const int32_t* __restrict__ colL,
                           const int32_t* __restrict__ posL, const int32_t* __restrict__ tposU,
                           const double* __restrict__ a, const float* __restrict__ srow,
                           const uint8_t* __restrict__ mask, float* __restrict__ eL,
                           float* __restrict__ eU) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const int lane = int(i & 31);
  const int32_t off = soffL[i >> 5], w = swL[i >> 5];
  for (int k = 0; k < w; ++k) {
    const int32_t e = off + k * kSlice + lane;
    const int32_t j = colL[e];
    if (j < 0) continue;
    const float v = (mask[i] || mask[j]) ? 0.f : float(a[posL[e]]) * srow[i] * srow[j];
    eL[e] = v;
    eU[tposU[e]] = v;
  }
}
// e_ij in the full layout.
__global__ void k_factor_efull(int64_t n, const int32_t* __restrict__ soff,
                               const int32_t* __restrict__ sw, const int32_t* __restrict__ col,
                               const double* __restrict__ a, const float* __restrict__ srow,
                               const uint8_t* __restrict__ mask, float* __restrict__ eF) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const int lane = int(i & 31);
  const int32_t off = soff[i >> 5], w = sw[i >> 5];
  for (int k = 0; k < w; ++k) {
    const int32_t e = off + k * kSlice + lane;
    const int32_t j = col[e];
    eF[e] = (j < 0 || j == i || mask[i] || mask[j]) ? 0.f : float(a[e]) * srow[i] * srow[j];
  }
}
// N_ij = c e_ij (the first-order factor, c = 1, or any uniform scaling), in
// the lower layout and, transposed, the upper one.
__global__ void k_factor_scaled(int64_t n, const int32_t* __restrict__ soffL,
                                const int32_t* __restrict__ swL, const int32_t* __restrict__ colL,
                                const int32_t* __restrict__ tposU, const float* __restrict__ eL,
                                float c, float* __restrict__ nvL, float* __restrict__ nvU) {
  int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
  const int lane = int(i & 31);
  const int32_t off = soffL[i >> 5], w = swL[i >> 5];
  for (int k = 0; k < w; ++k) {
    const int32_t e = off + k * kSlice + lane;
    const int32_t j = colL[e];
    if (j < 0) continue;
    const float v = c * eL[e];
    nvL[e] = v;
    nvU[tposU[e]] = v;
  }
}
__global__ void k_to_half(int64_t m, const float* __restrict__ a, __half* __restrict__ h) {
  int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (e < m) h[e] = __float2half_rn(a[e]);
}

// ---------------------------------------------------------------- host helpers

int read_scal(xg_ctx* c, CGDev* d, CGScalars* h) {
  XG_CUDA(c, cudaMemcpyAsync(h, d->scal, sizeof(CGScalars), cudaMemcpyDeviceToHost, c->stream));
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  return XG_OK;
}
int write_scal(xg_ctx* c, CGDev* d, const CGScalars* h) {
  XG_CUDA(c, cudaMemcpyAsync(d->scal, h, sizeof(CGScalars), cudaMemcpyHostToDevice, c->stream));
  // h lives on the caller's stack frame: complete the copy before returning
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  return XG_OK;
}

// Row scales and normalised couplings of the current working matrix.
int build_geom(xg_ctx* c, CGDev* d) {
  cudaStream_t s = c->stream;
  const unsigned nb = blocks_for(d->n, kBlock);
  k_factor_geom<<<nb, kBlock, 0, s>>>(d->n, d->a, d->diagpos, d->srow, d->bcmask, d->msrow);
  XG_CHECK_LAUNCH(c);
  k_factor_e<<<nb, kBlock, 0, s>>>(d->n, d->soffL, d->swL, d->colL, d->posL, d->tposU, d->a,
                                   d->srow, d->bcmask, d->eL, d->eU);
  XG_CHECK_LAUNCH(c);
  k_factor_efull<<<nb, kBlock, 0, s>>>(d->n, d->soff, d->swidth, d->col, d->a, d->srow, d->bcmask,
                                       d->eF);
  XG_CHECK_LAUNCH(c);
  d->geom_set = true;
  return XG_OK;
}

LpcGraph graph_of(const CGDev* d) {
  LpcGraph g;
  g.n = d->n;
  g.nslice = d->nslice;
  g.soff = d->soff;
  g.sw = d->swidth;
  g.col = d->col;
  g.eF = d->eF;
  g.soffL = d->soffL;
  g.swL = d->swL;
  g.colL = d->colL;
  g.eL = d->eL;
  g.tposU = d->tposU;
  g.soffU = d->soffU;
  g.swU = d->swU;
  g.colU = d->colU;
  g.eU = d->eU;
  g.srow = d->srow;
  g.mask = d->bcmask;
  g.nentL = d->nentL;
  g.nentU = d->nentU;
  return g;
}

// Scales, couplings and factor values (FP32 and FP16) of the current
// working matrix.
int build_factor(xg_ctx* c, CGDev* d) {
  cudaStream_t s = c->stream;
  const unsigned nb = blocks_for(d->n, kBlock);
  if (!d->geom_set) {
    int rg = build_geom(c, d);
    if (rg) return rg;
  }
  if (d->factor_model) {
    int rc = lpc_factor(c, d->factor_model, graph_of(d), d->nvL, d->nvU);
    if (rc) return rc;
  } else {
    k_factor_scaled<<<nb, kBlock, 0, s>>>(d->n, d->soffL, d->swL, d->colL, d->tposU, d->eL,
                                          float(d->factor_c), d->nvL, d->nvU);
    XG_CHECK_LAUNCH(c);
  }
  k_to_half<<<blocks_for(std::max<int64_t>(1, d->nentL), kBlock), kBlock, 0, s>>>(d->nentL, d->nvL,
                                                                                  d->hvL);
  k_to_half<<<blocks_for(std::max<int64_t>(1, d->nentU), kBlock), kBlock, 0, s>>>(d->nentU, d->nvU,
                                                                                  d->hvU);
  XG_CHECK_LAUNCH(c);
  d->factor_set = true;
  return XG_OK;
}

// z = M^-1 r with the factor in FP64 vectors (FP32 values): v = S r, then the
// two passes; rho = (r, z).
int factor_apply64(xg_ctx* c, CGDev* d, const double* r, double* z) {
  cudaStream_t s = c->stream;
  const int64_t n = d->n;
  k_scale<double><<<blocks_for(n, kBlock), kBlock, 0, s>>>(n, d->srow, r, d->v);
  launch_dep<k_pc_upper<double, float, Cols32>>(c, n, n, d->soffU, d->swU, Cols32{d->colU}, d->nvU,
      d->v, d->u, d->scal);
  launch_dep<k_pc_lower<double, float, Cols32, 0>>(c, n, n, d->soffL, d->swL, Cols32{d->colL},
      d->nvL, d->srow, d->bcmask, d->u, r, z, d->partial, d->scal);
  XG_CHECK_LAUNCH(c);
  return XG_OK;
}

// The FP32 factor passes on v32 = S r (already written, r the current
// residual): z32 and rho = (r, z32).
template <class CI>
void factor_apply32(xg_ctx* c, CGDev* d, CI cu, CI cl) {
  cudaStream_t s = c->stream;
  const int64_t n = d->n;
  launch_dep<k_pc_upper<float, __half, CI>>(c, n, n, d->soffU, d->swU, cu, d->hvU, d->v32, d->u32,
      d->scal);
  launch_dep<k_pc_lower<float, __half, CI, 0>>(c, n, n, d->soffL, d->swL, cl, d->hvL, d->srow,
      d->bcmask, d->u32, d->r32, d->z32, d->partial, d->scal);
}

// Rows per block of k_cg_loop and its blocks for n rows: contiguous runs of
// whole slices, one block per SM, at least kLoopMinRows rows each: a warp for
// each of the SM's four FP64 units, which take as long for one warp as for
// none beside it, and fewer blocks' sums to add.
constexpr int64_t kLoopMinRows = 128;
// its static shared memory, rounded up
constexpr size_t kLoopStatic = 4 * (kLoopThreads + 128) * 8 + 1024;
struct LoopShape {
  int per = 0;
  unsigned grid = 0;
  size_t smem = 0;
};
bool loop_shape(const xg_ctx* c, int64_t n, LoopShape* out) {
  const int64_t want = (n + c->nsm - 1) / c->nsm;
  const int64_t per = std::max<int64_t>(kLoopMinRows, (want + kSlice - 1) / kSlice * kSlice);
  out->smem = size_t(per) * 4 * sizeof(double);
  if (out->smem + kLoopStatic > c->smem) return false;
  out->per = static_cast<int>(per);
  out->grid = static_cast<unsigned>((n + per - 1) / per);
  return true;
}

// The FP64 solve of a small system by k_cg_cluster launches; false where it
// does not apply (rows, shared memory, or a device without such clusters).
constexpr int64_t kClusterIts = 65536;
constexpr size_t kClusterStatic = 32768;  // its static shared memory, rounded up
bool cluster_shape(const xg_ctx* c, const CGDev* d, int* per, int* ents, size_t* smem) {
  if (d->n > kClusterRows || d->n < kClusterSize * kSlice || c->cluster != 1) return false;
  *per = static_cast<int>((d->n + kClusterSize * kSlice - 1) / (kClusterSize * kSlice)) * kSlice;
  *ents = d->wmax * *per;
  *smem = size_t(*per) * 5 * sizeof(double) + size_t(*ents) * (sizeof(double) + sizeof(uint32_t));
  return *smem + kClusterStatic <= c->smem;
}
int cluster_solve(xg_ctx* c, CGDev* d, int per, int ents, size_t smem, CGScalars* h) {
  cudaStream_t s = c->stream;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kClusterSize);
  cfg.blockDim = dim3(kClusterThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kClusterSize;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const int64_t its = d->launch_its ? d->launch_its : kClusterIts;
  for (;;) {
    XG_CUDA(c, cudaLaunchKernelEx(&cfg, k_cg_cluster, d->n, per, ents, its,
                                  static_cast<const int32_t*>(d->soff),
                                  static_cast<const int32_t*>(d->swidth),
                                  static_cast<const int32_t*>(d->col),
                                  static_cast<const double*>(d->a),
                                  static_cast<const double*>(d->d), d->r, d->z, d->p[0], d->x,
                                  d->scal));
    const int rc = read_scal(c, d, h);
    if (rc) return rc;
    if (h->done) return XG_OK;
  }
}

// The FP64 solve by k_cg_loop launches of at most kLoopIts iterations (a
// launch is bounded in time; the state goes through global memory between
// launches).
constexpr int64_t kLoopIts = 8192;
template <class CI>
int loop_solve(xg_ctx* c, CGDev* d, const LoopShape& sh, CI ci, CGScalars* h) {
  cudaStream_t s = c->stream;
  XG_CUDA(c, allow_smem<k_cg_loop<CI>>(c, c->smem - kLoopStatic));
  int64_t n = d->n, its = d->launch_its ? d->launch_its : kLoopIts;
  int per = sh.per;
  const double *a = d->a, *dd = d->d;
  void* args[] = {&n,    &per,  &its,     &d->soff, &d->swidth, &ci,         &a,      &dd,
                  &d->r, &d->z, &d->p[0], &d->x,    &d->lpart,  &d->larrive, &d->scal};
  for (;;) {
    XG_CUDA(c, cudaMemsetAsync(d->larrive, 0, sizeof(unsigned int), s));
    XG_CUDA(c, cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_cg_loop<CI>),
                                           dim3(sh.grid), dim3(kLoopThreads), args, sh.smem, s));
    int rc = read_scal(c, d, h);
    if (rc) return rc;
    if (h->err) {
      d->ready = false;  // the vectors are of no iteration: a new init is due
      h->err = 0;
      rc = write_scal(c, d, h);
      return rc ? rc : fail(c, XG_ERR_DEVICE, "cg_solve: a grid barrier timed out");
    }
    if (h->done) return XG_OK;
  }
}

int cg_iterate(xg_ctx* c, CGDev* d, int64_t maxit, double tol, CGScalars* h) {
  cudaStream_t s = c->stream;
  // tol and maxit into the device scalars without touching the rest
  XG_CUDA(c, cudaMemcpyAsync(&d->scal->tol, &tol, sizeof(double), cudaMemcpyHostToDevice, s));
  XG_CUDA(c, cudaMemcpyAsync(&d->scal->maxit, &maxit, sizeof(int64_t), cudaMemcpyHostToDevice, s));
  const int64_t n = d->n;
  int per = 0, ents = 0;
  size_t smem = 0;
  if (d->pc != 2 && cluster_shape(c, d, &per, &ents, &smem))
    return cluster_solve(c, d, per, ents, smem, h);
  LoopShape sh;
  if (d->pc != 2 && loop_shape(c, n, &sh))
    return d->use16 ? loop_solve(c, d, sh, Cols16{d->col16}, h)
                    : loop_solve(c, d, sh, Cols32{d->col}, h);
  for (;;) {
    for (int k = 0; k < kBatch; ++k) {
      double* p0 = d->p[0];
      launch_dep<k_cg_p<double>>(c, n, n, d->z, p0, d->scal);
      launch_dep<k_cg_a<double, double, Cols32>>(c, n, n, d->soff, d->swidth, Cols32{d->col},
          d->a, p0, d->q, d->partial, d->scal);
      if (d->pc == 2) {
        launch_dep<k_cg_b<double, true>>(c, n, n, d->q, d->d, p0, d->srow, d->r, d->z,
            d->v, d->x, d->partial, d->scal);
        launch_dep<k_pc_upper<double, float, Cols32>>(c, n, n, d->soffU, d->swU, Cols32{d->colU},
            d->nvU, d->v, d->u, d->scal);
        launch_dep<k_pc_lower<double, float, Cols32, 1>>(c, n, n, d->soffL, d->swL, Cols32{d->colL},
            d->nvL, d->srow, d->bcmask, d->u, d->r, d->z, d->partial, d->scal);
      } else {
        launch_dep<k_cg_b<double, false>>(c, n, n, d->q, d->d, p0, d->srow, d->r, d->z,
            d->v, d->x, d->partial, d->scal);
      }
    }
    XG_CHECK_LAUNCH(c);
    int rc = read_scal(c, d, h);
    if (rc) return rc;
    if (h->done) break;
  }
  return XG_OK;
}

// The mixed solve's FP32 iterations up to the next residual replacement, by
// k_mixed_loop launches of at most kLoopIts iterations.
constexpr int kMixMinSlices = 4;  // slices per block at least: fewer blocks meet sooner
template <class CI, bool FACTOR>
int mixed_loop(xg_ctx* c, CGDev* d, CI ca, CI cu, CI cl, CGScalars* h) {
  cudaStream_t s = c->stream;
  const int64_t its = d->launch_its ? d->launch_its : kLoopIts;
  MixArgs<CI> A{d->n,     its,      d->soff, d->swidth, d->soffU, d->swU,  d->soffL,
                d->swL,   ca,       cu,      cl,        d->a32,   d->hvU,  d->hvL,
                d->rs32,  d->msrow, d->d32,  d->z32,    d->p32,
                d->q32,   d->r32,   d->v32,  d->u32,    d->zp32,  d->vt32, d->e64,
                d->lpart, d->larrive, d->scal};
  constexpr size_t smem = size_t(kMixThreads / 32) * SliceWalk<CI, float, kMixFull>::kBytes;
  constexpr auto kernel = k_mixed_loop<CI, FACTOR>;
  XG_CUDA(c, allow_smem<kernel>(c, smem));
  const int64_t ns = (d->n + kSlice - 1) / kSlice;
  const unsigned grid = static_cast<unsigned>(
      std::min<int64_t>(c->nsm, (ns + kMixMinSlices - 1) / kMixMinSlices));
  void* args[] = {&A};
  for (;;) {
    XG_CUDA(c, cudaMemsetAsync(d->larrive, 0, sizeof(unsigned int), s));
    XG_CUDA(c, cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(kernel), dim3(grid),
                                           dim3(kMixThreads), args, smem, s));
    int rc = read_scal(c, d, h);
    if (rc) return rc;
    if (h->err) {
      d->ready = false;  // the vectors are of no iteration: a new init is due
      h->err = 0;
      rc = write_scal(c, d, h);
      return rc ? rc : fail(c, XG_ERR_DEVICE, "cg_solve_mixed: a grid barrier timed out");
    }
    if (h->done) return XG_OK;
  }
}
template <class CI>
int mixed_loop(xg_ctx* c, CGDev* d, CI ca, CI cu, CI cl, CGScalars* h) {
  return d->pc == 2 ? mixed_loop<CI, true>(c, d, ca, cu, cl, h)
                    : mixed_loop<CI, false>(c, d, ca, cu, cl, h);
}

// True residual into the FP32 iteration (and the factor passes for z32).
int replace_residual(xg_ctx* c, CGDev* d, int first) {
  cudaStream_t s = c->stream;
  const int64_t n = d->n;
  k_outer_res<<<pgrid<k_outer_res>(c, n), kBlock, 0, s>>>(
      n, d->soff, d->swidth, d->col, d->a, d->x, d->b, d->d32, d->pc == 2 ? d->srow : nullptr,
      d->r32, d->z32, d->v32, first, d->partial, d->scal);
  XG_CHECK_LAUNCH(c);
  if (d->pc == 2) {
    if (d->use16)
      factor_apply32(c, d, Cols16{d->colU16}, Cols16{d->colL16});
    else
      factor_apply32(c, d, Cols32{d->colU}, Cols32{d->colL});
    XG_CHECK_LAUNCH(c);
  }
  return XG_OK;
}


// Whether a cluster of kClusterSize blocks of k_cg_cluster with the shared
// memory of its largest system can be resident on the context's device (a query,
// nothing runs), and the permission for such a cluster there: a kernel's
// attributes are per device.
bool cluster_ok(const xg_ctx* c) {
  if (cudaFuncSetAttribute(k_cg_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) !=
      cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  if (c->smem <= kClusterStatic) return false;
  const size_t most = c->smem - kClusterStatic;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kClusterSize);
  cfg.blockDim = dim3(kClusterThreads);
  cfg.dynamicSmemBytes = most;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = kClusterSize;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int num = 0;
  if (allow_smem<k_cg_cluster>(c, most) != cudaSuccess ||
      cudaOccupancyMaxActiveClusters(&num, k_cg_cluster, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  return num > 0;
}

}  // namespace

int cg_graph(xg_ctx* c, LpcGraph* g) {
  CGDev* d = c->cg;
  if (!d || !d->ready) return fail(c, XG_ERR_STATE, "learned preconditioner: no initialised CG system");
  if (!d->geom_set) {
    int rc = build_geom(c, d);
    if (rc) return rc;
  }
  *g = graph_of(d);
  return XG_OK;
}

int cg_set_dirichlet(xg_ctx* c, const uint8_t* mask, const double* val) {
  CGDev* d = c->cg;
  if (!d) return fail(c, XG_ERR_STATE, "pressure Dirichlet data before cg_setup");
  const int64_t n = d->n;
  uint64_t key = 1469598103934665603ull;  // FNV-1a over the mask, as xg_cg_init
  for (int64_t i = 0; i < n; ++i) key = (key ^ mask[i]) * 1099511628211ull;
  XG_CUDA(c, cudaMemcpyAsync(d->bcmask, mask, n, cudaMemcpyHostToDevice, c->stream));
  XG_CUDA(c, cudaMemcpyAsync(d->bcval, val, n * 8, cudaMemcpyHostToDevice, c->stream));
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  if (key != d->bc_key || !d->ready) {
    d->geom_set = false;
    d->factor_set = false;
  }
  d->bc_key = key;
  return XG_OK;
}

int cg_zero_solution(xg_ctx* c) {
  CGDev* d = c->cg;
  if (!d) return fail(c, XG_ERR_STATE, "cg_zero_solution before cg_setup");
  XG_CUDA(c, cudaMemsetAsync(d->x, 0, d->n * 8, c->stream));
  return XG_OK;
}

int cg_init_device(xg_ctx* c, const double* b_dev, int zero_values, int pc) {
  CGDev* d = c->cg;
  if (!d) return fail(c, XG_ERR_STATE, "cg_init_device before cg_setup");
  if (pc != 0 && pc != 1 && pc != 2) return fail(c, XG_ERR_ARG, "unknown preconditioner");
  cudaStream_t s = c->stream;
  const int64_t n = d->n;
  XG_CUDA(c, cudaMemcpyAsync(d->b, b_dev, n * 8, cudaMemcpyDeviceToDevice, s));
  const double* val = d->bcval;
  if (zero_values) {  // r is free until k_setup writes it
    XG_CUDA(c, cudaMemsetAsync(d->r, 0, n * 8, s));
    val = d->r;
  }
  d->pc = pc;
  d->apply = true;
  k_apply_bc<<<blocks_for(n, kBlock), kBlock, 0, s>>>(n, d->soff, d->swidth, d->col, d->a0, d->a,
                                                       d->a32, d->bcmask, val, nullptr, d->b);
  XG_CHECK_LAUNCH(c);
  k_row_sums<<<blocks_for(n, kBlock), kBlock, 0, s>>>(n, d->soff, d->swidth, d->col, d->a,
                                                      d->rs32);
  XG_CHECK_LAUNCH(c);
  CGScalars h{};
  h.pc = pc;
  h.guard = d->guard;
  XG_CUDA(c, cudaMemcpyAsync(d->scal, &h, sizeof(h), cudaMemcpyHostToDevice, s));
  k_setup<<<pgrid<k_setup>(c, n), kBlock, 0, s>>>(n, d->soff, d->swidth, d->col, d->a, d->diagpos,
                                               d->x, d->b, d->r, d->d, d->z, d->p[0], d->d32,
                                               d->partial, d->scal);
  XG_CHECK_LAUNCH(c);
  d->ready = true;
  if (pc == 2) {
    int rf = d->factor_set ? XG_OK : build_factor(c, d);
    if (rf) return rf;
    rf = factor_apply64(c, d, d->r, d->z);
    if (rf) return rf;
  }
  return XG_OK;
}

const double* cg_solution_device(xg_ctx* c) { return c->cg ? c->cg->x : nullptr; }
int64_t cg_rows(xg_ctx* c) { return c->cg ? c->cg->n : 0; }

// Values in CSR order, on the row pattern ia (zero-based, the pattern the
// context's system was set up with), into that system's SELL-32 layout: entry
// j of row i at soff[i / 32] + (j - ia[i]) 32 + i % 32, with the slice widths
// xg_cg_setup forms; padding entries 0.  dev_out holds nent() doubles.
int cg_to_sell(xg_ctx* c, const uint64_t* ia, const double* csr, double* dev_out) {
  CGDev* d = c->cg;
  if (!d) return fail(c, XG_ERR_STATE, "cg_to_sell before cg_setup");
  const int64_t nrow = d->n, nslice = (nrow + kSlice - 1) / kSlice;
  std::vector<int64_t> soff(nslice + 1, 0);
  for (int64_t s = 0; s < nslice; ++s) {
    uint64_t w = 0;
    for (int64_t i = s * kSlice; i < std::min(nrow, (s + 1) * kSlice); ++i)
      w = std::max<uint64_t>(w, ia[i + 1] - ia[i]);
    soff[s + 1] = soff[s] + int64_t(w) * kSlice;
  }
  if (soff[nslice] != d->nent) return fail(c, XG_ERR_ARG, "cg_to_sell: pattern mismatch");
  std::vector<double> v(static_cast<size_t>(d->nent), 0.0);
  for (int64_t i = 0; i < nrow; ++i) {
    const int64_t s = i / kSlice, lane = i % kSlice;
    for (uint64_t j = ia[i]; j < ia[i + 1]; ++j)
      v[soff[s] + int64_t(j - ia[i]) * kSlice + lane] = csr[j];
  }
  XG_CUDA(c, upload(c, dev_out, v.data(), v.size() * 8));
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  return XG_OK;
}
int64_t cg_nent(xg_ctx* c) { return c->cg ? c->cg->nent : 0; }
// The working values the solves read are formed from these originals.
double* cg_values_device(xg_ctx* c) { return c->cg ? c->cg->a0 : nullptr; }

}  // namespace xg

using namespace xg;

extern "C" {

int xg_cg_setup(xg_ctx* c, int64_t nrow, const uint64_t* ia, const uint64_t* ja, const double* a,
                int base) {
  XG_HOST_TRY
  int rc = use(c);
  if (rc) return rc;
  if (nrow <= 0 || !ia || !ja || !a || (base != 0 && base != 1))
    return fail(c, XG_ERR_ARG, "cg_setup: bad matrix");
  if (nrow >= (int64_t(1) << 31) - 64) return fail(c, XG_ERR_ARG, "cg_setup: too many rows");
  const uint64_t b0 = static_cast<uint64_t>(base);
  if (ia[0] != b0) return fail(c, XG_ERR_ARG, "cg_setup: ia[0] must equal the index base");
  std::vector<int32_t> diagk(nrow, -1);
  bool fits16 = true;
  for (int64_t i = 0; i < nrow; ++i) {
    if (ia[i + 1] < ia[i]) return fail(c, XG_ERR_ARG, "cg_setup: ia not monotonic");
    for (uint64_t j = ia[i]; j < ia[i + 1]; ++j) {
      uint64_t cc = ja[j - b0] - b0;
      if (cc >= static_cast<uint64_t>(nrow)) return fail(c, XG_ERR_ARG, "cg_setup: column id");
      if (static_cast<int64_t>(cc) == i) diagk[i] = static_cast<int32_t>(j - ia[i]);
      const int64_t dl = static_cast<int64_t>(cc) - i;
      if (dl <= int64_t(kPad16) || dl > int64_t(std::numeric_limits<int16_t>::max()))
        fits16 = false;
    }
    if (diagk[i] < 0) return fail(c, XG_ERR_ARG, "cg_setup: row without diagonal entry");
  }
  if (c->cluster < 0) c->cluster = cluster_ok(c) ? 1 : 0;
  const int64_t nslice = (nrow + kSlice - 1) / kSlice;
  std::vector<int32_t> soff(nslice + 1), sw(nslice);
  int64_t tot = 0;
  for (int64_t s = 0; s < nslice; ++s) {
    uint64_t w = 0;
    for (int64_t i = s * kSlice; i < std::min(nrow, (s + 1) * kSlice); ++i)
      w = std::max<uint64_t>(w, ia[i + 1] - ia[i]);
    sw[s] = static_cast<int32_t>(w);
    soff[s] = static_cast<int32_t>(tot);
    tot += int64_t(w) * kSlice;
    if (tot >= (int64_t(1) << 31)) return fail(c, XG_ERR_ARG, "cg_setup: matrix too large");
  }
  soff[nslice] = static_cast<int32_t>(tot);
  std::vector<int32_t> col(tot, kPad), dpos(nrow);
  std::vector<int16_t> col16(fits16 ? tot : 0, kPad16);
  std::vector<double> val(tot, 0.0);
  for (int64_t i = 0; i < nrow; ++i) {
    const int64_t s = i / kSlice, lane = i % kSlice;
    for (uint64_t j = ia[i]; j < ia[i + 1]; ++j) {
      const int64_t k = int64_t(j - ia[i]);
      const int64_t e = soff[s] + k * kSlice + lane;
      col[e] = static_cast<int32_t>(ja[j - b0] - b0);
      if (fits16) col16[e] = static_cast<int16_t>(col[e] - i);
      val[e] = a[j - b0];
    }
    dpos[i] = static_cast<int32_t>(soff[s] + int64_t(diagk[i]) * kSlice + lane);
  }
  // lower / upper triangles (off-diagonal) as SELL-32, rows sorted by column;
  // posL: the full-layout index of each lower entry; tposU: the upper-layout
  // index of its transposed entry (j,i)
  std::vector<int32_t> soffL(nslice + 1), swL(nslice), soffU(nslice + 1), swU(nslice);
  int64_t totL = 0, totU = 0;
  for (int64_t s2 = 0; s2 < nslice; ++s2) {
    int64_t wl = 0, wu = 0;
    for (int64_t i = s2 * kSlice; i < std::min(nrow, (s2 + 1) * kSlice); ++i) {
      int64_t nl = 0, nu = 0;
      for (uint64_t j = ia[i]; j < ia[i + 1]; ++j) {
        const int64_t cc = int64_t(ja[j - b0] - b0);
        if (cc < i) ++nl;
        if (cc > i) ++nu;
      }
      wl = std::max(wl, nl);
      wu = std::max(wu, nu);
    }
    swL[s2] = int32_t(wl);
    swU[s2] = int32_t(wu);
    soffL[s2] = int32_t(totL);
    soffU[s2] = int32_t(totU);
    totL += wl * kSlice;
    totU += wu * kSlice;
  }
  soffL[nslice] = int32_t(totL);
  soffU[nslice] = int32_t(totU);
  std::vector<int32_t> colL(std::max<int64_t>(1, totL), kPad), posL(std::max<int64_t>(1, totL), 0),
      colU(std::max<int64_t>(1, totU), kPad), tposU(std::max<int64_t>(1, totL), 0);
  std::vector<int16_t> colL16(fits16 ? colL.size() : 0, kPad16),
      colU16(fits16 ? colU.size() : 0, kPad16);
  for (int64_t i = 0; i < nrow; ++i) {
    const int64_t s2 = i / kSlice, lane = i % kSlice;
    int64_t kl = 0, ku = 0;
    for (uint64_t j = ia[i]; j < ia[i + 1]; ++j) {
      const int64_t cc = int64_t(ja[j - b0] - b0);
      const int64_t kfull = int64_t(j - ia[i]);
      if (cc < i) {
        const int64_t e = soffL[s2] + kl * kSlice + lane;
        colL[e] = int32_t(cc);
        if (fits16) colL16[e] = int16_t(cc - i);
        posL[e] = int32_t(soff[s2] + kfull * kSlice + lane);
        ++kl;
      } else if (cc > i) {
        const int64_t e = soffU[s2] + ku * kSlice + lane;
        colU[e] = int32_t(cc);
        if (fits16) colU16[e] = int16_t(cc - i);
        ++ku;
      }
    }
  }
  for (int64_t i = 0; i < nrow; ++i) {
    const int64_t s2 = i / kSlice, lane = i % kSlice;
    int64_t kl = 0;
    for (uint64_t j = ia[i]; j < ia[i + 1]; ++j) {
      const int64_t cc = int64_t(ja[j - b0] - b0);
      if (cc >= i) continue;
      // position of column i in row cc's upper list (rows sorted by column)
      const int64_t s3 = cc / kSlice, lane3 = cc % kSlice;
      int64_t ku = 0;
      bool found = false;
      for (uint64_t jj = ia[cc]; jj < ia[cc + 1]; ++jj) {
        const int64_t c3 = int64_t(ja[jj - b0] - b0);
        if (c3 <= cc) continue;
        if (c3 == i) {
          found = true;
          break;
        }
        ++ku;
      }
      if (!found) return fail(c, XG_ERR_ARG, "cg_setup: matrix graph is not symmetric");
      tposU[soffL[s2] + kl * kSlice + lane] = int32_t(soffU[s3] + ku * kSlice + lane3);
      ++kl;
    }
  }
  if (c->cg) {
    XG_CUDA(c, cudaStreamSynchronize(c->stream));
    destroy_cg(c->cg);
    c->cg = nullptr;
  }
  auto* d = new CGDev;
  c->cg = d;
  d->n = nrow;
  d->nslice = nslice;
  d->nent = tot;
  d->use16 = fits16;
  d->wmax = *std::max_element(sw.begin(), sw.end());
  d->maxgrid = int64_t(c->nsm) * (2048 / kBlock);
  for (int pass = 0; pass < 2; ++pass) {
    Arena& A = d->arena;
    A.plan(d->soff, nslice + 1);
    A.plan(d->swidth, nslice);
    A.plan(d->col, tot);
    A.plan(d->col16, fits16 ? tot : 1);
    A.plan(d->a0, tot);
    A.plan(d->a, tot);
    A.plan(d->a32, tot);
    A.plan(d->rs32, nrow);
    A.plan(d->diagpos, nrow);
    A.plan(d->bcmask, nrow);
    A.plan(d->bcval, nrow);
    A.plan(d->x, nrow);
    A.plan(d->b, nrow);
    A.plan(d->r, nrow);
    A.plan(d->q, nrow);
    A.plan(d->z, nrow);
    A.plan(d->d, nrow);
    A.plan(d->p[0], nrow);
    A.plan(d->p[1], nrow);
    A.plan(d->r32, nrow);
    A.plan(d->q32, nrow);
    A.plan(d->z32, nrow);
    A.plan(d->d32, nrow);
    A.plan(d->e64, nrow);
    A.plan(d->p32, nrow);
    A.plan(d->zp32, nrow);
    A.plan(d->vt32, nrow);
    A.plan(d->partial, 3 * d->maxgrid);
    A.plan(d->scal, 1);
    A.plan(d->lpart, size_t(6) * c->nsm);
    A.plan(d->larrive, 1);
    A.plan(d->soffL, nslice + 1);
    A.plan(d->swL, nslice);
    A.plan(d->colL, colL.size());
    A.plan(d->colL16, fits16 ? colL.size() : 1);
    A.plan(d->posL, posL.size());
    A.plan(d->tposU, tposU.size());
    A.plan(d->soffU, nslice + 1);
    A.plan(d->swU, nslice);
    A.plan(d->colU, colU.size());
    A.plan(d->colU16, fits16 ? colU.size() : 1);
    A.plan(d->nvL, colL.size());
    A.plan(d->nvU, colU.size());
    A.plan(d->hvL, colL.size());
    A.plan(d->hvU, colU.size());
    A.plan(d->eL, colL.size());
    A.plan(d->eU, colU.size());
    A.plan(d->eF, tot);
    A.plan(d->srow, nrow);
    A.plan(d->msrow, nrow);
    A.plan(d->v, nrow);
    A.plan(d->u, nrow);
    A.plan(d->t, nrow);
    A.plan(d->v32, nrow);
    A.plan(d->u32, nrow);
    if (pass == 0) {
      cudaError_t e = A.reserve();
      if (e != cudaSuccess) {
        destroy_cg(d);
        c->cg = nullptr;
        return fail(c, XG_ERR_CUDA, std::string("cg_setup: ") + cudaGetErrorString(e));
      }
    }
  }
  cudaStream_t s = c->stream;
  XG_CUDA(c, cudaMemcpyAsync(d->soff, soff.data(), soff.size() * 4, cudaMemcpyHostToDevice, s));
  XG_CUDA(c, cudaMemcpyAsync(d->swidth, sw.data(), sw.size() * 4, cudaMemcpyHostToDevice, s));
  XG_CUDA(c, cudaMemcpyAsync(d->col, col.data(), col.size() * 4, cudaMemcpyHostToDevice, s));
  if (fits16)
    XG_CUDA(c, cudaMemcpyAsync(d->col16, col16.data(), col16.size() * 2, cudaMemcpyHostToDevice, s));
  XG_CUDA(c, cudaMemcpyAsync(d->a0, val.data(), val.size() * 8, cudaMemcpyHostToDevice, s));
  XG_CUDA(c, cudaMemcpyAsync(d->diagpos, dpos.data(), dpos.size() * 4, cudaMemcpyHostToDevice, s));
  d->nentL = totL;
  d->nentU = totU;
  XG_CUDA(c, cudaMemcpyAsync(d->soffL, soffL.data(), soffL.size() * 4, cudaMemcpyHostToDevice, s));
  XG_CUDA(c, cudaMemcpyAsync(d->swL, swL.data(), swL.size() * 4, cudaMemcpyHostToDevice, s));
  XG_CUDA(c, cudaMemcpyAsync(d->colL, colL.data(), colL.size() * 4, cudaMemcpyHostToDevice, s));
  XG_CUDA(c, cudaMemcpyAsync(d->posL, posL.data(), posL.size() * 4, cudaMemcpyHostToDevice, s));
  XG_CUDA(c, cudaMemcpyAsync(d->tposU, tposU.data(), tposU.size() * 4, cudaMemcpyHostToDevice, s));
  XG_CUDA(c, cudaMemcpyAsync(d->soffU, soffU.data(), soffU.size() * 4, cudaMemcpyHostToDevice, s));
  XG_CUDA(c, cudaMemcpyAsync(d->swU, swU.data(), swU.size() * 4, cudaMemcpyHostToDevice, s));
  XG_CUDA(c, cudaMemcpyAsync(d->colU, colU.data(), colU.size() * 4, cudaMemcpyHostToDevice, s));
  if (fits16) {
    XG_CUDA(c, cudaMemcpyAsync(d->colL16, colL16.data(), colL16.size() * 2, cudaMemcpyHostToDevice,
                               s));
    XG_CUDA(c, cudaMemcpyAsync(d->colU16, colU16.data(), colU16.size() * 2, cudaMemcpyHostToDevice,
                               s));
  }
  XG_CUDA(c, cudaMemsetAsync(d->nvL, 0, colL.size() * 4, s));
  XG_CUDA(c, cudaMemsetAsync(d->nvU, 0, colU.size() * 4, s));
  XG_CUDA(c, cudaMemsetAsync(d->hvL, 0, colL.size() * 2, s));
  XG_CUDA(c, cudaMemsetAsync(d->hvU, 0, colU.size() * 2, s));
  XG_CUDA(c, cudaMemsetAsync(d->eU, 0, colU.size() * 4, s));
  XG_CUDA(c, cudaMemsetAsync(d->x, 0, nrow * 8, s));
  XG_CUDA(c, cudaMemsetAsync(d->b, 0, nrow * 8, s));
  XG_CUDA(c, cudaMemsetAsync(d->bcmask, 0, nrow, s));
  XG_CUDA(c, cudaMemsetAsync(d->scal, 0, sizeof(CGScalars), s));
  k_copy_values<<<blocks_for(tot, kBlock), kBlock, 0, s>>>(tot, d->a0, d->a, d->a32);
  XG_CHECK_LAUNCH(c);
  k_row_sums<<<blocks_for(nrow, kBlock), kBlock, 0, s>>>(nrow, d->soff, d->swidth, d->col, d->a,
                                                         d->rs32);
  XG_CHECK_LAUNCH(c);
  XG_CUDA(c, cudaStreamSynchronize(s));
  return XG_OK;
  XG_HOST_CATCH(c)
}

int xg_cg_mult(xg_ctx* c, const double* x, double* y) {
  int rc = use(c);
  if (rc) return rc;
  CGDev* d = c->cg;
  if (!d) return fail(c, XG_ERR_STATE, "cg_mult before cg_setup");
  if (!x || !y) return fail(c, XG_ERR_ARG, "cg_mult: null vector");
  XG_CUDA(c, cudaMemcpyAsync(d->r, x, d->n * 8, cudaMemcpyHostToDevice, c->stream));
  k_spmv<<<pgrid<k_spmv>(c, d->n), kBlock, 0, c->stream>>>(d->n, d->soff, d->swidth, d->col, d->a0,
                                                        d->r, d->q);
  XG_CHECK_LAUNCH(c);
  XG_CUDA(c, cudaMemcpyAsync(y, d->q, d->n * 8, cudaMemcpyDeviceToHost, c->stream));
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  return XG_OK;
}

int xg_cg_init(xg_ctx* c, const double* x, const double* b, const double* neubc, int64_t ndir,
               const uint64_t* dirnodes, const double* dirvals, int apply, int pc) {
  XG_HOST_TRY
  int rc = use(c);
  if (rc) return rc;
  CGDev* d = c->cg;
  if (!d) return fail(c, XG_ERR_STATE, "cg_init before cg_setup");
  if (pc != 0 && pc != 1 && pc != 2) return fail(c, XG_ERR_ARG, "cg_init: unknown preconditioner");
  if (ndir && (!dirnodes || !dirvals)) return fail(c, XG_ERR_ARG, "cg_init: null Dirichlet data");
  cudaStream_t s = c->stream;
  const int64_t n = d->n;
  if (x) XG_CUDA(c, cudaMemcpyAsync(d->x, x, n * 8, cudaMemcpyHostToDevice, s));
  if (b) XG_CUDA(c, cudaMemcpyAsync(d->b, b, n * 8, cudaMemcpyHostToDevice, s));
  d->pc = pc;
  d->apply = apply != 0;
  // the working matrix depends on the Dirichlet node set only: its scales,
  // couplings and factor survive re-initialisations with the same set (a
  // pressure solve per time step)
  uint64_t key = 1469598103934665603ull;  // FNV-1a over the mask, 0 without BCs
  if (d->apply) {
    std::vector<uint8_t> mask(n, 0);
    std::vector<double> val(n, 0.0);
    for (int64_t k = 0; k < ndir; ++k) {
      if (dirnodes[k] >= static_cast<uint64_t>(n))
        return fail(c, XG_ERR_ARG, "cg_init: Dirichlet node out of range");
      mask[dirnodes[k]] = 1;
      val[dirnodes[k]] = dirvals[k];
    }
    for (int64_t i = 0; i < n; ++i) key = (key ^ mask[i]) * 1099511628211ull;
    XG_CUDA(c, cudaMemcpyAsync(d->bcmask, mask.data(), n, cudaMemcpyHostToDevice, s));
    XG_CUDA(c, cudaMemcpyAsync(d->bcval, val.data(), n * 8, cudaMemcpyHostToDevice, s));
    double* neu = nullptr;
    if (neubc) {
      XG_CUDA(c, cudaMemcpyAsync(d->q, neubc, n * 8, cudaMemcpyHostToDevice, s));
      neu = d->q;
    }
    k_apply_bc<<<blocks_for(n, kBlock), kBlock, 0, s>>>(n, d->soff, d->swidth, d->col, d->a0,
                                                         d->a, d->a32, d->bcmask, d->bcval, neu,
                                                         d->b);
    XG_CHECK_LAUNCH(c);
    // mask and val are host vectors of this frame: complete their copies
    XG_CUDA(c, cudaStreamSynchronize(s));
  } else {
    key = 0;
    XG_CUDA(c, cudaMemsetAsync(d->bcmask, 0, n, s));
    k_copy_values<<<blocks_for(d->nent, kBlock), kBlock, 0, s>>>(d->nent, d->a0, d->a, d->a32);
    XG_CHECK_LAUNCH(c);
  }
  k_row_sums<<<blocks_for(n, kBlock), kBlock, 0, s>>>(n, d->soff, d->swidth, d->col, d->a,
                                                      d->rs32);
  XG_CHECK_LAUNCH(c);
  if (key != d->bc_key || !d->ready) {
    d->geom_set = false;
    d->factor_set = false;
  }
  d->bc_key = key;
  CGScalars h{};
  h.pc = pc;
  h.guard = d->guard;
  XG_CUDA(c, cudaMemcpyAsync(d->scal, &h, sizeof(h), cudaMemcpyHostToDevice, s));
  k_setup<<<pgrid<k_setup>(c, n), kBlock, 0, s>>>(n, d->soff, d->swidth, d->col, d->a, d->diagpos,
                                               d->x, d->b, d->r, d->d, d->z, d->p[0], d->d32,
                                               d->partial, d->scal);
  XG_CHECK_LAUNCH(c);
  if (pc == 2) {
    int rf = d->factor_set ? XG_OK : build_factor(c, d);
    if (rf) return rf;
    rf = factor_apply64(c, d, d->r, d->z);
    if (rf) return rf;
  }
  XG_CUDA(c, cudaStreamSynchronize(s));
  d->ready = true;
  return XG_OK;
  XG_HOST_CATCH(c)
}

int xg_cg_solve(xg_ctx* c, int64_t maxit, double tol, int64_t* it, double* normr,
                double* normb, int* converged) {
  int rc = use(c);
  if (rc) return rc;
  CGDev* d = c->cg;
  if (!d || !d->ready) return fail(c, XG_ERR_STATE, "cg_solve before cg_init");
  if (maxit <= 0 || !(tol >= 0)) return fail(c, XG_ERR_ARG, "cg_solve: bad maxit/tol");
  CGScalars h{};
  rc = cg_iterate(c, d, maxit, tol, &h);
  if (rc) return rc;
  d->last_it = h.it;
  d->last_normr = std::sqrt(h.rr);
  d->last_normb = h.normb;
  d->last_conv = h.converged;
  if (it) *it = h.it;
  if (normr) *normr = std::sqrt(h.rr);
  if (normb) *normb = h.normb;
  if (converged) *converged = h.converged;
  return XG_OK;
}

int xg_cg_solve_mixed(xg_ctx* c, int64_t maxit, double tol, double inner_tol,
                      int64_t inner_maxit, int64_t* outer, int64_t* inner, double* normr,
                      double* normb, int* converged) {
  int rc = use(c);
  if (rc) return rc;
  CGDev* d = c->cg;
  if (!d || !d->ready) return fail(c, XG_ERR_STATE, "cg_solve_mixed before cg_init");
  if (maxit <= 0 || inner_maxit <= 0 || !(tol >= 0) || !(inner_tol > 0) || !(inner_tol < 1))
    return fail(c, XG_ERR_ARG, "cg_solve_mixed: bad limits");
  cudaStream_t s = c->stream;
  CGScalars h{};
  rc = read_scal(c, d, &h);
  if (rc) return rc;
  const double nb0 = h.normb > 1.0e-14 ? h.normb : 1.0;
  XG_CUDA(c, cudaMemsetAsync(d->e64, 0, d->n * 8, s));
  // the first FP32 iteration reads p with weight beta = 0: make it finite
  XG_CUDA(c, cudaMemsetAsync(d->p32, 0, d->n * 4, s));
  rc = replace_residual(c, d, 1);
  if (rc) return rc;
  rc = read_scal(c, d, &h);
  if (rc) return rc;
  double nr = std::sqrt(h.rr);
  int64_t nout = 0;
  bool conv = nr < tol * nb0;
  int breakdown = 0;
  while (!conv && nout < maxit && h.it < inner_maxit && !breakdown) {
    h.tol = tol;
    h.delta = inner_tol;
    h.rlast = nr;
    h.maxit = inner_maxit;
    h.done = 0;
    rc = write_scal(c, d, &h);
    if (rc) return rc;
    rc = d->use16 ? mixed_loop(c, d, Cols16{d->col16}, Cols16{d->colU16}, Cols16{d->colL16}, &h)
                  : mixed_loop(c, d, Cols32{d->col}, Cols32{d->colU}, Cols32{d->colL}, &h);
    if (rc) return rc;
    breakdown = h.finished;
    k_add_correction<<<blocks_for(d->n, kBlock), kBlock, 0, s>>>(d->n, d->e64, d->x);
    XG_CHECK_LAUNCH(c);
    rc = replace_residual(c, d, 0);
    if (rc) return rc;
    rc = read_scal(c, d, &h);
    if (rc) return rc;
    nr = std::sqrt(h.rr);
    ++nout;
    conv = nr < tol * nb0;
  }
  d->last_it = h.it;
  d->last_normr = nr;
  d->last_normb = nb0;
  d->last_conv = conv;
  if (outer) *outer = nout;
  if (inner) *inner = h.it;
  if (normr) *normr = nr;
  if (normb) *normb = nb0;
  if (converged) *converged = conv ? 1 : 0;
  return XG_OK;
}

int xg_cg_set_factor(xg_ctx* c, xg_lpc* model, double scale) {
  int rc = use(c);
  if (rc) return rc;
  CGDev* d = c->cg;
  if (!d) return fail(c, XG_ERR_STATE, "cg_set_factor before cg_setup");
  d->factor_model = model;
  d->factor_c = scale;
  d->factor_set = false;
  return XG_OK;
}

int xg_cg_set_guard(xg_ctx* c, int guard) {
  int rc = use(c);
  if (rc) return rc;
  CGDev* d = c->cg;
  if (!d) return fail(c, XG_ERR_STATE, "cg_set_guard before cg_setup");
  if (guard != 0 && guard != 1) return fail(c, XG_ERR_ARG, "cg_set_guard: guard is 0 or 1");
  d->guard = guard;
  return XG_OK;
}

int xg_cg_set_launch_limit(xg_ctx* c, int64_t its) {
  int rc = use(c);
  if (rc) return rc;
  CGDev* d = c->cg;
  if (!d) return fail(c, XG_ERR_STATE, "cg_set_launch_limit before cg_setup");
  if (its < 0) return fail(c, XG_ERR_ARG, "cg_set_launch_limit: negative");
  d->launch_its = its;
  return XG_OK;
}

int xg_cg_precondition(xg_ctx* c, const double* r, double* z) {
  int rc = use(c);
  if (rc) return rc;
  CGDev* d = c->cg;
  if (!d || !d->ready) return fail(c, XG_ERR_STATE, "cg_precondition before cg_init");
  if (!r || !z) return fail(c, XG_ERR_ARG, "cg_precondition: null vector");
  cudaStream_t s = c->stream;
  XG_CUDA(c, cudaMemcpyAsync(d->q, r, d->n * 8, cudaMemcpyHostToDevice, s));
  // the passes run only while the solve is not done: save the scalars, clear
  // done, restore them afterwards
  CGScalars h{};
  rc = read_scal(c, d, &h);
  if (rc) return rc;
  CGScalars run = h;
  run.done = 0;
  rc = write_scal(c, d, &run);
  if (rc) return rc;
  if (d->pc == 2) {
    if (!d->factor_set) {
      rc = build_factor(c, d);
      if (rc) return rc;
    }
    rc = factor_apply64(c, d, d->q, d->t);
    if (rc) return rc;
  } else {
    k_jacobi_apply<<<blocks_for(d->n, kBlock), kBlock, 0, s>>>(d->n, d->q, d->d, d->t);
    XG_CHECK_LAUNCH(c);
  }
  rc = write_scal(c, d, &h);
  if (rc) return rc;
  XG_CUDA(c, cudaMemcpyAsync(z, d->t, d->n * 8, cudaMemcpyDeviceToHost, s));
  XG_CUDA(c, cudaStreamSynchronize(s));
  return XG_OK;
}

int xg_cg_solution(xg_ctx* c, double* x) {
  int rc = use(c);
  if (rc) return rc;
  CGDev* d = c->cg;
  if (!d) return fail(c, XG_ERR_STATE, "cg_solution before cg_setup");
  if (!x) return fail(c, XG_ERR_ARG, "cg_solution: null x");
  XG_CUDA(c, cudaMemcpyAsync(x, d->x, d->n * 8, cudaMemcpyDeviceToHost, c->stream));
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  return XG_OK;
}

}  // extern "C"
