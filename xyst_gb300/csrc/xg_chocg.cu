// ChoCG on one GB300: the chorin:: edge passes as node-gather kernels, the
// explicit RK momentum prediction, nodal BCs, CFL reduction and the
// pressure-increment projection around the context's CG solver.
//
// Reference path (all paths relative to the reference project root):
//   chorin::div/vgrad/grad/flux/rhs  src/Physics/Chorin.cpp:34-1044
//   ChoCG::merge/div/pinit/psolve/sgrad/psolved/pgrad
//                                    src/Inciter/ChoCG.cpp:739-764, 868-1281
//   ChoCG::BC/dt/advance/rhs/solve/pred/corr
//                                    src/Inciter/ChoCG.cpp:1333-1695
//   physics::dirbc/symbc/noslipbc    src/Physics/BC.cpp:27-145
//
// Layout in HBM (n nodes), FP64 throughout (the projection scheme is the
// configuration the reference runs in double precision):
//   u, u2, un     [3][n]  velocity (ping-pong) and the stage-0 copy
//   pr, div       [n]     pressure and the Poisson right-hand side
//   pgrad         [3][n]  pressure gradient
//   vgrad         [9][n]  velocity gradient (damp4 and the start-up flux)
//   flx           [3][n]  momentum flux (start-up only)
//   adjacency     SELL-32 over both ends of every edge, entry (k, lane) of
//                 slice s at off[s] + 32k + lane: the neighbour (~id when the
//                 node is the canonical second end) and (d0, d1, d2, d4), the
//                 dual-face normal and the viscous coefficient of the edge,
//                 plus |d| / |x_a - x_b| for the pressure damping
//   bnode, park   boundary-node list and [nb][9] domain sums between passes
// Each node owns its writes (no atomics except the scalar CFL minimum).  The
// linear edge terms and the fluxes are evaluated from the node outwards; only
// their sign changes with the orientation, to the last bit, so an edge makes no
// volume or momentum.  The damp4 reconstruction, whose regularisation depends on
// the orientation, is evaluated in the edge's canonical one.
// On GB300 an FP64 instruction holds an SM quarter's FP64 unit for 64 cycles,
// so these passes are written to their FP64 operation count, and signs are
// flipped on the bits.  A node's neighbours are
// visited in increasing id, which for an unrenumbered mesh is the order in
// which the reference's edge loop reaches the node.  Each node kernel runs
// as a domain pass over all nodes and a pass over the boundary nodes that
// adds the boundary-triangle terms (see node_of).

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>
#include <limits>
#include <string>
#include <vector>

#include "xg_fp64.cuh"
#include "xg_internal.hpp"

namespace xg {

namespace {
constexpr int kSlice = 32;
constexpr int32_t kPad = INT32_MIN;
constexpr int kBlock = 256;
// FP64 node passes run in small blocks: an SM's FP64 units take its blocks' work
// in turn, so an SM with one large block more than the others holds them up
// (and 20 blocks of 256 run a 17^3 system on 20 SMs: damp4 k_crhs 457 us).
constexpr int kNode = 64;
constexpr int kBL = 4;  // lanes per boundary node: they share its triangles
}  // namespace

// The four edge coefficients of an adjacency entry: d0, d1, d2 (dual-face
// normal) and d4 (viscous coefficient).
struct alignas(32) Coef4 {
  double x, y, z, w;
};

struct ChoCGDev {
  Arena arena;    // mesh-sized arrays
  Arena bcarena;  // boundary condition program
  int64_t n = 0, nslice = 0, nent = 0, nbn = 0;
  xg_chocg_params prm{};
  int32_t *soff = nullptr, *swidth = nullptr, *nbr = nullptr;
  Coef4* dd = nullptr;
  double* sdl = nullptr;  // per entry |d| / edge length (the pressure damping of chorin::div)
  int32_t *bidx = nullptr, *bptr = nullptr, *bent = nullptr, *btri = nullptr;
  int32_t* bnode = nullptr;  // boundary index -> node
  double* park = nullptr;    // [nbn][9] domain sums of boundary nodes between passes
  double *xyz = nullptr, *ivol = nullptr, *cbrtv = nullptr;  // coordinates, 1/vol, cbrt(vol)
  double *u = nullptr, *u2 = nullptr, *un = nullptr, *pr = nullptr, *pgrad = nullptr,
         *vgrad = nullptr, *div = nullptr, *flx = nullptr, *stage = nullptr;
  unsigned long long* dtmin = nullptr;
  // BC program, one thread per BC node
  int64_t nbc = 0, nsymbc = 0;
  int32_t *bcnode = nullptr, *bcdir = nullptr, *bcsymp = nullptr, *bcnoslip = nullptr,
          *dirmask = nullptr;
  double *dirval = nullptr, *symn = nullptr;
  bool pdir_set = false;
  double t = 0.0;
  bool ready = false;  // start-up done
  int64_t last_it = 0;
  std::vector<double> xyz_host;  // [3][n], for the momentum matrix
  // theta-implicit momentum prediction (ChoCG::lhs/solve/msolve/msolved):
  // its own CG system of 3n rows (row 3i + c), the stiffness and consistent
  // mass values on its pattern (SELL order), the rhs of the last stage
  // ([3][n]) and as the system's right-hand side (row order), and the
  // Dirichlet rows (velocity Dirichlet components and noslip nodes)
  double theta = 0.0;
  int mom_pc = 0;
  int64_t mom_iter = 10;
  double mom_tol = 1.0e-3;
  CGDev* mom = nullptr;
  Arena momarena;
  double *baseK = nullptr, *baseM = nullptr, *R3 = nullptr, *b3 = nullptr;
  std::vector<uint8_t> mommask;
  bool mommask_up = false;
  int64_t last_mit = 0;
};

void destroy_chocg(ChoCGDev* d) {
  if (d && d->mom) destroy_cg(d->mom);
  delete d;
}
size_t bytes_chocg(const ChoCGDev* d) {
  return d ? d->arena.bytes() + d->bcarena.bytes() + d->momarena.bytes() : 0;
}

namespace {

struct ChoAdj {
  const int32_t* soff;
  const int32_t* swidth;
  const int32_t* nbr;
  const Coef4* dd;
  const double* sdl;
};
struct ChoBnd {
  const int32_t* bidx;
  const int32_t* bptr;
  const int32_t* bent;  // (triangle << 2) | position of the node in it
  const int32_t* btri;
  const double* xyz;    // SoA coordinates
  const int32_t* bnode;  // boundary index -> node
  double* park;          // [nb][9]: a boundary node's domain sum between the passes
  int64_t nb;
};

// Every node kernel runs as two passes.  The domain pass (one thread per
// node) sums the edge terms; a boundary node parks that sum and returns.  The
// boundary pass (kBL lanes per boundary node, lane l of them) adds the
// boundary-triangle terms after it and applies the epilogue.  Folded into the
// domain pass, the few boundary nodes of a warp held all 32 lanes for their
// triangle loops; one lane per node was a serial chain of some 36-54 us at
// any size.  Past the last node bi and p are -1; the boundary pass's lanes
// all stay for the shuffles.
__device__ __forceinline__ void node_of(bool bnd_pass, int64_t n, const ChoBnd& b, int64_t& p,
                                        int32_t& bi, int& l) {
  const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  p = bi = -1;
  l = 0;
  if (bnd_pass) {
    l = static_cast<int>(t % kBL);
    if (t / kBL < b.nb) {
      bi = static_cast<int32_t>(t / kBL);
      p = __ldg(b.bnode + bi);
    }
  } else if (t < n) {
    p = t;
  }
}
// Adds the kBL lanes' values.
template <int N>
__device__ __forceinline__ void lane_add(double (&v)[N]) {
#pragma unroll
  for (int o = 1; o < kBL; o <<= 1)
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
}

// v, or -v when neg, on the sign bit.
__device__ __forceinline__ double flip(double v, bool neg) {
  return __longlong_as_double(__double_as_longlong(v) ^ (neg ? (1ll << 63) : 0ll));
}

__device__ __forceinline__ Coef4 ldd4(const Coef4* p) {
  const double2* q = reinterpret_cast<const double2*>(p);
  const double2 a = __ldg(q), b = __ldg(q + 1);
  return Coef4{a.x, a.y, b.x, b.y};
}

// Boundary-face normal / 48 of triangle t (tk::crossdiv(..., 6.0),
// src/Base/Vector.hpp:68-77, with the 1/8 of the vertex weights
// (6 f_own + f_other + f_other)/8, Chorin.cpp:183-205, which wavg leaves as
// (f_a + f_b + f_c) + 5 f_own).
__device__ __forceinline__ void tri_normal48(const ChoBnd& b, int64_t n, int32_t t, int32_t N[3],
                                             double nn[3]) {
  N[0] = __ldg(b.btri + 3 * t);
  N[1] = __ldg(b.btri + 3 * t + 1);
  N[2] = __ldg(b.btri + 3 * t + 2);
  const double* x = b.xyz;
  const double* y = b.xyz + n;
  const double* z = b.xyz + 2 * n;
  const double bax = x[N[1]] - x[N[0]], bay = y[N[1]] - y[N[0]], baz = z[N[1]] - z[N[0]];
  const double cax = x[N[2]] - x[N[0]], cay = y[N[2]] - y[N[0]], caz = z[N[2]] - z[N[0]];
  const double k = 1.0 / 48.0;
  nn[0] = (bay * caz - cay * baz) * k;
  nn[1] = (baz * cax - caz * bax) * k;
  nn[2] = (bax * cay - cax * bay) * k;
}
__device__ __forceinline__ double wavg(int pos, double a, double b, double c) {
  return (a + b + c) + 5.0 * (pos == 0 ? a : (pos == 1 ? b : c));
}

__device__ __forceinline__ void block_min(double v, unsigned long long* dst) {
  __shared__ double red[32];
  unsigned long long bits = __double_as_longlong(v);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long other = __shfl_xor_sync(0xffffffffu, bits, o);
    bits = other < bits ? other : bits;
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = __longlong_as_double(bits);
  __syncthreads();
  if (wid == 0) {
    const int nw = (blockDim.x + 31) >> 5;
    unsigned long long b = __double_as_longlong(lane < nw ? red[lane] : DBL_MAX);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      unsigned long long other = __shfl_xor_sync(0xffffffffu, b, o);
      b = other < b ? other : b;
    }
    if (lane == 0) atomicMin(dst, b);
  }
}

// Calls f(e, q, first) for the adjacency entries of a node in entry order
// (q the neighbour, first: the node is the edge's canonical first end), in
// rounds fully unrolled to exactly the entries left, at most XM (the slice
// width is uniform across the warp, so the dispatch does not diverge).  A
// round loads its neighbour ids first, so that its gathers are in flight
// together instead of one entry's load chain after another.
template <int R, class F>
__device__ __forceinline__ void adj_round(const int32_t* __restrict__ nbr, int32_t e0, F& f) {
  int32_t qq[R];
#pragma unroll
  for (int u = 0; u < R; ++u) qq[u] = __ldg(nbr + e0 + u * kSlice);
#pragma unroll
  for (int u = 0; u < R; ++u) {
    const int32_t q = qq[u];
    if (q != kPad) f(e0 + u * kSlice, q >= 0 ? q : ~q, q >= 0);
  }
}

template <int R, int XM, class F>
__device__ __forceinline__ void adj_tail(int r, const int32_t* __restrict__ nbr, int32_t e0,
                                         F& f) {
  if constexpr (R <= XM) {
    if (r == R) {
      adj_round<R>(nbr, e0, f);
      return;
    }
    adj_tail<R + 1, XM>(r, nbr, e0, f);
  }
}

template <int XM, class F>
__device__ __forceinline__ void for_adj(const ChoAdj& adj, int32_t off, int w, int lane, F f) {
  const int32_t e0 = off + lane;
  int k = 0;
  for (; w - k > XM; k += XM) adj_round<XM>(adj.nbr, e0 + k * kSlice, f);
  if (w > k) adj_tail<1, XM>(w - k, adj.nbr, e0 + k * kSlice, f);
}

// What the gradient kernel does with a node's gradient g of NC components.
enum GradOut { GRAD_RAW = 0, GRAD_DIVIDE = 1, GRAD_PROJECT = 2 };

// chorin::vgrad / chorin::grad (Chorin.cpp:211-449): G = sum over edges of
// -/+ d (u_p + u_q) plus the boundary-triangle term.  GRAD_RAW stores it,
// GRAD_DIVIDE stores G/vol (ChoCG::fingrad, src/Inciter/ChoCG.cpp:841-866),
// GRAD_PROJECT (NC = 1, the pressure increment) applies the projection of
// ChoCG::psolved (src/Inciter/ChoCG.cpp:1204-1216): u -= dt G/vol, and with
// addp the pressure update pr += increment (src/Inciter/ChoCG.cpp:1246-1250).
template <int NC, int MODE, bool BND>
__global__ void __launch_bounds__(kNode) k_cgrad(int64_t n, ChoAdj adj, const double* U,
                                                  ChoBnd bnd, const double* __restrict__ ivol,
                                                  double* __restrict__ G, double dt, int addp,
                                                  double* u, double* pr) {
  int64_t p;
  int32_t bi;
  int l;
  node_of(BND, n, bnd, p, bi, l);
  double g[3 * NC];
#pragma unroll
  for (int i = 0; i < 3 * NC; ++i) g[i] = 0.0;
  if (!BND) {
    if (p < 0) return;
    double up[NC];
#pragma unroll
    for (int i = 0; i < NC; ++i) up[i] = U[i * n + p];
    const int lane = static_cast<int>(p & (kSlice - 1));
    const int64_t s = p >> 5;
    const int32_t off = __ldg(adj.soff + s), w = __ldg(adj.swidth + s);
    for_adj<NC == 1 ? 16 : 8>(adj, off, w, lane, [&](int32_t e, int32_t q, bool first) {
      const Coef4 d = ldd4(adj.dd + e);
      const double dx = flip(d.x, first), dy = flip(d.y, first), dz = flip(d.z, first);
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        const double sum = U[i * n + q] + up[i];
        g[i * 3 + 0] += dx * sum;
        g[i * 3 + 1] += dy * sum;
        g[i * 3 + 2] += dz * sum;
      }
    });
    const int32_t b = __ldg(bnd.bidx + p);
    if (b >= 0) {
#pragma unroll
      for (int i = 0; i < 3 * NC; ++i) bnd.park[b * 9 + i] = g[i];
      return;
    }
  } else {
    if (bi >= 0) {
      if (l == 0) {
#pragma unroll
        for (int i = 0; i < 3 * NC; ++i) g[i] = bnd.park[bi * 9 + i];
      }
      for (int32_t j = __ldg(bnd.bptr + bi) + l; j < __ldg(bnd.bptr + bi + 1); j += kBL) {
        const int32_t ent = __ldg(bnd.bent + j);
        const int pos = ent & 3;
        int32_t N[3];
        double nn[3];
        tri_normal48(bnd, n, ent >> 2, N, nn);
#pragma unroll
        for (int i = 0; i < NC; ++i) {
          const double f = wavg(pos, U[i * n + N[0]], U[i * n + N[1]], U[i * n + N[2]]);
#pragma unroll
          for (int jj = 0; jj < 3; ++jj) g[i * 3 + jj] += f * nn[jj];
        }
      }
    }
    lane_add(g);
    if (bi < 0 || l != 0) return;
  }
  if (MODE == GRAD_RAW) {
#pragma unroll
    for (int i = 0; i < 3 * NC; ++i) G[i * n + p] = g[i];
  } else if (MODE == GRAD_DIVIDE) {
    const double iv = ivol[p];
#pragma unroll
    for (int i = 0; i < 3 * NC; ++i) G[i * n + p] = g[i] * iv;
  } else {
    const double iv = ivol[p] * dt;
#pragma unroll
    for (int jj = 0; jj < 3; ++jj) u[jj * n + p] -= g[jj] * iv;
    if (addp) pr[p] += U[p];
  }
}

// chorin::div (Chorin.cpp:34-209): divergence of the 3-component U with the
// 4th-order pressure damping when stab, optionally divided by dt
// (ChoCG::pinit, src/Inciter/ChoCG.cpp:1039).
template <bool BND>
__global__ void __launch_bounds__(kNode) k_cdiv(int64_t n, ChoAdj adj, const double* U,
                                                 const double* __restrict__ P,
                                                 const double* __restrict__ PG, ChoBnd bnd,
                                                 double dt, int stab, int bydt,
                                                 double* __restrict__ D) {
  int64_t p;
  int32_t bi;
  int l;
  node_of(BND, n, bnd, p, bi, l);
  double acc[1] = {0.0};
  if (!BND) {
    if (p < 0) return;
    const int lane = static_cast<int>(p & (kSlice - 1));
    const int64_t s = p >> 5;
    const int32_t off = __ldg(adj.soff + s), w = __ldg(adj.swidth + s);
    const double* x = bnd.xyz;
    const double* y = bnd.xyz + n;
    const double* z = bnd.xyz + 2 * n;
    const double up = U[p], vp = U[n + p], wp = U[2 * n + p];
    double xp = 0.0, yp = 0.0, zp = 0.0, pp = 0.0, gx = 0.0, gy = 0.0, gz = 0.0;
    if (stab) {
      xp = x[p], yp = y[p], zp = z[p];
      pp = P[p];
      gx = PG[p], gy = PG[n + p], gz = PG[2 * n + p];
    }
    for_adj<8>(adj, off, w, lane, [&](int32_t e, int32_t q, bool first) {
      const Coef4 d = ldd4(adj.dd + e);
      acc[0] += flip(d.x, first) * (up + U[q]) + flip(d.y, first) * (vp + U[n + q]) +
                flip(d.z, first) * (wp + U[2 * n + q]);
      if (stab) {
        // |d| / |x_p - x_q| is geometric: formed once at setup (two FP64
        // square roots and a division per edge and call are expensive on
        // GB300's FP64 pipe)
        const double p4 = (xp - x[q]) * (gx + PG[q]) + (yp - y[q]) * (gy + PG[n + q]) +
                          (zp - z[q]) * (gz + PG[2 * n + q]);
        acc[0] -= (__ldg(adj.sdl + e) * dt) * ((P[q] - pp) + 0.5 * p4);
      }
    });
    const int32_t b = __ldg(bnd.bidx + p);
    if (b >= 0) {
      bnd.park[b * 9] = acc[0];
      return;
    }
  } else {
    if (bi >= 0) {
      if (l == 0) acc[0] = bnd.park[bi * 9];
      for (int32_t j = __ldg(bnd.bptr + bi) + l; j < __ldg(bnd.bptr + bi + 1); j += kBL) {
        const int32_t ent = __ldg(bnd.bent + j);
        const int pos = ent & 3;
        int32_t N[3];
        double nn[3];
        tri_normal48(bnd, n, ent >> 2, N, nn);
        acc[0] += wavg(pos, U[N[0]], U[N[1]], U[N[2]]) * nn[0] +
                  wavg(pos, U[n + N[0]], U[n + N[1]], U[n + N[2]]) * nn[1] +
                  wavg(pos, U[2 * n + N[0]], U[2 * n + N[1]], U[2 * n + N[2]]) * nn[2];
      }
    }
    lane_add(acc);
    if (bi < 0 || l != 0) return;
  }
  D[p] = bydt ? acc[0] / dt : acc[0];
}

// Momentum flux tensor of chorin::flux at every node (Chorin.cpp:451-507):
// T_ij = mu (G_ij + G_ji - 2/3 d_ij tr G) - u_i u_j, symmetric, stored as
// xx, yy, zz, xy, xz, yz.  An edge's flux is the sum of its ends' tensors, so
// forming them per node leaves 15 operations an edge end for about 150.
__global__ void __launch_bounds__(kNode) k_mflux(int64_t n, const double* __restrict__ U,
                                                  const double* __restrict__ G, double mu,
                                                  double* __restrict__ T) {
  const int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (p >= n) return;
  const double u[3] = {U[p], U[n + p], U[2 * n + p]};
  constexpr int a[6] = {0, 1, 2, 0, 0, 1}, b[6] = {0, 1, 2, 1, 2, 2};
  double vis[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if (!(mu < DBL_EPSILON)) {
    const double tr = G[0 * n + p] + G[4 * n + p] + G[8 * n + p];
#pragma unroll
    for (int k = 0; k < 6; ++k) {
      vis[k] = G[(a[k] * 3 + b[k]) * n + p] + G[(b[k] * 3 + a[k]) * n + p];
      if (k < 3) vis[k] -= 2.0 / 3.0 * tr;
    }
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) T[k * n + p] = mu * vis[k] - u[a[k]] * u[b[k]];
}

// chorin::flux (Chorin.cpp:509-638): F_i = d[s_ij - u_i u_j]/dx_j from the node
// tensors T, raw or divided by the volume (ChoCG::div at start-up,
// src/Inciter/ChoCG.cpp:877).
template <bool BND>
__global__ void __launch_bounds__(kNode) k_cflux(int64_t n, ChoAdj adj,
                                                  const double* __restrict__ T, ChoBnd bnd,
                                                  const double* __restrict__ ivol, int divide,
                                                  double* __restrict__ F) {
  int64_t p;
  int32_t bi;
  int l;
  node_of(BND, n, bnd, p, bi, l);
  double acc[3] = {0.0, 0.0, 0.0};
  auto add = [&](const double t[6], double dx, double dy, double dz) {
    acc[0] += dx * t[0] + dy * t[3] + dz * t[4];
    acc[1] += dx * t[3] + dy * t[1] + dz * t[5];
    acc[2] += dx * t[4] + dy * t[5] + dz * t[2];
  };
  if (!BND) {
    if (p < 0) return;
    double tp[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) tp[k] = T[k * n + p];
    const int lane = static_cast<int>(p & (kSlice - 1));
    const int64_t s = p >> 5;
    const int32_t off = __ldg(adj.soff + s), w = __ldg(adj.swidth + s);
    for_adj<4>(adj, off, w, lane, [&](int32_t e, int32_t q, bool first) {
      const Coef4 d = ldd4(adj.dd + e);
      double t[6];
#pragma unroll
      for (int k = 0; k < 6; ++k) t[k] = tp[k] + __ldg(T + k * n + q);
      add(t, flip(d.x, first), flip(d.y, first), flip(d.z, first));
    });
    const int32_t b = __ldg(bnd.bidx + p);
    if (b >= 0) {
#pragma unroll
      for (int i = 0; i < 3; ++i) bnd.park[b * 9 + i] = acc[i];
      return;
    }
  } else {
    if (bi >= 0) {
      if (l == 0) {
#pragma unroll
        for (int i = 0; i < 3; ++i) acc[i] = bnd.park[bi * 9 + i];
      }
      for (int32_t j = __ldg(bnd.bptr + bi) + l; j < __ldg(bnd.bptr + bi + 1); j += kBL) {
        const int32_t ent = __ldg(bnd.bent + j);
        const int pos = ent & 3;
        int32_t N[3];
        double nn[3], t[6];
        tri_normal48(bnd, n, ent >> 2, N, nn);
#pragma unroll
        for (int k = 0; k < 6; ++k)
          t[k] = wavg(pos, T[k * n + N[0]], T[k * n + N[1]], T[k * n + N[2]]);
        add(t, nn[0], nn[1], nn[2]);
      }
    }
    lane_add(acc);
    if (bi < 0 || l != 0) return;
  }
  const double iv = divide ? ivol[p] : 1.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) F[i * n + p] = divide ? acc[i] * iv : acc[i];
}

struct AdvPrm {
  double mu, stab2coef;
  int stab, stab2;
};

// van Leer limited reconstruction of the three velocity components on the
// canonical edge a -> b (Chorin.cpp:711-829): uL, uR the ends' values on entry,
// the edge states on return.  With a = delta2 + eps, b = delta1 + eps of one
// sign, 0.25 ((1-k) delta1 phi(a/b) + (1+k) delta2 phi(b/a)) is, exactly,
// (a b - (eps/2) ((1-k) a + (1+k) b)) / (a + b), and 0 for a b <= 0: the numerator
// (a - h2)(b - h1) - h1 h2 with h1, h2 = (eps/2)(1 -+ k), and a + b = 2 (g1 + eps)
// as delta1 + delta2 = 2 g1.  Signs are tested on integer bits and a quotient
// takes three FP64 instructions (the reference: eight divisions a component).
__device__ __forceinline__ void reconstruct(const double g1[3], const double g2[3], double uL[3],
                                            double uR[3]) {
  constexpr double eps = 1.0e-9, k = 1.0 / 3.0;
  constexpr double h1 = 0.5 * eps * (1.0 - k), h2 = 0.5 * eps * (1.0 + k);
  constexpr double A0 = 0.5 * (eps - h2), B0 = eps - h1, H = 0.5 * h1 * h2;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double d2 = uR[c] - uL[c];
    const double d1 = 2.0 * g1[c] - d2, d3 = 2.0 * g2[c] - d2;
    const int sa = side(d2, -eps), pl = sa * side(d1, -eps), pr = sa * side(d3, -eps);
    const double A = 0.5 * d2 + A0;
    const double nl = A * (d1 + B0) - H, nr = A * (d3 + B0) - H;
    const double ql = recip(pl > 0 ? g1[c] + eps : 1.0), qr = recip(pr > 0 ? g2[c] + eps : 1.0);
    uL[c] += (pl > 0 ? nl : 0.0) * ql;
    uR[c] -= (pr > 0 ? nr : 0.0) * qr;
  }
}

// chorin::rhs (Chorin.cpp:831-1044) at every node, fused with the explicit
// stage update of ChoCG::solve (src/Inciter/ChoCG.cpp:1550-1566):
// u_out = un - dtk R / vol, where un is this stage's input at stage 0.
// With dtk == 0 and a null u_out only R is written (drop-in).  The edge flux
// (adv_damp2 / adv_damp4, Chorin.cpp:640-829) is symmetric in its ends but for
// the sign of d and of the velocity difference: from node p outwards, with d'
// = -d at the canonical first end and d at the second, the node receives
// u_p vn_p + u_q vn_q + (P_p + P_q) d' - (aw - v)(u_q - u_p), vn = u.d'.
template <bool DAMP4, bool BND>
__global__ void __launch_bounds__(kNode) k_crhs(int64_t n, ChoAdj adj, const double* U,
                                                 const double* G, const double* P, ChoBnd bnd,
                                                 AdvPrm ap, const double* __restrict__ ivol,
                                                 double dtk, int stage0, double* un,
                                                 double* __restrict__ uout,
                                                 double* __restrict__ R) {
  int64_t p;
  int32_t bi;
  int l;
  node_of(BND, n, bnd, p, bi, l);
  double acc[3] = {0.0, 0.0, 0.0};
  if (!BND) {
    if (p < 0) return;
    const int lane = static_cast<int>(p & (kSlice - 1));
    const int64_t s = p >> 5;
    const int32_t off = __ldg(adj.soff + s), w = __ldg(adj.swidth + s);
    const double* xyz = bnd.xyz;
    double u0[3], x0[3], g0[DAMP4 ? 9 : 1];
#pragma unroll
    for (int c = 0; c < 3; ++c) u0[c] = U[c * n + p];
    const double p0 = P[p];
    if (DAMP4) {
#pragma unroll
      for (int c = 0; c < 3; ++c) x0[c] = xyz[c * n + p];
#pragma unroll
      for (int c = 0; c < (DAMP4 ? 9 : 1); ++c) g0[c] = G[c * n + p];
    }
    for_adj<DAMP4 ? 4 : 8>(adj, off, w, lane, [&](int32_t e, int32_t q, bool first) {
      const Coef4 d = ldd4(adj.dd + e);
      const double dx = flip(d.x, first), dy = flip(d.y, first), dz = flip(d.z, first);
      double uq[3], du[3], a[3], b[3];  // a, b: the edge states at p and at q
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        uq[c] = U[c * n + q];
        du[c] = uq[c] - u0[c];
        a[c] = u0[c];
        b[c] = uq[c];
      }
      if constexpr (DAMP4) {
        const double ex = xyz[q] - x0[0], ey = xyz[n + q] - x0[1], ez = xyz[2 * n + q] - x0[2];
        double gp[3], gq[3];  // G.(x_q - x_p) at p and at q
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          gp[c] = g0[c * 3] * ex + g0[c * 3 + 1] * ey + g0[c * 3 + 2] * ez;
          gq[c] = G[(c * 3) * n + q] * ex + G[(c * 3 + 1) * n + q] * ey +
                  G[(c * 3 + 2) * n + q] * ez;
        }
        // in the canonical orientation: left the first end, and the
        // projections change sign with the edge vector
        double uL[3], uR[3], g1[3], g2[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          uL[c] = first ? a[c] : b[c];
          uR[c] = first ? b[c] : a[c];
          g1[c] = flip(first ? gp[c] : gq[c], !first);
          g2[c] = flip(first ? gq[c] : gp[c], !first);
        }
        reconstruct(g1, g2, uL, uR);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          a[c] = first ? uL[c] : uR[c];
          b[c] = first ? uR[c] : uL[c];
        }
      }
      const double va = a[0] * dx + a[1] * dy + a[2] * dz;
      const double vb = b[0] * dx + b[1] * dy + b[2] * dz;
      double aw = 0.0;
      if (ap.stab) aw = 0.5 * fabs(va + vb);
      if (ap.stab2) aw += ap.stab2coef * fmax(fabs(va), fabs(vb));
      const double v = d.w * ap.mu;
      const double pf = p0 + P[q];
      const double dd[3] = {dx, dy, dz};
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        // a sum of two rounded products, as a fused one would round the two
        // ends' products differently and the ends' terms would not cancel
        acc[c] += __dadd_rn(__dmul_rn(a[c], va), __dmul_rn(b[c], vb)) + pf * dd[c];
        if (DAMP4)
          acc[c] -= aw * (b[c] - a[c]) - v * du[c];
        else
          acc[c] -= (aw - v) * du[c];
      }
    });
    const int32_t b = __ldg(bnd.bidx + p);
    if (b >= 0) {
#pragma unroll
      for (int c = 0; c < 3; ++c) bnd.park[b * 9 + c] = acc[c];
      return;
    }
  } else {
    if (bi >= 0) {
      if (l == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] = bnd.park[bi * 9 + c];
      }
      for (int32_t j = __ldg(bnd.bptr + bi) + l; j < __ldg(bnd.bptr + bi + 1); j += kBL) {
        const int32_t ent = __ldg(bnd.bent + j);
        const int pos = ent & 3;
        int32_t N[3];
        double nn[3];
        tri_normal48(bnd, n, ent >> 2, N, nn);
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const double uu = U[N[a]], vv = U[n + N[a]], ww = U[2 * n + N[a]];
          const double wt = pos == a ? 6.0 : 1.0, pw = wt * P[N[a]];
          const double vn = wt * (nn[0] * uu + nn[1] * vv + nn[2] * ww);
          acc[0] += uu * vn + pw * nn[0];
          acc[1] += vv * vn + pw * nn[1];
          acc[2] += ww * vn + pw * nn[2];
        }
      }
    }
    lane_add(acc);
    if (bi < 0 || l != 0) return;
  }
  if (R) {
#pragma unroll
    for (int c = 0; c < 3; ++c) R[c * n + p] = acc[c];
  }
  if (uout) {
    const double f = dtk * ivol[p];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double u0;
      if (stage0) {
        u0 = U[c * n + p];
        un[c * n + p] = u0;
      } else {
        u0 = un[c * n + p];
      }
      uout[c * n + p] = u0 - f * acc[c];
    }
  }
}

// ChoCG::BC (src/Inciter/ChoCG.cpp:1333-1354) per BC node, in the
// reference's order: Dirichlet components, symmetry projections (one per
// set holding the node), noslip.  sym_only applies just the symmetry
// projections (to the start-up momentum flux, ChoCG.cpp:878).
__global__ void k_cbc(int64_t n, int64_t nbc, const int32_t* __restrict__ node,
                      const int32_t* __restrict__ dir, const int32_t* __restrict__ symp,
                      const int32_t* __restrict__ noslip, const int32_t* __restrict__ dirmask,
                      const double* __restrict__ dirval, const double* __restrict__ symn,
                      int sym_only, double* U) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= nbc) return;
  const int64_t p = node[i];
  double u[3] = {U[p], U[n + p], U[2 * n + p]};
  const int32_t dd = dir[i];
  if (!sym_only && dd >= 0) {
#pragma unroll
    for (int c = 0; c < 3; ++c)
      if (dirmask[dd * 3 + c]) u[c] = dirval[dd * 3 + c];
  }
  for (int32_t k = symp[i]; k < symp[i + 1]; ++k) {
    const double* nn = symn + 3 * k;
    const double vn = u[0] * nn[0] + u[1] * nn[1] + u[2] * nn[2];
    u[0] -= vn * nn[0];
    u[1] -= vn * nn[1];
    u[2] -= vn * nn[2];
  }
  if (!sym_only && noslip[i]) u[0] = u[1] = u[2] = 0.0;
  U[p] = u[0];
  U[n + p] = u[1];
  U[2 * n + p] = u[2];
}

// ChoCG::dt (src/Inciter/ChoCG.cpp:1356-1412): min over nodes of
// cbrt(V)/max(|u|, 1e-8) and, with viscosity, V^(2/3)/mu.
__global__ void __launch_bounds__(kBlock) k_cdt(int64_t n, const double* __restrict__ U,
                                                 const double* __restrict__ cbrtv, double mu,
                                                 unsigned long long* dtmin) {
  const int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  double m = DBL_MAX;
  if (p < n) {
    const double u = U[p], v = U[n + p], w = U[2 * n + p];
    const double vel = sqrt(u * u + v * v + w * w);
    const double L = cbrtv[p];
    m = fmin(m, L / fmax(vel, 1.0e-8));
    if (mu > DBL_EPSILON) m = fmin(m, L * L / mu);
  }
  block_min(m, dtmin);
}

// 1/vol and cbrt(vol).
__global__ void k_node_factors(int64_t n, const double* __restrict__ vol,
                               double* __restrict__ ivol, double* __restrict__ cbrtv) {
  const int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (p >= n) return;
  ivol[p] = 1.0 / vol[p];
  cbrtv[p] = cbrt(vol[p]);
}

__global__ void k_aos_soa(int64_t n, int nc, const double* __restrict__ a, double* __restrict__ s) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n * nc) return;
  const int64_t p = i / nc;
  const int c = static_cast<int>(i - p * nc);
  s[c * n + p] = a[i];
}
__global__ void k_soa_aos(int64_t n, int nc, const double* __restrict__ s, double* __restrict__ a) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n * nc) return;
  const int64_t p = i / nc;
  const int c = static_cast<int>(i - p * nc);
  a[i] = s[c * n + p];
}

// ---------------------------------------------------------------- host side

ChoAdj adj_of(ChoCGDev* d) { return ChoAdj{d->soff, d->swidth, d->nbr, d->dd, d->sdl}; }
ChoBnd bnd_of(ChoCGDev* d) {
  return ChoBnd{d->bidx, d->bptr, d->bent, d->btri, d->xyz, d->bnode, d->park, d->nbn};
}

// Both passes of a node kernel (domain pass over the n nodes, then the
// boundary pass over the boundary nodes), the same arguments to each.
template <auto KD, auto KB, class... A>
void two_pass(cudaStream_t s, int64_t n, int64_t nb, A... args) {
  KD<<<blocks_for(n, kNode), kNode, 0, s>>>(args...);
  if (nb > 0) KB<<<blocks_for(nb * kBL, kNode), kNode, 0, s>>>(args...);
}
AdvPrm adv_of(ChoCGDev* d) {
  return AdvPrm{d->prm.mu, d->prm.stab2coef, d->prm.stab != 0, d->prm.stab2 != 0};
}

int get_ctx(xg_ctx* c, ChoCGDev** out, bool need_cg) {
  int rc = use(c);
  if (rc) return rc;
  ChoCGDev* d = c->chocg;
  if (!d) return fail(c, XG_ERR_STATE, "chocg: no operators (xg_chocg_setup)");
  if (need_cg && cg_rows(c) != d->n)
    return fail(c, XG_ERR_STATE, "chocg: the context's CG system is not the pressure matrix");
  *out = d;
  return XG_OK;
}

template <int NC, int MODE>
int launch_grad(xg_ctx* c, ChoCGDev* d, const double* U, double* G, double dt = 0.0,
                int addp = 0) {
  two_pass<k_cgrad<NC, MODE, false>, k_cgrad<NC, MODE, true>>(
      c->stream, d->n, d->nbn, d->n, adj_of(d), U, bnd_of(d), d->ivol, G, dt, addp, d->u, d->pr);
  XG_CHECK_LAUNCH(c);
  return XG_OK;
}

int launch_bc(xg_ctx* c, ChoCGDev* d, double* U, int sym_only) {
  if (d->nbc == 0) return XG_OK;
  k_cbc<<<blocks_for(d->nbc, kBlock), kBlock, 0, c->stream>>>(
      d->n, d->nbc, d->bcnode, d->bcdir, d->bcsymp, d->bcnoslip, d->dirmask, d->dirval, d->symn,
      sym_only, U);
  XG_CHECK_LAUNCH(c);
  return XG_OK;
}

int launch_div(xg_ctx* c, ChoCGDev* d, const double* U, double dt, int stab, int bydt) {
  two_pass<k_cdiv<false>, k_cdiv<true>>(c->stream, d->n, d->nbn, d->n, adj_of(d), U, d->pr,
                                        d->pgrad, bnd_of(d), dt, stab, bydt, d->div);
  XG_CHECK_LAUNCH(c);
  return XG_OK;
}

int launch_rhs(xg_ctx* c, ChoCGDev* d, const double* U, double dtk, int stage0, double* uout,
               double* R) {
  const AdvPrm ap = adv_of(d);
  if (d->prm.flux == XG_DAMP4)
    two_pass<k_crhs<true, false>, k_crhs<true, true>>(c->stream, d->n, d->nbn, d->n, adj_of(d), U,
                                                       d->vgrad, d->pr, bnd_of(d), ap, d->ivol,
                                                       dtk, stage0, d->un, uout, R);
  else
    two_pass<k_crhs<false, false>, k_crhs<false, true>>(c->stream, d->n, d->nbn, d->n, adj_of(d),
                                                         U, d->vgrad, d->pr, bnd_of(d), ap, d->ivol,
                                                         dtk, stage0, d->un, uout, R);
  XG_CHECK_LAUNCH(c);
  return XG_OK;
}

// theta-implicit momentum system, per step (ChoCG::lhs, ChoCG.cpp:1433-1477):
// A = -(M / dt + theta mu K) with M the consistent mass sum_e J/120 (1 + d_ab)
// and K the stiffness sum_e grad_a.grad_b / J / 6, both on A's pattern.
__global__ void k_mom_values(int64_t nent, const double* __restrict__ K,
                             const double* __restrict__ M, double thmu, double dt,
                             double* __restrict__ a) {
  const int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (e >= nent) return;
  a[e] = -(M[e] / dt + thmu * K[e]);
}
// [3][n] -> row order 3i + c, and the update u = un + du of ChoCG::msolved
// (ChoCG.cpp:1626-1645).
__global__ void k_to_rows3(int64_t n, const double* __restrict__ R, double* __restrict__ b) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
#pragma unroll
  for (int c = 0; c < 3; ++c) b[i * 3 + c] = R[c * n + i];
}
__global__ void k_mom_update(int64_t n, const double* __restrict__ un,
                             const double* __restrict__ du, double* __restrict__ u) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= n) return;
#pragma unroll
  for (int c = 0; c < 3; ++c) u[c * n + i] = un[c * n + i] + du[i * 3 + c];
}

// The semi-implicit last stage of ChoCG::solve (ChoCG.cpp:1576-1606): the
// momentum system A du = R (R the stage's rhs, [3][n] in d->R3) with the
// Dirichlet rows at zero increment, warm-started from the previous
// increment, mom_iter iterations at most to mom_tol, then u = un + du.  The
// momentum system is the context's CG system while it solves.
int momentum_solve(xg_ctx* c, ChoCGDev* d, double dt) {
  const int64_t n = d->n;
  cudaStream_t s = c->stream;
  CGDev* const saved = c->cg;
  c->cg = d->mom;
  int rc = XG_OK;
  do {
    const int64_t nent = cg_nent(c);
    k_mom_values<<<blocks_for(nent, kBlock), kBlock, 0, s>>>(
        nent, d->baseK, d->baseM, d->theta * d->prm.mu, dt, cg_values_device(c));
    XG_CHECK_LAUNCH(c);
    k_to_rows3<<<blocks_for(n, kBlock), kBlock, 0, s>>>(n, d->R3, d->b3);
    XG_CHECK_LAUNCH(c);
    if (!d->mommask_up) {
      std::vector<uint8_t> mask = d->mommask;
      mask.resize(n * 3, 0);
      std::vector<double> zero(n * 3, 0.0);
      rc = cg_set_dirichlet(c, mask.data(), zero.data());
      if (rc) break;
      d->mommask_up = true;
    }
    rc = cg_init_device(c, d->b3, 1, d->mom_pc);
    if (rc) break;
    int64_t it = 0;
    double normr = 0, normb = 0;
    int conv = 0;
    rc = xg_cg_solve(c, d->mom_iter, d->mom_tol, &it, &normr, &normb, &conv);
    if (rc == XG_ERR_NOTCONV) rc = XG_OK;  // the reference carries on
    if (rc) break;
    d->last_mit = conv ? it : -it;
    k_mom_update<<<blocks_for(n, kBlock), kBlock, 0, s>>>(n, d->un, cg_solution_device(c), d->u);
    XG_CHECK_LAUNCH(c);
  } while (false);
  c->cg = saved;
  return rc;
}

// One pressure solve of ChoCG::pinit/psolve on the context's CG system with
// the device right-hand side d->div: Dirichlet values of the first solves or
// zero, warm start from the previous solution.  As in the reference, a solve
// that stops short of the tolerance (iteration limit or the (p,q) breakdown
// guard) does not stop the scheme: last_it is then the negated count.
int pressure_solve(xg_ctx* c, ChoCGDev* d, int zero_values) {
  int rc = xg_cg_set_guard(c, d->prm.pguard);
  if (rc) return rc;
  rc = cg_init_device(c, d->div, zero_values, d->prm.ppc);
  if (rc) return rc;
  int64_t it = 0, outer = 0;
  double normr = 0, normb = 0;
  int conv = 0;
  if (d->prm.pmixed)
    rc = xg_cg_solve_mixed(c, 1000, d->prm.ptol, d->prm.pinner_tol, d->prm.pmaxit, &outer, &it,
                           &normr, &normb, &conv);
  else
    rc = xg_cg_solve(c, d->prm.pmaxit, d->prm.ptol, &it, &normr, &normb, &conv);
  if (rc && rc != XG_ERR_NOTCONV) return rc;
  d->last_it = conv ? it : -it;
  return XG_OK;
}

// Time step size of the device state (ChoCG::dt): synchronises.
int step_dt(xg_ctx* c, ChoCGDev* d, double* dt) {
  if (std::fabs(d->prm.const_dt) > DBL_EPSILON) {
    *dt = d->prm.const_dt;
    return XG_OK;
  }
  const unsigned long long big = 0x7fefffffffffffffull;  // DBL_MAX bits
  XG_CUDA(c, cudaMemcpyAsync(d->dtmin, &big, sizeof(big), cudaMemcpyHostToDevice, c->stream));
  k_cdt<<<blocks_for(d->n, kBlock), kBlock, 0, c->stream>>>(d->n, d->u, d->cbrtv, d->prm.mu,
                                                             d->dtmin);
  XG_CHECK_LAUNCH(c);
  unsigned long long bits = 0;
  XG_CUDA(c, cudaMemcpyAsync(&bits, d->dtmin, sizeof(bits), cudaMemcpyDeviceToHost, c->stream));
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  double m;
  std::memcpy(&m, &bits, sizeof(m));
  *dt = m * d->prm.cfl;
  return XG_OK;
}

struct EdgeRec {
  int64_t a, b;
  double d[5];
};

}  // namespace

}  // namespace xg

using namespace xg;

extern "C" {

int xg_chocg_setup(xg_ctx* c, const xg_chocg_params* prm, int64_t npoin, const double* coord,
                   const double* vol, int64_t ntet, const uint64_t* dsupedge0,
                   const double* dsupint0, int64_t ntri, const uint64_t* dsupedge1,
                   const double* dsupint1, int64_t nedge, const uint64_t* dsupedge2,
                   const double* dsupint2, int64_t nbtri, const uint64_t* triinpoel) {
  XG_HOST_TRY
  int rc = use(c);
  if (rc) return rc;
  if (!prm || npoin <= 0 || !coord || !vol) return fail(c, XG_ERR_ARG, "chocg_setup: bad mesh");
  if (npoin >= (int64_t(1) << 31) - 64) return fail(c, XG_ERR_ARG, "chocg_setup: too many nodes");
  if (prm->flux != XG_DAMP2 && prm->flux != XG_DAMP4)
    return fail(c, XG_ERR_ARG, "Flux not correctly configured");
  if (prm->rk < 1 || prm->rk > 4) return fail(c, XG_ERR_ARG, "chocg_setup: rk must be 1..4");
  if (prm->ppc < 0 || prm->ppc > 2) return fail(c, XG_ERR_ARG, "chocg_setup: unknown pressure pc");
  if (prm->pguard != 0 && prm->pguard != 1)
    return fail(c, XG_ERR_ARG, "chocg_setup: pressure guard is 0 or 1");
  if (prm->pmaxit <= 0 || !(prm->ptol >= 0))
    return fail(c, XG_ERR_ARG, "chocg_setup: bad pressure iteration limit or tolerance");
  if ((ntet && (!dsupedge0 || !dsupint0)) || (ntri && (!dsupedge1 || !dsupint1)) ||
      (nedge && (!dsupedge2 || !dsupint2)) || (nbtri && !triinpoel))
    return fail(c, XG_ERR_ARG, "chocg_setup: null superedge or boundary array");
  const int64_t n = npoin;
  // superedges -> edges in the orientation chorin:: evaluates them
  // (Chorin.cpp:122-170: tet group (0,1),(1,2),(2,0),(0,3),(1,3),(2,3),
  // triangle group (0,1),(1,2),(2,0))
  std::vector<EdgeRec> E;
  E.reserve(static_cast<size_t>(ntet * 6 + ntri * 3 + nedge));
  static const int tp[6][2] = {{0, 1}, {1, 2}, {2, 0}, {0, 3}, {1, 3}, {2, 3}};
  static const int rp[3][2] = {{0, 1}, {1, 2}, {2, 0}};
  auto bad = [&](uint64_t id) { return id >= static_cast<uint64_t>(n); };
  auto push = [&](uint64_t a, uint64_t b, const double* dd) -> bool {
    if (bad(a) || bad(b) || a == b) return false;
    EdgeRec r{int64_t(a), int64_t(b), {dd[0], dd[1], dd[2], dd[3], dd[4]}};
    E.push_back(r);
    return true;
  };
  for (int64_t e = 0; e < ntet; ++e)
    for (int k = 0; k < 6; ++k)
      if (!push(dsupedge0[e * 4 + tp[k][0]], dsupedge0[e * 4 + tp[k][1]],
                dsupint0 + (e * 6 + k) * 5))
        return fail(c, XG_ERR_ARG, "chocg_setup: tet superedge id");
  for (int64_t e = 0; e < ntri; ++e)
    for (int k = 0; k < 3; ++k)
      if (!push(dsupedge1[e * 3 + rp[k][0]], dsupedge1[e * 3 + rp[k][1]],
                dsupint1 + (e * 3 + k) * 5))
        return fail(c, XG_ERR_ARG, "chocg_setup: triangle superedge id");
  for (int64_t e = 0; e < nedge; ++e)
    if (!push(dsupedge2[e * 2], dsupedge2[e * 2 + 1], dsupint2 + e * 5))
      return fail(c, XG_ERR_ARG, "chocg_setup: edge id");
  // per-node entries sorted by neighbour id
  std::vector<int64_t> start(n + 1, 0);
  for (auto& e : E) {
    ++start[e.a + 1];
    ++start[e.b + 1];
  }
  for (int64_t i = 0; i < n; ++i) start[i + 1] += start[i];
  struct Ent {
    int64_t q, eid;
    bool first;
  };
  std::vector<Ent> ent(static_cast<size_t>(start[n]));
  {
    std::vector<int64_t> fill(start.begin(), start.end() - 1);
    for (size_t k = 0; k < E.size(); ++k) {
      ent[fill[E[k].a]++] = {E[k].b, int64_t(k), true};
      ent[fill[E[k].b]++] = {E[k].a, int64_t(k), false};
    }
  }
  for (int64_t p = 0; p < n; ++p)
    std::sort(ent.begin() + start[p], ent.begin() + start[p + 1],
              [](const Ent& x, const Ent& y) { return x.q < y.q || (x.q == y.q && x.eid < y.eid); });
  const int64_t nslice = (n + kSlice - 1) / kSlice;
  std::vector<int32_t> soff(nslice + 1), swidth(nslice);
  int64_t total = 0;
  for (int64_t s = 0; s < nslice; ++s) {
    int64_t w = 0;
    for (int64_t p = s * kSlice; p < std::min(n, (s + 1) * kSlice); ++p)
      w = std::max<int64_t>(w, start[p + 1] - start[p]);
    swidth[s] = static_cast<int32_t>(w);
    soff[s] = static_cast<int32_t>(total);
    total += w * kSlice;
    if (total >= (int64_t(1) << 31)) return fail(c, XG_ERR_ARG, "chocg_setup: adjacency too large");
  }
  soff[nslice] = static_cast<int32_t>(total);
  std::vector<int32_t> nbr(static_cast<size_t>(std::max<int64_t>(1, total)), kPad);
  std::vector<Coef4> dd(nbr.size(), Coef4{0.0, 0.0, 0.0, 0.0});
  std::vector<double> sdl(nbr.size(), 0.0);
  for (int64_t p = 0; p < n; ++p) {
    const int64_t s = p / kSlice, lane = p % kSlice;
    for (int64_t k = 0; k < start[p + 1] - start[p]; ++k) {
      const Ent& en = ent[start[p] + k];
      const int64_t idx = soff[s] + k * kSlice + lane;
      nbr[idx] = en.first ? static_cast<int32_t>(en.q) : ~static_cast<int32_t>(en.q);
      const double* r = E[en.eid].d;
      dd[idx] = Coef4{r[0], r[1], r[2], r[4]};
      const double dx = coord[p] - coord[en.q], dy = coord[n + p] - coord[n + en.q],
                   dz = coord[2 * n + p] - coord[2 * n + en.q];
      sdl[idx] = std::sqrt(r[0] * r[0] + r[1] * r[1] + r[2] * r[2]) /
                 std::sqrt(dx * dx + dy * dy + dz * dz);
    }
  }
  // boundary triangles, per boundary node the (triangle, position) pairs in
  // triangle order
  std::vector<int32_t> bidx(n, -1), btri(std::max<int64_t>(1, nbtri * 3));
  std::vector<int32_t> bcount;
  int64_t nbn = 0;
  for (int64_t t = 0; t < nbtri; ++t)
    for (int a = 0; a < 3; ++a) {
      const uint64_t p = triinpoel[t * 3 + a];
      if (bad(p)) return fail(c, XG_ERR_ARG, "chocg_setup: triinpoel id");
      btri[t * 3 + a] = static_cast<int32_t>(p);
      if (bidx[p] < 0) {
        bidx[p] = static_cast<int32_t>(nbn++);
        bcount.push_back(0);
      }
      ++bcount[bidx[p]];
    }
  std::vector<int32_t> bptr(nbn + 1, 0), bent(std::max<int64_t>(1, nbtri * 3));
  std::vector<int32_t> bnode(std::max<int64_t>(1, nbn), 0);
  for (int64_t p = 0; p < n; ++p)
    if (bidx[p] >= 0) bnode[bidx[p]] = static_cast<int32_t>(p);
  for (int64_t i = 0; i < nbn; ++i) bptr[i + 1] = bptr[i] + bcount[i];
  {
    std::vector<int32_t> fill(bptr.begin(), bptr.end() - 1);
    for (int64_t t = 0; t < nbtri; ++t)
      for (int a = 0; a < 3; ++a)
        bent[fill[bidx[triinpoel[t * 3 + a]]]++] = static_cast<int32_t>(t * 4 + a);
  }
  if (c->chocg) {
    XG_CUDA(c, cudaStreamSynchronize(c->stream));
    destroy_chocg(c->chocg);
    c->chocg = nullptr;
  }
  auto* d = new ChoCGDev;
  c->chocg = d;
  d->n = n;
  d->prm = *prm;
  d->nslice = nslice;
  d->nent = total;
  d->nbn = nbn;
  for (int pass = 0; pass < 2; ++pass) {
    Arena& A = d->arena;
    A.plan(d->soff, soff.size());
    A.plan(d->swidth, swidth.size());
    A.plan(d->nbr, nbr.size());
    A.plan(d->dd, dd.size());
    A.plan(d->sdl, sdl.size());
    A.plan(d->bidx, n);
    A.plan(d->bptr, bptr.size());
    A.plan(d->bent, bent.size());
    A.plan(d->btri, btri.size());
    A.plan(d->bnode, bnode.size());
    A.plan(d->park, bnode.size() * 9);
    A.plan(d->xyz, 3 * n);
    A.plan(d->ivol, n);
    A.plan(d->cbrtv, n);
    A.plan(d->u, 3 * n);
    A.plan(d->u2, 3 * n);
    A.plan(d->un, 3 * n);
    A.plan(d->pr, n);
    A.plan(d->pgrad, 3 * n);
    A.plan(d->vgrad, 9 * n);
    A.plan(d->div, n);
    A.plan(d->flx, 3 * n);
    A.plan(d->stage, 9 * n);
    A.plan(d->dtmin, 1);
    if (pass == 0) {
      cudaError_t e = A.reserve();
      if (e != cudaSuccess) {
        destroy_chocg(d);
        c->chocg = nullptr;
        return fail(c, XG_ERR_CUDA, std::string("chocg_setup: ") + cudaGetErrorString(e));
      }
    }
  }
  auto up = [&](void* dst, const void* src, size_t bytes) { return upload(c, dst, src, bytes); };
  XG_CUDA(c, up(d->soff, soff.data(), soff.size() * 4));
  XG_CUDA(c, up(d->swidth, swidth.data(), swidth.size() * 4));
  XG_CUDA(c, up(d->nbr, nbr.data(), nbr.size() * 4));
  XG_CUDA(c, up(d->dd, dd.data(), dd.size() * sizeof(Coef4)));
  XG_CUDA(c, up(d->sdl, sdl.data(), sdl.size() * 8));
  XG_CUDA(c, up(d->bidx, bidx.data(), n * 4));
  XG_CUDA(c, up(d->bptr, bptr.data(), bptr.size() * 4));
  XG_CUDA(c, up(d->bent, bent.data(), bent.size() * 4));
  XG_CUDA(c, up(d->btri, btri.data(), btri.size() * 4));
  XG_CUDA(c, up(d->bnode, bnode.data(), bnode.size() * 4));
  XG_CUDA(c, up(d->xyz, coord, 3 * n * 8));
  d->xyz_host.assign(coord, coord + 3 * n);
  // through the staging buffer
  XG_CUDA(c, up(d->stage, vol, n * 8));
  k_node_factors<<<blocks_for(n, kBlock), kBlock, 0, c->stream>>>(n, d->stage, d->ivol, d->cbrtv);
  XG_CHECK_LAUNCH(c);
  for (double* z : {d->u, d->u2, d->un, d->pr, d->pgrad, d->vgrad, d->div, d->flx})
    XG_CUDA(c, cudaMemsetAsync(
                   z, 0, (z == d->vgrad ? 9 : (z == d->pr || z == d->div ? 1 : 3)) * n * 8, c->stream));
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  return XG_OK;
  XG_HOST_CATCH(c)
}

int xg_chocg_set_theta(xg_ctx* c, double theta, int64_t ntet, const uint64_t* inpoel, int mom_pc,
                       int64_t mom_iter, double mom_tol) {
  XG_HOST_TRY
  ChoCGDev* d = nullptr;
  int rc = get_ctx(c, &d, false);
  if (rc) return rc;
  if (!(theta >= 0.0) || mom_iter < 0 || !(mom_tol > 0.0) || (mom_pc != 0 && mom_pc != 1))
    return fail(c, XG_ERR_ARG, "chocg_set_theta: bad theta, iteration limit, tolerance or pc");
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  if (d->mom) {
    destroy_cg(d->mom);
    d->mom = nullptr;
  }
  d->momarena.release();
  d->theta = 0.0;
  if (theta < std::numeric_limits<double>::epsilon()) return XG_OK;  // explicit prediction
  const int64_t n = d->n;
  if (ntet <= 0 || !inpoel) return fail(c, XG_ERR_ARG, "chocg_set_theta: no tetrahedra");
  for (int64_t k = 0; k < ntet * 4; ++k)
    if (inpoel[k] >= static_cast<uint64_t>(n))
      return fail(c, XG_ERR_ARG, "chocg_set_theta: tetrahedron node out of range");
  // the node pattern (every pair of nodes sharing a tetrahedron, and the
  // diagonal), columns sorted
  std::vector<std::vector<int64_t>> nb(n);
  for (int64_t e = 0; e < ntet; ++e)
    for (int a = 0; a < 4; ++a)
      for (int b = 0; b < 4; ++b) nb[inpoel[e * 4 + a]].push_back(int64_t(inpoel[e * 4 + b]));
  std::vector<uint64_t> ia(n + 1, 0);
  std::vector<int64_t> ja;
  for (int64_t i = 0; i < n; ++i) {
    auto& v = nb[i];
    v.push_back(i);
    std::sort(v.begin(), v.end());
    v.erase(std::unique(v.begin(), v.end()), v.end());
    ia[i + 1] = ia[i] + v.size();
    ja.insert(ja.end(), v.begin(), v.end());
    std::vector<int64_t>().swap(v);
  }
  // stiffness grad_a.grad_b / J / 6 and consistent mass J/120 (1 + d_ab),
  // summed over the elements in element order (ChoCG::lhs)
  std::vector<double> K(ja.size(), 0.0), M(ja.size(), 0.0);
  const double* X = d->xyz_host.data();
  const double* Y = X + n;
  const double* Z = Y + n;
  auto pos = [&](int64_t i, int64_t j) {
    return static_cast<int64_t>(std::lower_bound(ja.begin() + ia[i], ja.begin() + ia[i + 1], j) -
                                ja.begin());
  };
  for (int64_t e = 0; e < ntet; ++e) {
    const uint64_t* N = inpoel + e * 4;
    const double ba[3] = {X[N[1]] - X[N[0]], Y[N[1]] - Y[N[0]], Z[N[1]] - Z[N[0]]};
    const double ca[3] = {X[N[2]] - X[N[0]], Y[N[2]] - Y[N[0]], Z[N[2]] - Z[N[0]]};
    const double da[3] = {X[N[3]] - X[N[0]], Y[N[3]] - Y[N[0]], Z[N[3]] - Z[N[0]]};
    auto cross = [](const double u[3], const double v[3], double w[3]) {
      w[0] = u[1] * v[2] - v[1] * u[2];
      w[1] = u[2] * v[0] - v[2] * u[0];
      w[2] = u[0] * v[1] - v[0] * u[1];
    };
    double g[4][3];
    cross(ca, da, g[1]);
    cross(da, ba, g[2]);
    cross(ba, ca, g[3]);
    for (int k = 0; k < 3; ++k) g[0][k] = -g[1][k] - g[2][k] - g[3][k];
    const double J = ba[0] * g[1][0] + ba[1] * g[1][1] + ba[2] * g[1][2];
    if (!(J > 0.0)) return fail(c, XG_ERR_ARG, "chocg_set_theta: element Jacobian non-positive");
    for (int a = 0; a < 4; ++a)
      for (int b = 0; b < 4; ++b) {
        const int64_t q = pos(int64_t(N[a]), int64_t(N[b]));
        M[q] += J / 120.0 * ((a == b) ? 2.0 : 1.0);
        K[q] += (g[a][0] * g[b][0] + g[a][1] * g[b][1] + g[a][2] * g[b][2]) / J / 6.0;
      }
  }
  // three components per node: row 3i + c, columns 3j + c
  std::vector<uint64_t> ia3(n * 3 + 1, 0), ja3;
  std::vector<double> K3, M3;
  ja3.reserve(ja.size() * 3);
  K3.reserve(ja.size() * 3);
  M3.reserve(ja.size() * 3);
  for (int64_t i = 0; i < n; ++i)
    for (int cc = 0; cc < 3; ++cc) {
      for (uint64_t k = ia[i]; k < ia[i + 1]; ++k) {
        ja3.push_back(uint64_t(ja[k]) * 3 + cc);
        K3.push_back(K[k]);
        M3.push_back(M[k]);
      }
      ia3[i * 3 + cc + 1] = ja3.size();
    }
  // the momentum CG system, set up while it stands in for the context's
  CGDev* const saved = c->cg;
  c->cg = nullptr;
  rc = xg_cg_setup(c, n * 3, ia3.data(), ja3.data(), K3.data(), 0);
  d->mom = c->cg;
  if (rc == XG_OK) {
    const int64_t nent = cg_nent(c);
    for (int pass = 0; pass < 2; ++pass) {
      Arena& A = d->momarena;
      A.plan(d->baseK, nent);
      A.plan(d->baseM, nent);
      A.plan(d->R3, n * 3);
      A.plan(d->b3, n * 3);
      if (pass == 0) {
        const cudaError_t ce = A.reserve();
        if (ce != cudaSuccess) {
          rc = fail(c, XG_ERR_CUDA, std::string("chocg_set_theta: ") + cudaGetErrorString(ce));
          break;
        }
      }
    }
    if (rc == XG_OK) rc = cg_to_sell(c, ia3.data(), K3.data(), d->baseK);
    if (rc == XG_OK) rc = cg_to_sell(c, ia3.data(), M3.data(), d->baseM);
  }
  c->cg = saved;
  if (rc) {
    if (d->mom) destroy_cg(d->mom);
    d->mom = nullptr;
    d->momarena.release();
    return rc;
  }
  d->theta = theta;
  d->mom_pc = mom_pc;
  d->mom_iter = mom_iter;
  d->mom_tol = mom_tol;
  d->mommask_up = false;
  d->last_mit = 0;
  return XG_OK;
  XG_HOST_CATCH(c)
}

int xg_chocg_momentum_its(xg_ctx* c, int64_t* it) {
  ChoCGDev* d = nullptr;
  int rc = get_ctx(c, &d, false);
  if (rc) return rc;
  if (it) *it = d->last_mit;
  return XG_OK;
}

int xg_chocg_set_bc(xg_ctx* c, int64_t ndir, const uint64_t* dirnodes, const int32_t* dirmask,
                    const double* dirvals, int64_t nsym, const uint64_t* symnodes,
                    const double* symnorms, int64_t nnoslip, const uint64_t* noslipnodes,
                    int64_t npdir, const uint64_t* pdirnodes, const double* pdirvals) {
  XG_HOST_TRY
  ChoCGDev* d = nullptr;
  int rc = get_ctx(c, &d, false);
  if (rc) return rc;
  if ((ndir && (!dirnodes || !dirmask || !dirvals)) || (nsym && (!symnodes || !symnorms)) ||
      (nnoslip && !noslipnodes) || (npdir && (!pdirnodes || !pdirvals)) || ndir < 0 ||
      nsym < 0 || nnoslip < 0 || npdir < 0)
    return fail(c, XG_ERR_ARG, "chocg_set_bc: bad BC arrays");
  const int64_t n = d->n;
  auto bad = [&](uint64_t id) { return id >= static_cast<uint64_t>(n); };
  // BC program: one entry per distinct BC node, in node order
  std::vector<int32_t> dirof(n, -1), noslip(n, 0);
  std::vector<std::vector<int32_t>> symof;
  for (int64_t k = 0; k < ndir; ++k) {
    if (bad(dirnodes[k])) return fail(c, XG_ERR_ARG, "chocg_set_bc: Dirichlet node out of range");
    dirof[dirnodes[k]] = static_cast<int32_t>(k);
  }
  for (int64_t k = 0; k < nnoslip; ++k) {
    if (bad(noslipnodes[k])) return fail(c, XG_ERR_ARG, "chocg_set_bc: noslip node out of range");
    noslip[noslipnodes[k]] = 1;
  }
  std::vector<int64_t> symcount(n, 0);
  for (int64_t k = 0; k < nsym; ++k) {
    if (bad(symnodes[k])) return fail(c, XG_ERR_ARG, "chocg_set_bc: symmetry node out of range");
    ++symcount[symnodes[k]];
  }
  std::vector<int32_t> node, dir, nsl, symp(1, 0);
  std::vector<double> symn;
  std::vector<std::vector<int64_t>> symlist(n);
  for (int64_t k = 0; k < nsym; ++k) symlist[symnodes[k]].push_back(k);
  for (int64_t p = 0; p < n; ++p) {
    if (dirof[p] < 0 && !noslip[p] && symcount[p] == 0) continue;
    node.push_back(static_cast<int32_t>(p));
    dir.push_back(dirof[p]);
    nsl.push_back(noslip[p]);
    for (int64_t k : symlist[p])
      for (int a = 0; a < 3; ++a) symn.push_back(symnorms[k * 3 + a]);
    symp.push_back(static_cast<int32_t>(symn.size() / 3));
  }
  d->bcarena.release();
  d->nbc = static_cast<int64_t>(node.size());
  for (int pass = 0; pass < 2; ++pass) {
    Arena& A = d->bcarena;
    A.plan(d->bcnode, std::max<size_t>(1, node.size()));
    A.plan(d->bcdir, std::max<size_t>(1, dir.size()));
    A.plan(d->bcnoslip, std::max<size_t>(1, nsl.size()));
    A.plan(d->bcsymp, symp.size());
    A.plan(d->symn, std::max<size_t>(1, symn.size()));
    A.plan(d->dirmask, std::max<int64_t>(1, ndir * 3));
    A.plan(d->dirval, std::max<int64_t>(1, ndir * 3));
    if (pass == 0) XG_CUDA(c, A.reserve());
  }
  auto up = [&](void* dst, const void* src, size_t bytes) { return upload(c, dst, src, bytes); };
  XG_CUDA(c, up(d->bcnode, node.data(), node.size() * 4));
  XG_CUDA(c, up(d->bcdir, dir.data(), dir.size() * 4));
  XG_CUDA(c, up(d->bcnoslip, nsl.data(), nsl.size() * 4));
  XG_CUDA(c, up(d->bcsymp, symp.data(), symp.size() * 4));
  XG_CUDA(c, up(d->symn, symn.data(), symn.size() * 8));
  XG_CUDA(c, up(d->dirmask, dirmask, ndir * 3 * 4));
  XG_CUDA(c, up(d->dirval, dirvals, ndir * 3 * 8));
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  // Dirichlet rows of the theta-implicit momentum system (ChoCG::solve,
  // ChoCG.cpp:1580-1600): the masked velocity components of the Dirichlet
  // nodes and all three of the noslip nodes, increment 0
  d->mommask.assign(n * 3, 0);
  for (int64_t k = 0; k < ndir; ++k)
    for (int cc = 0; cc < 3; ++cc)
      if (dirmask[k * 3 + cc]) d->mommask[dirnodes[k] * 3 + cc] = 1;
  for (int64_t k = 0; k < nnoslip; ++k)
    for (int cc = 0; cc < 3; ++cc) d->mommask[noslipnodes[k] * 3 + cc] = 1;
  d->mommask_up = false;
  // pressure Dirichlet nodes on the context's CG system
  if (cg_rows(c) != n)
    return fail(c, XG_ERR_STATE, "chocg_set_bc: set up the pressure matrix (xg_cg_setup) first");
  std::vector<uint8_t> mask(n, 0);
  std::vector<double> val(n, 0.0);
  for (int64_t k = 0; k < npdir; ++k) {
    if (bad(pdirnodes[k]))
      return fail(c, XG_ERR_ARG, "chocg_set_bc: pressure Dirichlet node out of range");
    mask[pdirnodes[k]] = 1;
    val[pdirnodes[k]] = pdirvals[k];
  }
  rc = cg_set_dirichlet(c, mask.data(), val.data());
  if (rc) return rc;
  d->pdir_set = true;
  return XG_OK;
  XG_HOST_CATCH(c)
}

int xg_chocg_set_state(xg_ctx* c, const double* u, const double* p, double t) {
  ChoCGDev* d = nullptr;
  int rc = get_ctx(c, &d, false);
  if (rc) return rc;
  if (!u) return fail(c, XG_ERR_ARG, "chocg_set_state: null velocity");
  const int64_t n = d->n;
  XG_CUDA(c, cudaMemcpyAsync(d->stage, u, n * 3 * 8, cudaMemcpyHostToDevice, c->stream));
  k_aos_soa<<<blocks_for(n * 3, kBlock), kBlock, 0, c->stream>>>(n, 3, d->stage, d->u);
  XG_CHECK_LAUNCH(c);
  if (p)
    XG_CUDA(c, cudaMemcpyAsync(d->pr, p, n * 8, cudaMemcpyHostToDevice, c->stream));
  else
    XG_CUDA(c, cudaMemsetAsync(d->pr, 0, n * 8, c->stream));
  XG_CUDA(c, cudaMemsetAsync(d->pgrad, 0, n * 3 * 8, c->stream));
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  d->t = t;
  d->ready = false;
  return XG_OK;
}

int xg_chocg_get_state(xg_ctx* c, double* u, double* p, double* t) {
  ChoCGDev* d = nullptr;
  int rc = get_ctx(c, &d, false);
  if (rc) return rc;
  const int64_t n = d->n;
  if (u) {
    k_soa_aos<<<blocks_for(n * 3, kBlock), kBlock, 0, c->stream>>>(n, 3, d->u, d->stage);
    XG_CHECK_LAUNCH(c);
    XG_CUDA(c, cudaMemcpyAsync(u, d->stage, n * 3 * 8, cudaMemcpyDeviceToHost, c->stream));
  }
  if (p) XG_CUDA(c, cudaMemcpyAsync(p, d->pr, n * 8, cudaMemcpyDeviceToHost, c->stream));
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  if (t) *t = d->t;
  return XG_OK;
}

int xg_chocg_init(xg_ctx* c, int64_t* it) {
  ChoCGDev* d = nullptr;
  int rc = get_ctx(c, &d, true);
  if (rc) return rc;
  if (!d->pdir_set) return fail(c, XG_ERR_STATE, "chocg_init: no BCs (xg_chocg_set_bc)");
  // m_np = 0 (ChoCG::merge -> div -> pinit -> psolve -> sgrad -> psolved):
  // BCs, divergence without stabilisation, projection with dt = 1
  rc = launch_bc(c, d, d->u, 0);
  if (rc) return rc;
  rc = cg_zero_solution(c);
  if (rc) return rc;
  rc = launch_div(c, d, d->u, 0.0, 0, 0);
  if (rc) return rc;
  rc = pressure_solve(c, d, 0);
  if (rc) return rc;
  rc = launch_grad<1, GRAD_PROJECT>(c, d, cg_solution_device(c), nullptr, 1.0, 0);
  if (rc) return rc;
  rc = launch_bc(c, d, d->u, 0);
  if (rc) return rc;
  // m_np = 1 (velgrad -> flux -> div -> pinit -> psolve -> psolved): the
  // divergence of the volume-divided momentum flux with symmetry applied
  rc = launch_grad<3, GRAD_DIVIDE>(c, d, d->u, d->vgrad);
  if (rc) return rc;
  // the node tensors in the staging buffer ([9][n])
  k_mflux<<<blocks_for(d->n, kNode), kNode, 0, c->stream>>>(d->n, d->u, d->vgrad, d->prm.mu,
                                                            d->stage);
  two_pass<k_cflux<false>, k_cflux<true>>(c->stream, d->n, d->nbn, d->n, adj_of(d), d->stage,
                                          bnd_of(d), d->ivol, 1, d->flx);
  XG_CHECK_LAUNCH(c);
  rc = launch_bc(c, d, d->flx, 1);
  if (rc) return rc;
  rc = launch_div(c, d, d->flx, 0.0, 0, 0);
  if (rc) return rc;
  rc = pressure_solve(c, d, 0);
  if (rc) return rc;
  // m_np = 2: initial pressure and its gradient
  XG_CUDA(c, cudaMemcpyAsync(d->pr, cg_solution_device(c), d->n * 8, cudaMemcpyDeviceToDevice,
                             c->stream));
  rc = launch_grad<1, GRAD_DIVIDE>(c, d, d->pr, d->pgrad);
  if (rc) return rc;
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  d->ready = true;
  if (it) *it = d->last_it;
  return XG_OK;
}

int xg_chocg_run(xg_ctx* c, int64_t nstep, double* dts, int64_t* its, float* ms) {
  ChoCGDev* d = nullptr;
  int rc = get_ctx(c, &d, true);
  if (rc) return rc;
  if (!d->ready) return fail(c, XG_ERR_STATE, "chocg_run before chocg_init");
  const int64_t n = d->n;
  static const double rkc[4][4] = {{1.0, 0, 0, 0},
                                   {1.0 / 2.0, 1.0, 0, 0},
                                   {1.0 / 3.0, 1.0 / 2.0, 1.0, 0},
                                   {1.0 / 4.0, 1.0 / 3.0, 1.0 / 2.0, 1.0}};
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (ms) {
    XG_CUDA(c, cudaEventCreate(&e0));
    XG_CUDA(c, cudaEventCreate(&e1));
    XG_CUDA(c, cudaEventRecord(e0, c->stream));
  }
  int status = XG_OK;
  for (int64_t st = 0; st < nstep; ++st) {
    double dt = 0.0;
    rc = step_dt(c, d, &dt);
    if (rc) return rc;
    if (dt < DBL_EPSILON) {
      status = XG_ERR_BLOWUP;
      fail(c, XG_ERR_BLOWUP, "chocg: dt below eps");
      break;
    }
    // momentum prediction (ChoCG::rhs -> solve -> pred -> corr, per stage)
    for (int k = 0; k < d->prm.rk; ++k) {
      if (d->mom && k + 1 == d->prm.rk) {
        // semi-implicit last stage: the stage rhs, then the momentum solve
        rc = launch_rhs(c, d, d->u, 0.0, 0, nullptr, d->R3);
        if (rc) return rc;
        if (k == 0) XG_CUDA(c, cudaMemcpyAsync(d->un, d->u, n * 3 * 8, cudaMemcpyDeviceToDevice,
                                              c->stream));
        rc = momentum_solve(c, d, dt);
        if (rc) return rc;
      } else {
        rc = launch_rhs(c, d, d->u, rkc[d->prm.rk - 1][k] * dt, k == 0, d->u2, nullptr);
        if (rc) return rc;
        std::swap(d->u, d->u2);
      }
      rc = launch_bc(c, d, d->u, 0);
      if (rc) return rc;
      if (d->prm.flux == XG_DAMP4) {
        rc = launch_grad<3, GRAD_DIVIDE>(c, d, d->u, d->vgrad);
        if (rc) return rc;
      }
    }
    // pressure increment (ChoCG::div -> pinit -> psolve) and projection
    // (sgrad -> psolved -> pgrad)
    rc = launch_div(c, d, d->u, dt, 1, 1);
    if (rc) return rc;
    rc = pressure_solve(c, d, 1);
    if (rc) return rc;
    rc = launch_grad<1, GRAD_PROJECT>(c, d, cg_solution_device(c), nullptr, dt, 1);
    if (rc) return rc;
    rc = launch_bc(c, d, d->u, 0);
    if (rc) return rc;
    rc = launch_grad<1, GRAD_DIVIDE>(c, d, d->pr, d->pgrad);
    if (rc) return rc;
    d->t += dt;
    if (dts) dts[st] = dt;
    if (its) its[st] = d->last_it;
  }
  if (ms) {
    XG_CUDA(c, cudaEventRecord(e1, c->stream));
    XG_CUDA(c, cudaEventSynchronize(e1));
    XG_CUDA(c, cudaEventElapsedTime(ms, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
  }
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  return status;
}

int xg_chocg_fields(xg_ctx* c, int what, double* out) {
  ChoCGDev* d = nullptr;
  int rc = get_ctx(c, &d, false);
  if (rc) return rc;
  if (!out) return fail(c, XG_ERR_ARG, "chocg_fields: null output");
  const int64_t n = d->n;
  const double* src = nullptr;
  int nc = 1;
  switch (what) {
    case 0: src = d->un; nc = 3; break;
    case 1: src = d->pgrad; nc = 3; break;
    case 2: src = d->vgrad; nc = 9; break;
    case 3: src = d->div; break;
    case 4:
      src = cg_solution_device(c);
      if (!src || cg_rows(c) != n) return fail(c, XG_ERR_STATE, "chocg_fields: no pressure solve");
      break;
    default: return fail(c, XG_ERR_ARG, "chocg_fields: unknown field");
  }
  k_soa_aos<<<blocks_for(n * nc, kBlock), kBlock, 0, c->stream>>>(n, nc, src, d->stage);
  XG_CHECK_LAUNCH(c);
  XG_CUDA(c, cudaMemcpyAsync(out, d->stage, n * nc * 8, cudaMemcpyDeviceToHost, c->stream));
  XG_CUDA(c, cudaStreamSynchronize(c->stream));
  return XG_OK;
}

// ---- drop-ins: host node-major arrays through per-call device buffers (the
// device state of xg_chocg_run is left untouched)

int xg_chorin_div(xg_ctx* c, const double* U, const double* P, const double* G, double dt,
                  int stab, double* D) {
  ChoCGDev* d = nullptr;
  int rc = get_ctx(c, &d, false);
  if (rc) return rc;
  if (!U || !P || !G || !D) return fail(c, XG_ERR_ARG, "chorin_div: null array");
  const int64_t n = d->n;
  double *u, *p, *g, *out;
  Arena A;
  for (int pass = 0; pass < 2; ++pass) {
    A.plan(u, 3 * n);
    A.plan(p, n);
    A.plan(g, 3 * n);
    A.plan(out, 3 * n);
    if (pass == 0) XG_CUDA(c, A.reserve());
  }
  cudaStream_t s = c->stream;
  XG_CUDA(c, cudaMemcpyAsync(out, U, n * 24, cudaMemcpyHostToDevice, s));
  k_aos_soa<<<blocks_for(n * 3, kBlock), kBlock, 0, s>>>(n, 3, out, u);
  XG_CUDA(c, cudaMemcpyAsync(out, G, n * 24, cudaMemcpyHostToDevice, s));
  k_aos_soa<<<blocks_for(n * 3, kBlock), kBlock, 0, s>>>(n, 3, out, g);
  XG_CUDA(c, cudaMemcpyAsync(p, P, n * 8, cudaMemcpyHostToDevice, s));
  two_pass<k_cdiv<false>, k_cdiv<true>>(s, n, d->nbn, n, adj_of(d), u, p, g, bnd_of(d), dt, stab,
                                        0, out);
  XG_CHECK_LAUNCH(c);
  XG_CUDA(c, cudaMemcpyAsync(D, out, n * 8, cudaMemcpyDeviceToHost, s));
  XG_CUDA(c, cudaStreamSynchronize(s));
  return XG_OK;
}

int xg_chorin_grad(xg_ctx* c, const double* S, double* Gout) {
  ChoCGDev* d = nullptr;
  int rc = get_ctx(c, &d, false);
  if (rc) return rc;
  if (!S || !Gout) return fail(c, XG_ERR_ARG, "chorin_grad: null array");
  const int64_t n = d->n;
  double *sv, *g, *out;
  Arena A;
  for (int pass = 0; pass < 2; ++pass) {
    A.plan(sv, n);
    A.plan(g, 3 * n);
    A.plan(out, 3 * n);
    if (pass == 0) XG_CUDA(c, A.reserve());
  }
  cudaStream_t s = c->stream;
  XG_CUDA(c, cudaMemcpyAsync(sv, S, n * 8, cudaMemcpyHostToDevice, s));
  two_pass<k_cgrad<1, GRAD_RAW, false>, k_cgrad<1, GRAD_RAW, true>>(
      s, n, d->nbn, n, adj_of(d), sv, bnd_of(d), d->ivol, g, 0.0, 0, nullptr, nullptr);
  XG_CHECK_LAUNCH(c);
  k_soa_aos<<<blocks_for(n * 3, kBlock), kBlock, 0, s>>>(n, 3, g, out);
  XG_CUDA(c, cudaMemcpyAsync(Gout, out, n * 24, cudaMemcpyDeviceToHost, s));
  XG_CUDA(c, cudaStreamSynchronize(s));
  return XG_OK;
}

int xg_chorin_vgrad(xg_ctx* c, const double* U, double* Gout) {
  ChoCGDev* d = nullptr;
  int rc = get_ctx(c, &d, false);
  if (rc) return rc;
  if (!U || !Gout) return fail(c, XG_ERR_ARG, "chorin_vgrad: null array");
  const int64_t n = d->n;
  double *u, *g, *out;
  Arena A;
  for (int pass = 0; pass < 2; ++pass) {
    A.plan(u, 3 * n);
    A.plan(g, 9 * n);
    A.plan(out, 9 * n);
    if (pass == 0) XG_CUDA(c, A.reserve());
  }
  cudaStream_t s = c->stream;
  XG_CUDA(c, cudaMemcpyAsync(out, U, n * 24, cudaMemcpyHostToDevice, s));
  k_aos_soa<<<blocks_for(n * 3, kBlock), kBlock, 0, s>>>(n, 3, out, u);
  two_pass<k_cgrad<3, GRAD_RAW, false>, k_cgrad<3, GRAD_RAW, true>>(
      s, n, d->nbn, n, adj_of(d), u, bnd_of(d), d->ivol, g, 0.0, 0, nullptr, nullptr);
  XG_CHECK_LAUNCH(c);
  k_soa_aos<<<blocks_for(n * 9, kBlock), kBlock, 0, s>>>(n, 9, g, out);
  XG_CUDA(c, cudaMemcpyAsync(Gout, out, n * 72, cudaMemcpyDeviceToHost, s));
  XG_CUDA(c, cudaStreamSynchronize(s));
  return XG_OK;
}

int xg_chorin_flux(xg_ctx* c, const double* U, const double* G, double* F) {
  ChoCGDev* d = nullptr;
  int rc = get_ctx(c, &d, false);
  if (rc) return rc;
  if (!U || !G || !F) return fail(c, XG_ERR_ARG, "chorin_flux: null array");
  const int64_t n = d->n;
  double *u, *g, *f, *tmp;
  Arena A;
  for (int pass = 0; pass < 2; ++pass) {
    A.plan(u, 3 * n);
    A.plan(g, 9 * n);
    A.plan(f, 3 * n);
    A.plan(tmp, 9 * n);
    if (pass == 0) XG_CUDA(c, A.reserve());
  }
  cudaStream_t s = c->stream;
  XG_CUDA(c, cudaMemcpyAsync(tmp, U, n * 24, cudaMemcpyHostToDevice, s));
  k_aos_soa<<<blocks_for(n * 3, kBlock), kBlock, 0, s>>>(n, 3, tmp, u);
  XG_CUDA(c, cudaMemcpyAsync(tmp, G, n * 72, cudaMemcpyHostToDevice, s));
  k_aos_soa<<<blocks_for(n * 9, kBlock), kBlock, 0, s>>>(n, 9, tmp, g);
  k_mflux<<<blocks_for(n, kNode), kNode, 0, s>>>(n, u, g, d->prm.mu, tmp);
  two_pass<k_cflux<false>, k_cflux<true>>(s, n, d->nbn, n, adj_of(d), tmp, bnd_of(d), d->ivol, 0,
                                          f);
  XG_CHECK_LAUNCH(c);
  k_soa_aos<<<blocks_for(n * 3, kBlock), kBlock, 0, s>>>(n, 3, f, tmp);
  XG_CUDA(c, cudaMemcpyAsync(F, tmp, n * 24, cudaMemcpyDeviceToHost, s));
  XG_CUDA(c, cudaStreamSynchronize(s));
  return XG_OK;
}

int xg_chorin_rhs(xg_ctx* c, const double* P, const double* U, const double* G, double* R) {
  ChoCGDev* d = nullptr;
  int rc = get_ctx(c, &d, false);
  if (rc) return rc;
  if (!P || !U || !G || !R) return fail(c, XG_ERR_ARG, "chorin_rhs: null array");
  const int64_t n = d->n;
  double *u, *g, *p, *r, *tmp;
  Arena A;
  for (int pass = 0; pass < 2; ++pass) {
    A.plan(u, 3 * n);
    A.plan(g, 9 * n);
    A.plan(p, n);
    A.plan(r, 3 * n);
    A.plan(tmp, 9 * n);
    if (pass == 0) XG_CUDA(c, A.reserve());
  }
  cudaStream_t s = c->stream;
  XG_CUDA(c, cudaMemcpyAsync(tmp, U, n * 24, cudaMemcpyHostToDevice, s));
  k_aos_soa<<<blocks_for(n * 3, kBlock), kBlock, 0, s>>>(n, 3, tmp, u);
  XG_CUDA(c, cudaMemcpyAsync(tmp, G, n * 72, cudaMemcpyHostToDevice, s));
  k_aos_soa<<<blocks_for(n * 9, kBlock), kBlock, 0, s>>>(n, 9, tmp, g);
  XG_CUDA(c, cudaMemcpyAsync(p, P, n * 8, cudaMemcpyHostToDevice, s));
  const AdvPrm ap = adv_of(d);
  if (d->prm.flux == XG_DAMP4)
    two_pass<k_crhs<true, false>, k_crhs<true, true>>(s, n, d->nbn, n, adj_of(d), u, g, p,
                                                       bnd_of(d), ap, d->ivol, 0.0, 0, nullptr,
                                                       nullptr, r);
  else
    two_pass<k_crhs<false, false>, k_crhs<false, true>>(s, n, d->nbn, n, adj_of(d), u, g, p,
                                                         bnd_of(d), ap, d->ivol, 0.0, 0, nullptr,
                                                         nullptr, r);
  XG_CHECK_LAUNCH(c);
  k_soa_aos<<<blocks_for(n * 3, kBlock), kBlock, 0, s>>>(n, 3, r, tmp);
  XG_CUDA(c, cudaMemcpyAsync(R, tmp, n * 24, cudaMemcpyDeviceToHost, s));
  XG_CUDA(c, cudaStreamSynchronize(s));
  return XG_OK;
}

}  // extern "C"
