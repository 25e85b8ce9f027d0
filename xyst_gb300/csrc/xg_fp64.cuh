// Device helpers for kernels bound by GB300's narrow FP64 pipe.
#pragma once

#include <cuda_runtime.h>

namespace xg {
namespace {

// Comparisons of doubles on their bits: on GB300 an FP64 instruction holds
// its unit for 64 cycles, a comparison too, and integer ones run beside it.
// The key orders as the numbers do, with -0 at +0.
__device__ __forceinline__ long long order_key(double x) {
  const long long b = __double_as_longlong(x);
  return b < 0 ? (long long)(0x8000000000000000ull) - b : b;
}
__device__ __forceinline__ bool is_nan(double x) {
  // by halves: a compiler turns the 64-bit form back into an FP64 comparison
  return (unsigned(__double2hiint(x)) & 0x7fffffffu) + (__double2loint(x) != 0) > 0x7ff00000u;
}
// a < b, false with a NaN
__device__ __forceinline__ bool less(double a, double b) {
  return order_key(a) < order_key(b) && !is_nan(a) && !is_nan(b);
}
// a < -b
__device__ __forceinline__ bool less_neg(double a, double b) {
  return order_key(a) < -order_key(b) && !is_nan(a) && !is_nan(b);
}
// a <= b
__device__ __forceinline__ bool at_most(double a, double b) {
  return order_key(a) <= order_key(b) && !is_nan(a) && !is_nan(b);
}
__device__ __forceinline__ bool at_most(float a, float b) { return a <= b; }
__device__ __forceinline__ bool less(float a, float b) { return a < b; }
__device__ __forceinline__ bool less_neg(float a, float b) { return a < -b; }
// The sign of x - y (y not a NaN), 0 for a NaN x.
__device__ __forceinline__ int side(double x, double y) {
  const long long kx = order_key(x), ky = order_key(y);
  return is_nan(x) ? 0 : kx > ky ? 1 : kx < ky ? -1 : 0;
}
__device__ __forceinline__ int side(float x, float y) { return x > y ? 1 : x < y ? -1 : 0; }
// x with its sign flipped if `flip`, on the bits.
__device__ __forceinline__ double flip_if(double x, bool flip) {
  return __longlong_as_double(__double_as_longlong(x) ^ ((long long)(flip) << 63));
}
__device__ __forceinline__ float flip_if(float x, bool flip) {
  return __uint_as_float(__float_as_uint(x) ^ (unsigned(flip) << 31));
}
// |x| cut to a float and back, on the bits (conversions are as slow as FP64
// arithmetic), for 2^-120 <= |x| < 2^120 (in_float).
__device__ __forceinline__ bool in_float(double x) {
  return ((unsigned(__double2hiint(x)) >> 20) & 0x7ffu) - 903u < 240u;
}
__device__ __forceinline__ float cut_abs(double x) {
  const unsigned hi = unsigned(__double2hiint(x)) & 0x7fffffffu;
  return __uint_as_float(((hi - (896u << 20)) << 3) | (unsigned(__double2loint(x)) >> 29));
}
__device__ __forceinline__ double widen(float x, unsigned sign) {  // x > 0
  const unsigned b = __float_as_uint(x);
  return __hiloint2double(int(((b >> 3) + (896u << 20)) | sign), int(b << 29));
}
// 1/d from the FP32 approximation x of 1/d (about 22 bits): with e = 1 - d x,
// 1/d = x / (1 - e), taken to e^2 (the third-order Householder step; the rest
// is e^3, below 1e-18): three FP64 instructions, within 1.1e-16 (one rounding).
__device__ __forceinline__ double recip(double d) {
  if (!in_float(d)) return 1.0 / d;
  float a;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(cut_abs(d)));
  const double x = widen(a, unsigned(__double2hiint(d)) & 0x80000000u);
  const double e = fma(-d, x, 1.0);
  return fma(x, fma(e, e, e), x);
}
__device__ __forceinline__ float recip(float d) { return 1.0f / d; }
// a / b, in double as a times ib = recip(b), within 2.2e-16
__device__ __forceinline__ double over(double a, double, double ib) { return a * ib; }
__device__ __forceinline__ float over(float a, float b, float) { return a / b; }
// sqrt: in double from the FP32 approximation y of 1/sqrt(x) (about 22 bits):
// with s = x y and e = 1 - x y^2, sqrt(x) = s / sqrt(1 - e) =
// s (1 + e/2 + 3 e^2/8 + ...), the rest below 1e-18: five FP64 instructions,
// within 1.7e-16; the library's root for negative x and outside FP32's range.
__device__ __forceinline__ double xsqrt(double x) {
  if (!in_float(x) || __double2hiint(x) < 0) return sqrt(x);
  float a;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(a) : "f"(cut_abs(x)));
  const double y = widen(a, 0u);
  const double s = x * y, e = fma(-s, y, 1.0);
  return fma(s * e, fma(0.375, e, 0.5), s);
}
// In float x * rsqrt(x) (x >= 0).
__device__ __forceinline__ float xsqrt(float x) { return x > 0.f ? x * rsqrtf(x) : 0.f; }

// A node's CFL time step before the CFL factor (src/Inciter/RieCG.cpp:827-838,
// KozCG.cpp:613-688), L = cbrt(vol), with one quotient by the density: a
// division is about ten FP64 instructions.
__device__ __forceinline__ double node_dt(const double u[5], double L, double g) {
  const double ir = recip(u[0]);
  const double uu = u[1] * ir, vv = u[2] * ir, ww = u[3] * ir;
  const double k2 = uu * uu + vv * vv + ww * ww;
  const double pr = (u[4] - 0.5 * u[0] * k2) * (g - 1.0);
  const double c = xsqrt(g * fmax(pr, 0.0) * ir);
  return L * recip(fmax(xsqrt(k2) + c, 1.0e-8));
}

}  // namespace
}  // namespace xg
