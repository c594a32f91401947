// fp64_math.cuh -- FP64 elementary functions for the walks of this library.
//
// GB300 issues one FP64 warp instruction per 64 cycles and SM partition, so the
// FP64 kernels are bound by the number of those instructions and by nothing
// else.  Measured (cycles of one warp, dependent calls): log 2087, exp 1334,
// a / b 641, sqrt 676, sincospi 1948, against 64 for one multiply-add.  The
// forms below trade arithmetic for small tables and integer work, which runs on
// other pipes:
//  - log and exp after the table-driven scheme of P. T. P. Tang (ACM TOMS 15,
//    1989 and 16, 1990): the argument's leading bits select a tabulated value,
//    a short Taylor polynomial of the small remainder does the rest;
//  - the reciprocal and the reciprocal square root refine the hardware's
//    approximation by the binomial series of its residual;
//  - comparisons, minima and uniforms on the bit patterns.
// Largest errors found against extended precision on the ranges that the walks use,
// in units of the last place: log 1.8 (below 3/4, where its two parts cancel), exp 1.0
// (their fine forms 1.1 and 0.51),
// 1/x 0.51, 1/sqrt 1.0, sqrt 1.7, a/b 1.5, 1/(beta gamma) 1.7 (bounds and their reasons:
// tests/test_gpu_fp64_bounds.py).  Outside (zeros, negative or subnormal arguments,
// infinities, NaN) log, exp and sqrt call CUDA's; the others are not used there.
#pragma once
#include <stdint.h>

#include "common.cuh"

namespace dp {
namespace f64 {

#include "fp64_tables.inc"

__device__ __forceinline__ int hi32(double x) { return __double2hiint(x); }
// The integer k as a double: one subtraction instead of a conversion.
__device__ __forceinline__ double from_int(int k) {
  return __hiloint2double(0x43300000, int(uint32_t(k) ^ 0x80000000u)) - 4503601774854144.0;
}

// A float as a double: integer work for normal values instead of a conversion.
__device__ __forceinline__ double widen(float f) {
  const uint32_t u = __float_as_uint(f), m = u & 0x7fffffffu;
  if (m - 0x00800000u >= 0x7f000000u) return double(f);  // zero, subnormal, infinity, NaN
  return __hiloint2double(int((u & 0x80000000u) | ((m >> 3) + 0x38000000u)), int(u << 29));
}
__device__ __forceinline__ double widen(double d) { return d; }

// log x, x normal and positive: 10 FP64 instructions.  x = 2^k m with m / c in
// [1 - 2^-9, 1 + 2^-9] of the table's c; c = 1 around x = 1, where the result
// is the polynomial alone.  FINE: 11, the sum of the tabulated parts being exact.
template <bool FINE>
__device__ __forceinline__ double log_by_table(double x) {
  const int hi = hi32(x);
  if (uint32_t(hi - 0x00100000) >= 0x7fe00000u) return ::log(x);
  const int k = ((hi + 0x00080800) >> 20) - 1023;
  const int j = ((hi & 0xfffff) + 0x800) >> 12;
  const double2 t = FINE ? kLogFine[j] : kLogTab[j];
  const double m = __hiloint2double(hi - (k << 20), __double2loint(x));
  const double r = fma(m, t.x, -1.0);
  const double p = fma(r, fma(r, fma(r, fma(r, -1.0 / 6.0, 0.2), -0.25), 1.0 / 3.0), -0.5);
  const double kd = from_int(k), q = fma(r * r, p, r);
  if (FINE) return fma(kd, 0.6931471805598903, t.y) + fma(kd, 5.497923018708371e-14, q);
  return fma(kd, 0.6931471805599453, t.y) + q;
}
__device__ __forceinline__ double log(double x) { return log_by_table<false>(x); }
__device__ __forceinline__ double log_fine(double x) { return log_by_table<true>(x); }

// exp x: 10 FP64 instructions; x = (128 k + j) log 2 / 128 + r, |r| <= log 2 / 256.
// FINE: 11, with the table's rounding.
template <bool FINE>
__device__ __forceinline__ double exp_by_table(double x) {
  if (uint32_t(hi32(x) & 0x7fffffff) >= 0x40862000u) return ::exp(x);  // |x| >= 708
  const double s = fma(x, 184.6649652337873, 6755399441055744.0);  // 1.5 2^52: nearest integer
  const int n = __double2loint(s);
  const double d = s - 6755399441055744.0;
  const double r = fma(d, -1.2864023111638346e-14, fma(d, -0.005415212348111709, x));
  const double p = fma(r, fma(r, fma(r, fma(r, 1.0 / 120.0, 1.0 / 24.0), 1.0 / 6.0), 0.5), 1.0);
  const double t = kExpTab[n & 127], y = FINE ? t + fma(t, r * p, kExpLow[n & 127]) : fma(t, r * p, t);
  return __hiloint2double(hi32(y) + ((n >> 7) << 20), __double2loint(y));
}
__device__ __forceinline__ double exp(double x) { return exp_by_table<false>(x); }
__device__ __forceinline__ double exp_fine(double x) { return exp_by_table<true>(x); }

// 1 / x for normal x whose reciprocal is normal: 3 FP64 instructions.
__device__ __forceinline__ double rcp(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ double div(double a, double b) { return a * rcp(b); }
// a / b correctly rounded, y = __drcp_rn(b): 5 FP64 instructions.  Markstein,
// "IA-64 and Elementary Functions" (2000): a quotient within one unit, corrected
// by its exact remainder times the rounded reciprocal, is the rounded one.  For b
// and the quotient well inside the normal range (a tiny a keeps a tiny quotient).
__device__ __forceinline__ double div_rn(double a, double b, double y) {
  double q = a * y;
  q = fma(fma(-b, q, a), y, q);
  return fma(fma(-b, q, a), y, q);
}

// 1 / sqrt(x) and sqrt(x) for normal positive x: 5 and 6 FP64 instructions.
__device__ __forceinline__ double rsqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}
__device__ __forceinline__ double sqrt(double x) { return x > 0.0 ? x * rsqrt(x) : ::sqrt(x); }

// sin(pi x) and cos(pi x) for |x| <= 1: 18 FP64 instructions; the nearest
// multiple of 1/32 from the table and quadrant symmetry, the remainder
// |d| <= pi / 64 by Taylor polynomials.
__device__ __forceinline__ void sincospi(double x, double* sn, double* cs) {
  const double s = fma(x, 32.0, 6755399441055744.0);
  const int n = __double2loint(s) & 63;
  const double d = fma(s - 6755399441055744.0, -0.03125, x) * kPi, d2 = d * d;
  const double sd = fma(d * d2, fma(d2, fma(d2, -1.0 / 5040.0, 1.0 / 120.0), -1.0 / 6.0), d);
  const double cd = d2 * fma(d2, fma(d2, fma(d2, 1.0 / 40320.0, -1.0 / 720.0), 1.0 / 24.0), -0.5);  // cos d - 1
  const int q = n >> 4, j = n & 15;
  const double2 t = kSinTab[j];
  const double a = fma(t.x, cd, fma(t.y, sd, t.x)), b = fma(t.y, cd, fma(-t.x, sd, t.y));
  // quadrant q of pi/2: (sin, cos) -> (cos, -sin) ...
  const double u = (q & 1) ? b : a, v = (q & 1) ? a : b;
  *sn = __hiloint2double(hi32(u) ^ ((q & 2) << 30), __double2loint(u));
  *cs = __hiloint2double(hi32(v) ^ (((q + 1) & 2) << 30), __double2loint(v));
}

// a < b for non-negative a and b (or both NaN-free and of one order by bits).
__device__ __forceinline__ bool lt_pos(double a, double b) {
  return __double_as_longlong(a) < __double_as_longlong(b);
}
__device__ __forceinline__ double min_pos(double a, double b) { return lt_pos(b, a) ? b : a; }
__device__ __forceinline__ double max_pos(double a, double b) { return lt_pos(a, b) ? b : a; }

// Offset of lx, in widths, on the interval of the increasing grid x that it lies
// in: (lx - x[i]) inv[i] (inv: inverse widths), searched from interval i, which
// becomes that interval.  The searches decide by the sign and the exponent of the
// offset, which the caller wants anyway: no FP64 comparison.  One way only: beside
// a node the rounded offsets of both its intervals can point at the other one (a
// last place below a node near 0 is below 0 on the one and rounds to 1 on the
// other), and either then stands for the node.
__device__ __forceinline__ double grid_offset(const double* x, const double* inv, int n, double lx, int& i) {
  for (int way = 0;;) {
    const double t = (lx - x[i]) * inv[i];
    const int h = hi32(t), step = h < 0 && i > 0 ? -1 : (h >= 0x3ff00000 && i < n - 2 ? 1 : 0);
    if (step == 0 || step == -way) return t;
    way = step;
    i += step;
  }
}

// u01 on the bit pattern: m 2^-53 of the 53-bit integer m, no FP64 instruction.
__device__ __forceinline__ double uniform(uint32_t a, uint32_t b) {
  const uint64_t m = (uint64_t(a >> 5) << 26) | uint64_t(b >> 6);
  if (m == 0) return 0.0;
  const int z = __clzll(m);  // 11 ... 63
  return __longlong_as_double((m << (z - 11) & 0xfffffffffffffull) | (uint64_t(1033 - z) << 52));
}

// 1 / (beta gamma) at the kinetic energy x (in masses), beta >= 1e-6, and its
// derivative in x (src/Geometry.jl:1083-1107).
__device__ __forceinline__ double inv_beta_gamma(double x, double* d) {
  // x < 1e-12 (the clamp of beta; negative energies) or > 1e100 (x^2 overflows at 1e154)
  if (uint32_t(hi32(x)) - 0x3d719799u >= 0x54b249adu - 0x3d719799u) {
    const double g = 1.0 + x, b2 = 1.0 - 1.0 / (g * g);
    const double b = ::sqrt(b2 >= 1e-12 ? b2 : 1e-12), r = 1.0 / (b * g);
    *d = b2 >= 1e-12 ? -r / (b2 * g * g * g) - r / g : -r / g;
    return r;
  }
  const double r = rsqrt(x * (x + 2.0));  // gamma^2 - 1
  *d = -(x + 1.0) * (r * r * r);
  return r;
}

}  // namespace f64
}  // namespace dp
