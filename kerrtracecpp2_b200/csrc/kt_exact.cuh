// kt_exact.cuh -- correctly rounded quotients for the exact right-hand sides.
//
// The exact kernels spend two fifths of their FP64 pipe on IEEE divisions:
// five quotients per inverse metric over three denominators.  The compiler's
// division handles every operand and is expanded per quotient with its own
// reciprocal, range test and slow-path call.  Here the operands are known to
// lie in a moderate range (a test per right-hand side, below), quotients over
// one denominator share its reciprocal, and there is no slow path inline.
//
// Method: Newton-Raphson reciprocal and the quotient correction of
// P. Markstein (IBM J. Res. Dev. 34(1), 1990), in this form.  For b > 0 with
// significand b_m in [1, 2) (signs do not matter):
//   y0 = 1/b within 2^-19 (the hardware seed);
//   y1 = y0 + y0 (1 - b y0), within 2^-38;  y2 = y1 + y1 (1 - b y1), whose
//   value before its rounding is within 2^-74 of 1/b, so y2 = (1 + d)/b with
//   |d| <= 2^-54 b_m + 2^-74;
//   q0 = RN(a y1), q1 = RN(q0 + y1 RN(a - b q0)): before its rounding within
//   2^-74 of a/b, so |q1 - a/b| <= (1/2 + 2^-20) ulp;
//   r = a - b q1 is exact, and q = RN(q1 + r y2).
// q1 + r y2 = a/b + (a/b - q1) d, off by less than (1/2 + 2^-20) |d| ulp.
// a/b in units of its ulp is an integer over b_i = 2^52 b_m and never a
// rounding midpoint, so it lies at least 1/(2 b_i) from every midpoint, and q
// is RN(a/b) when (1 + 2^-19) |d| < 1/b_i, that is when
// b_m^2 (1 + 2^-19) + 2^-20 b_m (1 + 2^-19) < 4: for all b_m < 2 - 2^-18.
// (Two more operations per quotient than the single correction: with only
// q0 = RN(a y2), which can be 1.5 ulp off, the bound fails for b_m > 1.15.)
// The excluded significands (the top 18 bits all ones) are part of the
// range test; their quotients take the division.  Nothing over- or
// underflows for |b| in [2^-350, 2^300] and non-zero |a| in [2^-500, 2^500]
// (the smallest intermediate, a residual, is 2^-106 |a|).
#pragma once

#include "ktmath.h"

#if defined(__CUDACC__)
#define KT_EX __host__ __device__ __forceinline__
#else
#define KT_EX inline
#endif

namespace kt {

KT_EX uint32_t hi_word(double x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2hiint(x);
#else
  return (uint32_t)(ktm_bits(x) >> 32);
#endif
}
KT_EX uint32_t lo_word(double x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2loint(x);
#else
  return (uint32_t)ktm_bits(x);
#endif
}

// 2^-k <= |x| < 2^k, from the high word.
KT_EX bool in_range(double x, int k) {
  const uint32_t lo = (uint32_t)(1023 - k) << 20, span = (uint32_t)(2 * k) << 20;
  return (hi_word(x) & 0x7fffffffu) - lo < span;
}
KT_EX bool is_zero(double x) { return ((hi_word(x) & 0x7fffffffu) | lo_word(x)) == 0u; }

// Bit kTopBit is set when the significand's top 18 bits are all ones.
constexpr uint32_t kTopBit = 1u << 20;
KT_EX uint32_t top_ones(double b) {
  const uint32_t h = hi_word(b);
  return (h + 4u) ^ h;
}

// 1/b within 2^-19 (the hardware's largest error, over every significand, is
// 2^-19.94; tests/exact_device.cu).  The host twin keeps 20 bits.
KT_EX double rcp_seed(double b) {
#if defined(__CUDA_ARCH__)
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
#else
  return ktm_from_bits(ktm_bits(1.0 / b) & 0xffffffff00000000ull);
#endif
}

// The two reciprocals (y1, y2) of a denominator.
struct Rcp {
  double b, y1, y2;
};
KT_EX Rcp make_rcp_seeded(double b, double y0) {
  Rcp R;
  R.b = b;
  R.y1 = fma(fma(-b, y0, 1.0), y0, y0);
  R.y2 = fma(fma(-b, R.y1, 1.0), R.y1, R.y1);
  return R;
}
KT_EX Rcp make_rcp(double b) { return make_rcp_seeded(b, rcp_seed(b)); }
// RN(a / b); a zero numerator gives a zero of either sign (quot_signed: of
// the quotient's).
KT_EX double quot(double a, const Rcp& R) {
  const double q0 = a * R.y1;
  const double q1 = fma(fma(-R.b, q0, a), R.y1, q0);
  return fma(fma(-R.b, q1, a), R.y2, q1);
}
KT_EX double quot_signed(double a, const Rcp& R) { return is_zero(a) ? a * R.y1 : quot(a, R); }
// RN(1 / b): q1 is y2.
KT_EX double quot_one(const Rcp& R) { return fma(fma(-R.b, R.y2, 1.0), R.y2, R.y2); }

// A denominator whose reciprocal is known within 2^-38 already.
KT_EX Rcp make_rcp_from(double b, double y1) {
  Rcp R;
  R.b = b;
  R.y1 = y1;
  R.y2 = fma(fma(-b, y1, 1.0), y1, y1);
  return R;
}

// ---- square roots ----------------------------------------------------------
// RN(sqrt(x)), and 1/sqrt(x) within 2^-52, which the quotients by the root
// and by its square start from (make_rcp_from).  Markstein's correction
// g + (x - g^2) h of an approximate root g, h = 1/(2 sqrt(x)):
//   y0 = 1/sqrt(x) within 2^-19 (the hardware seed: 2^-20.03);
//   e = 1 - RN(x y0) y0, y = y0 (1 + e/2 + 3 e^2/8) = (1 + d)/sqrt(x);
//   g = RN(x y), then two corrections with h = y/2.
// Scale x into [1, 4) and write sqrt(x) = K u with u = 2^-52, 2^52 <= K < 2^53,
// k = K/2^53.  In units of 2^-53, d has
//   1/(4 k) from the rounding of x y0 < 2 (half an ulp, 2^-53, over sqrt(x) =
//     2 k, halved by e/2; x y0 < 2 because x < 4 (1 - 2^-18), below),
//   0.157 from the term 5 e^3/16 left out, |e| < 2^-18 (1 + 2^-20),
//   k from y's own rounding (half an ulp of a number below 1), and less than
//   2^-15 from e's, the polynomial's and the product's:
// |d| k 2^53 < 1/4 + 0.157 k + k^2 + 2^-15 < 1.41, that is |d| < 1.41/K.
// The first correction leaves g within (1/2 + 2^-40) ulp.  For the second let
// g = K u now be its result and x - g^2 = D u^2 (exact in the fma: |D| < K +
// 2^14 < 2^53), so that sqrt(x) is g + D/(2 K) (1 - D/(4 K^2)) ulp and the
// correction adds c = D/(2 K) (1 - D/(2 K^2)) (1 + d) ulp, up to K^-2.
// RN(sqrt(x)) is g exactly when -K < D <= K, and the result is g when
// |c| < 1/2.  x is a multiple of 2^52 u^2, so K^2 + D is one of 2^52; with
// |D| = K + j (j of either sign) that makes j even, and j = 0 only for K = 2^52
// and K = 2^53 - 1, that is x next to a power of four, which the range test
// hands to sqrt().  From |j| >= 2 on, 2 |c| = (1 + j/K)(1 -+ 1/(2 K))(1 + d)
// lies on the side of 1 that j's sign says when |d| < (|j| - 1/2)/K, and
// 1.41 < 3/2.
KT_EX double rsqrt_seed(double x) {
#if defined(__CUDA_ARCH__)
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
#else
  return ktm_from_bits(ktm_bits(1.0 / sqrt(x)) & 0xffffffff00000000ull);
#endif
}
struct Root {
  double g, y;  // RN(sqrt(x)); 1/sqrt(x) within 2^-52
};
KT_EX Root make_root_seeded(double x, double y0) {
  Root R;
  const double e = fma(-(x * y0), y0, 1.0);
  R.y = fma(y0 * e, fma(0.375, e, 0.5), y0);
  const double h = 0.5 * R.y;
  double g = x * R.y;
  g = fma(fma(-g, g, x), h, g);
  R.g = fma(fma(-g, g, x), h, g);
  return R;
}
KT_EX Root make_root(double x) { return make_root_seeded(x, rsqrt_seed(x)); }
// Bit kTopBit is set when the significand's top 17 bits are all ones or all
// zeros (x >= 4 (1 - 2^-18) and x < 4 (1 + 2^-17) among them).
KT_EX uint32_t top_edge(double x) {
  const uint32_t h = hi_word(x);
  return ((h + 8u) ^ h) | ((h - 8u) ^ h);
}
// 2^-k <= x < 2^k (positive).
KT_EX bool in_range_pos(double x, int k) {
  const uint32_t lo = (uint32_t)(1023 - k) << 20, span = (uint32_t)(2 * k) << 20;
  return hi_word(x) - lo < span;
}

}  // namespace kt
