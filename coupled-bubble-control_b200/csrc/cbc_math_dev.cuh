// cbc_math_dev.cuh -- device forms of the elementary functions of cbc_math.h
// for arguments in the normal range, several at a time and without a branch.
//
// They perform the same roundings in the same order as cbc_math.h, so every
// result has the same bits; what differs is how the machine gets there:
//   * N arguments go through every step together.  A dependent FP64
//     operation takes 8.4 cycles on a B200 and an independent one 2.1 (one
//     warp, measured), so one Horner chain alone leaves three quarters of the
//     pipe idle; interleaved chains fill it.
//   * No division and no reciprocal from the compiler: each of those ends in a
//     branch to its special cases, which cuts the block the scheduler works
//     on (four independent 1/x took 74 cycles each, the latency of one,
//     measured).  rcp() and quot() below have none.
//   * Rounding to an integer, conversion to int and scaling by 2^n are an
//     addition of 1.5 2^52 and integer operations on the exponent field.
// The caller guarantees the ranges given at each function (fast_until and
// state_in_range test them; outside, the general functions are taken).
#pragma once

#include "cbc_math.h"

namespace cbcd {

// 1.5 * 2^52: adding it rounds |v| < 2^51 to an integer, ties to even (as
// rint), and leaves that integer's two's complement in the low word.
constexpr double RINT_MAGIC = 6755399441055744.0;

// 1/x correctly rounded, for 2^-1000 <= |x| <= 2^1000, from a seed y of relative
// error |e0| < 2^-19, e0 = 1 - x y.  Three terms of the geometric series
// 1/x = y / (1 - e0) = y (1 + e0 + e0^2 + ...) leave e0^3 < 2^-57 before their
// rounding, then Markstein's correction y + y (1 - x y) (P. Markstein, "IA-64 and
// Elementary Functions", 2000, ch. 8): 1 - x y is exact, the corrected value differs
// from 1/x by e^2 / x with |e| the relative error of the rounded y.  A 53-bit
// quotient 1/x misses a rounding boundary by 2^-106 at least, and only where the
// significand X of x divides 2^106 - 1 with a 53-bit X: the only divisor of
// (2^53 - 1)(2^53 + 1) in [2^52, 2^53) is 2^53 - 1.  There 1/x lies just above the
// middle of 2^-k and its upper neighbour, which it rounds to; the correction ends
// on either of the two, with the sign of the seed's error, and both have the same
// high word, so the low word is set.
CBC_HD int low_word(double x) {
#if defined(__CUDA_ARCH__)
  return __double2loint(x);
#else
  return (int)(uint32_t)cbcm::double_to_bits(x);
#endif
}
CBC_HD int high_word(double x) {
#if defined(__CUDA_ARCH__)
  return __double2hiint(x);
#else
  return (int)(uint32_t)(cbcm::double_to_bits(x) >> 32);
#endif
}
CBC_HD double join_words(int hi, int lo) {
#if defined(__CUDA_ARCH__)
  return __hiloint2double(hi, lo);
#else
  return cbcm::bits_to_double((uint64_t)(uint32_t)hi << 32 | (uint32_t)lo);
#endif
}
CBC_HD double rcp_last(double x, double y) {
  const unsigned ones = (unsigned)low_word(x) & ((unsigned)high_word(x) | 0xfff00000u);
  return join_words(high_word(y), ones == 0xffffffffu ? 1 : low_word(y));
}
template <int N>
CBC_HD void rcp_refine(const double (&x)[N], double (&y)[N]) {
  double e[N];
#pragma unroll
  for (int i = 0; i < N; ++i) e[i] = fma(-x[i], y[i], 1.0);
#pragma unroll
  for (int i = 0; i < N; ++i) e[i] = fma(e[i], e[i], e[i]);
#pragma unroll
  for (int i = 0; i < N; ++i) y[i] = fma(e[i], y[i], y[i]);
#pragma unroll
  for (int i = 0; i < N; ++i) e[i] = fma(-x[i], y[i], 1.0);
#pragma unroll
  for (int i = 0; i < N; ++i) y[i] = rcp_last(x[i], fma(e[i], y[i], y[i]));
}
// The seed: relative error 2^-19.9 at most over all high words of the significand
// (measured), the only part of x that it depends on.
template <int N>
__device__ __forceinline__ void rcp(const double (&x)[N], double (&y)[N]) {
#pragma unroll
  for (int i = 0; i < N; ++i) asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y[i]) : "d"(x[i]));
  rcp_refine(x, y);
}

// a/b correctly rounded, for a and b with exponents well inside the range (no
// product or residual below under- or overflows): q = a y with y = 1/b, then
// two corrections q + y (a - b q).  After the first the error of q is half a
// unit and a little, so the residual of the second is exact and its product
// with y is off by less than 2^-53 units, while a 53-bit quotient misses a
// rounding boundary by at least that.
template <int N>
__device__ __forceinline__ void quot(const double (&a)[N], const double (&b)[N], double (&q)[N]) {
  double y[N], r[N];
  rcp(b, y);
#pragma unroll
  for (int i = 0; i < N; ++i) q[i] = a[i] * y[i];
#pragma unroll
  for (int it = 0; it < 2; ++it) {
#pragma unroll
    for (int i = 0; i < N; ++i) r[i] = fma(-b[i], q[i], a[i]);
#pragma unroll
    for (int i = 0; i < N; ++i) q[i] = fma(r[i], y[i], q[i]);
  }
}

// sin and cos of |x| < 2^50 (cbcm::sincos).
template <int N>
__device__ __forceinline__ void sincos(const double (&x)[N], double (&s)[N], double (&c)[N]) {
  double r[N], z[N], ps[N], pc[N];
  int q[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double t = x[i] * CBCM_K(cbcm::SC_RED, 3) + RINT_MAGIC;
    q[i] = __double2loint(t);
    const double kd = t - RINT_MAGIC;
    r[i] = fma(-kd, CBCM_K(cbcm::SC_RED, 0), x[i]);
    z[i] = kd;
  }
#pragma unroll
  for (int i = 0; i < N; ++i) r[i] = fma(-z[i], CBCM_K(cbcm::SC_RED, 1), r[i]);
#pragma unroll
  for (int i = 0; i < N; ++i) r[i] = fma(-z[i], CBCM_K(cbcm::SC_RED, 2), r[i]);
#pragma unroll
  for (int i = 0; i < N; ++i) z[i] = r[i] * r[i];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    ps[i] = fma(CBCM_K(cbcm::SIN_P, 8), z[i], CBCM_K(cbcm::SIN_P, 7));
    pc[i] = fma(CBCM_K(cbcm::COS_P, 8), z[i], CBCM_K(cbcm::COS_P, 7));
  }
#pragma unroll
  for (int k = 6; k >= 0; --k)
#pragma unroll
    for (int i = 0; i < N; ++i) {
      ps[i] = fma(ps[i], z[i], CBCM_K(cbcm::SIN_P, k));
      pc[i] = fma(pc[i], z[i], CBCM_K(cbcm::COS_P, k));
    }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double sr = fma(r[i] * z[i], ps[i], r[i]);
    const double cr = fma(z[i], pc[i], 1.0);
    const double a = (q[i] & 1) ? cr : sr, b = (q[i] & 1) ? sr : cr;
    s[i] = __hiloint2double(__double2hiint(a) ^ ((q[i] & 2) << 30), __double2loint(a));
    c[i] = __hiloint2double(__double2hiint(b) ^ (((q[i] + 1) & 2) << 30), __double2loint(b));
  }
}

// x^y = exp(y log x) (cbcm::pow_pos) for x normal and positive with
// |y log x| < 690: log, exp and the scaling by 2^n stay in the normal range.
template <int N>
__device__ __forceinline__ void pow_pos(const double (&x)[N], const double (&y)[N], double (&out)[N]) {
  double a[N], b[N], f[N], s[N], p[N], r[N];
  int e[N];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int hi = __double2hiint(x[i]), lo = __double2loint(x[i]);
    const int mh = hi & 0x000fffff;
    // m > sqrt(2): the significand above that of 2 SQRT1_2 (0x1.6a09e667f3bcdp+0)
    const bool big = mh > 0x6a09e || (mh == 0x6a09e && (unsigned)lo > 0x667f3bcdu);
    e[i] = (hi >> 20) - 1023 + (big ? 1 : 0);
    const double m = __hiloint2double(mh | (big ? 0x3fe00000 : 0x3ff00000), lo);
    a[i] = m - 1.0;
    b[i] = m + 1.0;
  }
  quot(a, b, f);
#pragma unroll
  for (int i = 0; i < N; ++i) s[i] = f[i] * f[i];
#pragma unroll
  for (int i = 0; i < N; ++i) p[i] = fma(CBCM_K(cbcm::LOG_P, 10), s[i], CBCM_K(cbcm::LOG_P, 9));
#pragma unroll
  for (int k = 8; k >= 0; --k)
#pragma unroll
    for (int i = 0; i < N; ++i) p[i] = fma(p[i], s[i], CBCM_K(cbcm::LOG_P, k));
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double f2 = f[i] + f[i];
    const double logm = fma(f2 * s[i], p[i], f2);
    const double ed = (double)e[i];
    a[i] = y[i] * fma(ed, CBCM_K(cbcm::LOG_C, 0), fma(ed, CBCM_K(cbcm::LOG_C, 1), logm));
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double t = a[i] * CBCM_K(cbcm::EXP_RED, 0) + RINT_MAGIC;
    e[i] = __double2loint(t);
    b[i] = t - RINT_MAGIC;
  }
#pragma unroll
  for (int i = 0; i < N; ++i) r[i] = fma(-b[i], CBCM_K(cbcm::EXP_RED, 1), a[i]);
#pragma unroll
  for (int i = 0; i < N; ++i) r[i] = fma(-b[i], CBCM_K(cbcm::EXP_RED, 2), r[i]);
#pragma unroll
  for (int i = 0; i < N; ++i) p[i] = fma(CBCM_K(cbcm::EXP_P, 11), r[i], CBCM_K(cbcm::EXP_P, 10));
#pragma unroll
  for (int k = 9; k >= 0; --k)
#pragma unroll
    for (int i = 0; i < N; ++i) p[i] = fma(p[i], r[i], CBCM_K(cbcm::EXP_P, k));
#pragma unroll
  for (int i = 0; i < N; ++i) p[i] = fma(p[i], r[i], 1.0);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double v = fma(p[i], r[i], 1.0);
    out[i] = __hiloint2double(__double2hiint(v) + (e[i] << 20), __double2loint(v));
  }
}

// Whether 2^lo <= |x| < 2^hi (exponent bounds; false for zero, inf, NaN).
template <int LO, int HI>
__device__ __forceinline__ bool exp_in(double x) {
  return (unsigned)((__double2hiint(x) & 0x7fffffff) - ((1023 + LO) << 20)) < (unsigned)((HI - LO) << 20);
}

}  // namespace cbcd
