// exp(x) in FP64 for the softmax weights, by Tang's table-driven method
// (P. T. P. Tang, "Table-driven implementation of the exponential function
// in IEEE floating-point arithmetic", ACM TOMS 15(2), 1989), with a table of
// 64 entries: x = (64m + j)·ln2/64 + r, |r| <= ln2/128, and
// exp(x) = 2^m · 2^(j/64) · p(r), p the degree-5 Taylor polynomial of e^r
// (truncation below 4e-17 relative). The reduction splits ln2/64 into a
// 36-bit head, whose products with |64m + j| < 2^17 are exact, and a tail.
// Results are within 3 units in the last place of the exact value (2.17
// the largest error measured over 1.1e7 arguments on [-708, 709]);
// arguments below -708 (subnormal or zero results), above 709 and NaN go
// to the math library's exp.
#pragma once

#include <cstdint>

#include "ptx.cuh"

namespace ef {

constexpr double kLn2Over64Hi = 0x1.62e42fefa0000p-7;
constexpr double kLn2Over64Lo = 0x1.cf79abc9e3b3ap-46;
constexpr double k64OverLn2 = 92.33248261689366;

// The table 2^(j/64), j < 64, for the calling thread's device (computed in
// long double on the host and rounded once); kernels copy it to shared
// memory.
const double* exp_table(int device);

__device__ __forceinline__ double exp_tang(double x, const double* __restrict__ table) {
  if (!(x >= -708.0 && x <= 709.0)) return exp(x);
  // k = x·64/ln2 rounded to the nearest integer by adding 1.5·2^52 (one
  // rounding of the exact product), read from the sum's low word.
  const double t = fma(x, k64OverLn2, 6755399441055744.0);
  const double kf = t - 6755399441055744.0;
  const int k = __double2loint(t);
  double r = fma(-kf, kLn2Over64Hi, x);
  r = fma(-kf, kLn2Over64Lo, r);
  double p = fma(r, 1.0 / 120.0, 1.0 / 24.0);
  p = fma(p, r, 1.0 / 6.0);
  p = fma(p, r, 0.5);
  p = fma(p, r, 1.0);
  p = fma(p, r, 1.0);
  return p * table[k & 63] * ptx::pow2(k >> 6);
}

// 2^shift · exp(x) for softmax weights (x <= 0 and 0 <= shift <= 64, or
// shift = 0), without the range test: x is clamped to [-708, 709] (by its high
// word: to within 2^-11 of the bound), so the result stays normal. Below -708
// the result (under 2^(shift-1021)) stands in for a weight that no digit of
// W = 2^shift · w keeps and that a sum of weights holding the row's heaviest one
// (2^shift) absorbs. A NaN argument gives a finite value, for callers that
// select another one for it. The powers of two go into the exponent field.
__device__ __forceinline__ double exp_weight(double x, const double* __restrict__ table, int shift) {
  const int h = min(__double2hiint(x), 0x40862800);                       // 709
  x = __hiloint2double((int)min((unsigned)h, 0xc0862000u), __double2loint(x));  // -708
  const double magic = 6755399441055744.0 + 64.0 * shift;
  const double t = fma(x, k64OverLn2, magic);
  const double kf = t - magic;
  const int k = __double2loint(t);  // k + 64·shift
  double r = fma(-kf, kLn2Over64Hi, x);
  r = fma(-kf, kLn2Over64Lo, r);
  double p = fma(r, 1.0 / 120.0, 1.0 / 24.0);
  p = fma(p, r, 1.0 / 6.0);
  p = fma(p, r, 0.5);
  p = fma(p, r, 1.0);
  p = fma(p, r, 1.0);
  p *= table[k & 63];
  return __hiloint2double(__double2hiint(p) + ((k & ~63) << 14), __double2loint(p));
}

// exp(s·y) for a scale y given as an unevaluated sum yhi + ylo (so that y = 1/h
// divides without a rounding), by the same method with 256 table entries of two
// doubles each, 2^(j/256) = hi + lo: s·y = (256m + j)·ln2/256 + r,
// |r| <= ln2/512, and exp = 2^m·(hi + (hi·q + lo)), q = e^r - 1 to degree 4 with
// the cubic coefficient raised by 0.9·(ln2/512)^2/120, which takes up all but
// 6e-18 of the degree-5 term. The head of ln2/256 has 28 bits, so its products
// with |256m + j| < 2^20 are exact, and r = fma(s, yhi, -k·head) loses nothing to
// the cancellation. Within 0.51 units in the last place of exp of the exact s·y
// (the library's exp of the rounded s·y: 1 unit and half a unit of s·y).
// |s·y| <= 700 (the caller clamps s). `table` is the caller's copy of
// exp_scaled_table, entry j at table[j·stride]; yk is y·256/ln2.
constexpr int kExpScaledEntries = 256;
constexpr double kLn2Over256Hi = 0x1.62e42ff000000p-9;
constexpr double kLn2Over256Lo = -0x1.718432a1b0e26p-43;
constexpr double k256OverLn2 = 369.32993046757464;

const double2* exp_scaled_table(int device);

__device__ __forceinline__ double exp_scaled(double s, double yk, double yhi, double ylo,
                                             const double2* __restrict__ table, int stride) {
  constexpr double a = 0x1.62e42fefa39efp-10;  // ln2/512
  const double t = fma(s, yk, 6755399441055744.0);
  const double kf = t - 6755399441055744.0;
  const int k = __double2loint(t);
  double r = fma(s, yhi, -__dmul_rn(kf, kLn2Over256Hi));
  r = fma(s, ylo, r);
  r = fma(kf, -kLn2Over256Lo, r);
  double q = fma(r, 1.0 / 24.0, 1.0 / 6.0 + 0.9 * a * a / 120.0);
  q = fma(q, r, 0.5);
  q = fma(q, r * r, r);
  const double2 e = table[(k & (kExpScaledEntries - 1)) * stride];
  const double w = e.x + fma(e.x, q, e.y);
  return __hiloint2double(__double2hiint(w) + ((k & ~(kExpScaledEntries - 1)) << 12), __double2loint(w));
}

}  // namespace ef
