// divide.cuh -- FP64 division from a precomputed reciprocal, correctly
// rounded (the quotient the division operator gives), for divisors that
// stay fixed over many divisions: the reference SOR's diagonal (the reciprocal
// in two words, at the end of this file), the plain path's metric factors and
// implicit-damping factors.  GB300's FP64 rate is
// low; the division operator takes about twice the FP64 operations of the
// sequence below.
#pragma once
#include <cuda_runtime.h>

namespace swm {

// a / b rounded to nearest from y = 1/b rounded to nearest, by Markstein's
// theorem (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34, 1990; also Muller et
// al., Handbook of Floating-Point Arithmetic, the FMA-based division
// section): if y is within half an ulp of 1/b and q within one ulp of a/b,
// then q + (a - b q) y, each operation rounded to nearest and the remainder
// taken with one FMA, is a/b rounded to nearest.  q = a y can be up to 1.5
// ulp off, so a first correction brings it within an ulp and the second
// gives the rounded quotient.  Valid while no step underflows or overflows:
// for a and b with binary exponents in [-500, 500] (div_rn_range).
__device__ __forceinline__ double div_rn(double a, double b, double y) {
  double q = __dmul_rn(a, y);
  double r = __fma_rn(-q, b, a);
  q = __fma_rn(r, y, q);
  r = __fma_rn(-q, b, a);
  return __fma_rn(r, y, q);
}

// x is finite, nonzero, normal and of binary exponent in [-500, 500]
__device__ __forceinline__ bool div_rn_range(double x) {
  const unsigned e = ((unsigned)__double2hiint(x) >> 20) & 0x7ffu;
  return e - 523u <= 1000u;
}

// a / b given y = 1/b rounded to nearest, with b of binary exponent in
// [-500, 500]: div_rn where a is in its range, a * y for a zero numerator
// (the zero of the quotient's sign), the division operator otherwise
__device__ __forceinline__ double div_fast(double a, double b, double y) {
  if (div_rn_range(a)) return div_rn(a, b, y);
  return a == 0. ? a * y : a / b;
}

// A divisor that stays fixed, with 1/b in two words: yh = 1/b and yl = 1/b -
// yh, each rounded to nearest.  a yl, rounded, then a yh + that in one FMA
// gives a/b in two FP64 operations (N. Brisebarre, J.-M. Muller, S. K. Raina,
// "Accelerating correctly rounded floating-point division when the divisor is
// known in advance", IEEE Trans. Computers 53, 2004).  With the significands
// of a and b in [1, 2), the sum before its rounding is less than 2^-106 off
// a/b (less than 2^-107 from 1/b - yh - yl, at most 2^-107 from rounding
// a yl), and a/b is n / (B 2^53) away from a midpoint of two doubles when a >=
// b, n / (B 2^54) when a < b, for B = 2^52 b < 2^53 and an integer n >= 1.  So
// the rounding can only go wrong for a < b and n = 1, which asks for an odd B
// and A 2^54 = +-1 modulo B (A = 2^52 a): two numerators for each divisor.
// div_class tries both.  cls 0: two operations are enough for every
// numerator; 1: one of the two fails, and a Markstein correction follows (the
// quotient before it is within an ulp); 2: a divisor out of range, the
// division operator.
struct FixedDiv {
  double b, yh, yl;
  int cls, pad;
};

// the two-operation quotient
__device__ __forceinline__ double div2(double a, double yh, double yl) { return __fma_rn(a, yh, __dmul_rn(a, yl)); }

// binary exponent of b in [-400, 400]: with a numerator in div_rn_range, what
// a yl loses to underflow then stays below 2^-108 of the quotient
__device__ __forceinline__ int div_class(double b) {
  const unsigned e = ((unsigned)__double2hiint(b) >> 20) & 0x7ffu;
  if (e - 623u > 800u) return 2;
  const unsigned long long one = 1ull << 52;
  const unsigned long long B = ((unsigned long long)__double_as_longlong(b) & (one - 1)) | one;
  if (!(B & 1)) return 0;
  unsigned long long x = 1;  // 2^-54 modulo B
  for (int k = 0; k < 54; k++) x = (x & 1) ? (x + B) >> 1 : x >> 1;
  const double bs = __longlong_as_double((long long)((1023ull << 52) | (B & (one - 1))));
  const double yh = __ddiv_rn(1., bs), yl = __ddiv_rn(__fma_rn(-bs, yh, 1.), bs);
  for (int k = 0; k < 2; k++, x = B - x) {
    if (x < one) continue;
    const double a = __longlong_as_double((long long)((1023ull << 52) | (x & (one - 1))));
    if (div2(a, yh, yl) != __ddiv_rn(a, bs)) return 1;
  }
  return 0;
}

__device__ __forceinline__ FixedDiv fixed_div(double b) {
  FixedDiv d;
  d.b = b;
  d.yh = __ddiv_rn(1., b);
  d.cls = div_class(b);
  d.yl = d.cls == 2 ? 0. : __ddiv_rn(__fma_rn(-b, d.yh, 1.), b);
  d.pad = 0;
  return d;
}

// a / b, the division operator's quotient bit for bit
__device__ __forceinline__ double div_fixed(double a, const FixedDiv &d) {
  if (d.cls != 2) {
    if (div_rn_range(a)) {
      double q = div2(a, d.yh, d.yl);
      if (d.cls) q = __fma_rn(__fma_rn(-q, d.b, a), d.yh, q);
      return q;
    }
    if ((__double_as_longlong(a) << 1) == 0) return __dmul_rn(a, d.yh);  // the zero of the quotient's sign
  }
  return __ddiv_rn(a, d.b);
}

}  // namespace swm
