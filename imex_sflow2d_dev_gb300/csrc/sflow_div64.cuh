// sflow_div64.cuh -- FP64 quotients by one divisor, and FP64 comparisons on
// the integer pipe, for the plain FP64 form.
//
// GB300 executes FP64 instructions (compares included) at 1/64 of the FP32
// rate: 2 lanes per clock and SM, while the integer pipes of the SM start
// 64 lanes per clock.  The FP64 kernels are bound by the number of FP64
// instructions, so
//  * several quotients by one divisor share its reciprocal: a quotient then
//    takes 4 FP64 operations instead of the ~9 of a division;
//  * sign tests, comparisons and maxima work on the bit patterns.
// Every function returns the bits of the plain FP64 expression it stands
// for (tests/test_div64.py compiles this header on the host and compares).
#pragma once
#include <math.h>
#include <stdint.h>

#if defined(__CUDACC__)
#define D64_FN static __device__ __forceinline__
#define D64_FMA(a, b, c) __fma_rn((a), (b), (c))
#define D64_MUL(a, b) __dmul_rn((a), (b))
#define D64_DIV(a, b) __ddiv_rn((a), (b))
#define D64_COLD static __device__ __noinline__
#else
#include <string.h>
#define D64_FN static inline
#define D64_FMA(a, b, c) fma((a), (b), (c))
#define D64_MUL(a, b) ((a) * (b))
#define D64_DIV(a, b) ((a) / (b))
#define D64_COLD static inline
#endif

namespace sflow {

#if defined(__CUDACC__)
D64_FN long long d64_bits(double x) { return __double_as_longlong(x); }
D64_FN double d64_from(long long b) { return __longlong_as_double(b); }
D64_FN int d64_hi(double x) { return __double2hiint(x); }
#else
D64_FN long long d64_bits(double x) { long long b; memcpy(&b, &x, sizeof b); return b; }
D64_FN double d64_from(long long b) { double x; memcpy(&x, &b, sizeof x); return x; }
D64_FN int d64_hi(double x) { return (int)(d64_bits(x) >> 32); }
#endif

constexpr long long kD64Abs = 0x7fffffffffffffffll;
constexpr long long kD64Inf = 0x7ff0000000000000ll;

// x > t for a positive constant t (false for NaN)
D64_FN bool d64_gt_pos(double x, double t) { return d64_bits(x) > d64_bits(t) && d64_bits(x) <= kD64Inf; }
// x > 0, x < 0, x == 0 (false for NaN)
D64_FN bool d64_pos(double x) { return d64_bits(x) > 0 && d64_bits(x) <= kD64Inf; }
D64_FN bool d64_zero(double x) { return (d64_bits(x) & kD64Abs) == 0; }
D64_FN bool d64_neg(double x) {
  const long long m = d64_bits(x) & kD64Abs;
  return d64_bits(x) < 0 && m != 0 && m <= kD64Inf;
}
// a < b of any doubles (false when either is NaN, -0 equals +0)
D64_FN bool d64_lt(double a, double b) {
  const long long ma = d64_bits(a) & kD64Abs, mb = d64_bits(b) & kD64Abs;
  const long long ka = d64_bits(a) < 0 ? -ma : ma, kb = d64_bits(b) < 0 ? -mb : mb;
  return ka < kb && ma <= kD64Inf && mb <= kD64Inf;
}
// (a > b ? a : b) of |.| patterns: b when either is NaN, as the comparison gives
D64_FN long long d64_absmax(long long a, long long b) { return (a > b && a <= kD64Inf) ? a : b; }

// A divisor d with its reciprocal in two parts: zh = 1/d rounded to nearest,
// zl the rest to ~2^-52 of it.
struct Div64 {
  double d, zh, zl;
};
// both magnitudes within 2^-423 .. 2^423: no partial result below over- or
// underflows
D64_FN bool d64_mid(double x) {
  const unsigned e = ((unsigned)d64_hi(x) >> 20) & 0x7ffu;
  return e - 600u <= 846u;
}
D64_FN Div64 div64(double d) {
  Div64 r;
  r.d = d;
  r.zh = D64_DIV(1.0, d);
  r.zl = D64_MUL(D64_FMA(-d, r.zh, 1.0), r.zh);
  return r;
}
// a / d rounded to nearest.  q = a zh + a zl is within half a unit in the
// last place and 2^-50 of one of a/d, so its remainder is exact and the last
// step gives the correctly rounded quotient (P. Markstein, Computation of
// elementary functions on the IBM RISC System/6000 processor, IBM J. Res.
// Dev. 34(1), 1990: zh is 1/d correctly rounded, q a faithful quotient).
// Operands outside the middle of the range take the plain division.
D64_FN double quot64(double a, const Div64& v) {
  if (!(d64_mid(a) && d64_mid(v.d))) {
    if (d64_zero(a) && d64_mid(v.d)) return D64_MUL(a, v.zh);   // a zero of the right sign
    return D64_DIV(a, v.d);
  }
  const double q = D64_FMA(a, v.zh, D64_MUL(a, v.zl));
  return D64_FMA(D64_FMA(-v.d, q, a), v.zh, q);
}

}  // namespace sflow
