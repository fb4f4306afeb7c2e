// sflow_div64.cuh -- FP64 division, square root and comparisons on the
// integer pipes, for the plain FP64 form.
//
// GB300 executes FP64 instructions (compares included) at 1/64 of the FP32
// rate: an FP64 instruction of a warp holds the SM's FP64 pipe for 16
// cycles, in which the SM issues up to 64 others.  A division is about 9 of
// them and a square root more, and they made up most of the FP64 kernels.
// Here both are computed on integers: a float estimate of the reciprocal
// (of the reciprocal root), two Newton steps in 64-bit fixed point to within
// 2^-61, the product with the dividend, and an exact integer test of the
// remainder against the midpoint, which gives the correctly rounded result
// -- the bits of the FP64 operation (tests/test_div64.py compiles this
// header on the host and compares; tests/test_gpu_parity.py holds the
// kernels' bits).  About 60 instructions a quotient, 25 for a further one by
// the same divisor.  Operands outside the middle of the range, infinities
// and NaN take the FP64 operation itself.
// Measured with the power on the integer pipes (sflow_pow.h), before -> after:
// 512^2 current with settling, 8 steps, 23.9 -> 14.1 ms; 200^2 dam break to
// 10 s 115.0 -> 48.6 ms; 360 x 180 eroding flood, 32 steps, 42.9 -> 24.3 ms.
// Newton's iteration for reciprocals in fixed point with a remainder
// correction: M. J. Flynn, On division by functional iteration, IEEE Trans.
// Comput. C-19(8), 1970.
#pragma once
#include <math.h>
#include <stdint.h>

#if defined(__CUDACC__)
#define D64_FN static __device__ __forceinline__
#define D64_COLD static __device__ __noinline__
// called, not inlined: a kernel holds a hundred of them, and the instruction
// cache and the build are better off
#define D64_CALL static __device__ __noinline__
#else
#include <string.h>
#define D64_FN static inline
#define D64_COLD static inline
#define D64_CALL static inline
#endif

namespace sflow {

#if defined(__CUDACC__)
D64_FN long long d64_bits(double x) { return __double_as_longlong(x); }
D64_FN double d64_from(long long b) { return __longlong_as_double(b); }
D64_FN int d64_hi(double x) { return __double2hiint(x); }
D64_FN uint64_t d64_mulhi(uint64_t a, uint64_t b) { return __umul64hi(a, b); }
D64_FN uint32_t d64_mulhi32(uint32_t a, uint32_t b) { return __umulhi(a, b); }
// 1/m 2^31 and 1/sqrt(m) 2^31 of a float's bits, to about 2^-22
D64_FN uint32_t d64_rcp_seed(uint32_t fbits) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fbits)));
  return __float2uint_rz(r * 2147483648.0f);
}
D64_FN uint32_t d64_rsqrt_seed(uint32_t fbits) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fbits)));
  return __float2uint_rz(r * 2147483648.0f);
}
D64_COLD double d64_div_hw(double a, double b) { return __ddiv_rn(a, b); }
D64_COLD double d64_sqrt_hw(double x) { return __dsqrt_rn(x); }
#else
D64_FN long long d64_bits(double x) { long long b; memcpy(&b, &x, sizeof b); return b; }
D64_FN double d64_from(long long b) { double x; memcpy(&x, &b, sizeof x); return x; }
D64_FN int d64_hi(double x) { return (int)(d64_bits(x) >> 32); }
D64_FN uint64_t d64_mulhi(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a * b) >> 64); }
D64_FN uint32_t d64_mulhi32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
#ifndef D64_SEED_NOISE
#define D64_SEED_NOISE 0   // units of 2^-31 by which the host's estimates are off (a test varies it)
#endif
D64_FN float d64_flt(uint32_t b) { float f; memcpy(&f, &b, sizeof f); return f; }
D64_FN uint32_t d64_rcp_seed(uint32_t b) { return (uint32_t)((1.0f / d64_flt(b)) * 2147483648.0f + (D64_SEED_NOISE)); }
D64_FN uint32_t d64_rsqrt_seed(uint32_t b) {
  return (uint32_t)((1.0f / sqrtf(d64_flt(b))) * 2147483648.0f + (D64_SEED_NOISE));
}
D64_COLD double d64_div_hw(double a, double b) { return a / b; }
D64_COLD double d64_sqrt_hw(double x) { return sqrt(x); }
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

// magnitude within 2^-423 .. 2^423: no quotient or root of two such values
// leaves the normal range
D64_FN bool d64_mid(double x) {
  const unsigned e = ((unsigned)d64_hi(x) >> 20) & 0x7ffu;
  return e - 600u <= 846u;
}
D64_FN uint64_t d64_mant(double x) { return ((uint64_t)d64_bits(x) & 0xfffffffffffffull) | 0x10000000000000ull; }

// A divisor d and 2^63 / m of its significand m in [1, 2), to 2^-61.
struct Div64 {
  double d;
  uint64_t R;
};
D64_CALL Div64 div64(double d) {
  const uint64_t mant = d64_mant(d), M = mant << 11;
  const uint32_t seed = d64_rcp_seed(0x3f800000u | ((uint32_t)(mant >> 29) & 0x7fffffu));
  const uint32_t R0 = seed < 0x7fffffffu ? seed : 0x7fffffffu;
  // first step: 1 - m r0 at 2^-62, r0 corrected to ~2^-43
  const uint64_t t = (uint64_t)R0 * (uint32_t)(M >> 32) + d64_mulhi32(R0, (uint32_t)M);
  const int32_t e0 = (int32_t)((int64_t)(0x4000000000000000ull - t) >> 11);
  const uint64_t R1 = ((uint64_t)R0 << 32) + (uint64_t)(((int64_t)(int32_t)R0 * e0) >> 19);
  // second step
  const int32_t e1 = (int32_t)(0x4000000000000000ull - d64_mulhi(R1, M));
  const uint32_t h1 = (uint32_t)(R1 >> 32);
  Div64 v;
  v.d = d;
  v.R = R1 + (uint64_t)(((int64_t)(int32_t)(h1 < 0x7fffffffu ? h1 : 0x7fffffffu) * e1) >> 30);
  return v;
}
// a / v.d, correctly rounded
D64_CALL double quot64(double a, Div64 v) {
  const long long ba = d64_bits(a), bd = d64_bits(v.d);
  const long long sign = (ba ^ bd) & ~kD64Abs;
  if (!(d64_mid(a) && d64_mid(v.d))) {
    if ((ba & kD64Abs) == 0 && d64_mid(v.d)) return d64_from(sign);   // a zero
    return d64_div_hw(a, v.d);
  }
  const uint64_t ma = d64_mant(a), md = d64_mant(v.d);
  const uint64_t Q = d64_mulhi(ma << 11, v.R);      // a/d of the significands times 2^62, within 4
  const int lt = (Q >> 62) ? 0 : 1;
  uint64_t q = Q >> (10 - lt);
  // round up when the quotient lies above q + 1/2 (it cannot equal it): the
  // sign of 2 (a - (q + 1/2) d), whose magnitude is far below 2^63
  const int64_t rem = (int64_t)((ma << (53 + lt)) - (2 * q + 1) * md);
  q += rem > 0 ? 1 : 0;
  const int e = (int)((ba >> 52) & 0x7ff) - (int)((bd >> 52) & 0x7ff) + 1022 - lt;
  return d64_from(sign | (long long)(((uint64_t)e << 52) + q));
}
// a / b, correctly rounded
D64_CALL double ddiv64(double a, double b) { return quot64(a, div64(b)); }

// sqrt(x), correctly rounded
D64_CALL double dsqrt64(double x) {
  const long long b = d64_bits(x);
  if (b < 0 || !d64_mid(x)) return (b & kD64Abs) == 0 ? x : d64_sqrt_hw(x);
  const int e = (int)(b >> 52) - 1023, odd = e & 1;
  const uint64_t mant = d64_mant(x);
  const uint64_t M = mant << (10 + odd);            // significand m in [1, 4) times 2^62
  const uint32_t seed = d64_rsqrt_seed((odd ? 0x40000000u : 0x3f800000u) | ((uint32_t)(mant >> 29) & 0x7fffffu));
  const uint32_t Y0 = seed < 0x7fffffffu ? seed : 0x7fffffffu;
  // y0 -> y1 = y0 (1 + (1 - m y0^2)/2), ~2^-43
  const int32_t e0 = (int32_t)((int64_t)(0x1000000000000000ull - d64_mulhi(M, (uint64_t)Y0 * Y0)) >> 10);
  const uint64_t Y1 = ((uint64_t)Y0 << 32) + (uint64_t)(((int64_t)(int32_t)Y0 * e0) >> 19);
  // s1 = m y1, s = s1 (1 + (1 - s1 y1)/2), times 2^63
  const uint64_t S1 = d64_mulhi(M, Y1) << 2;
  const int32_t e1 = (int32_t)(0x4000000000000000ull - d64_mulhi(S1, Y1));
  const uint64_t S = S1 + (uint64_t)(((int64_t)(int32_t)(uint32_t)(S1 >> 33) * e1) >> 30);
  uint64_t q = S >> 11;
  // round up when x lies above (q + 1/2)^2
  const int64_t rem = (int64_t)((mant << (52 + odd)) - (q * q + q));
  q += rem > 0 ? 1 : 0;
  return d64_from((long long)(((uint64_t)((e - odd) / 2 + 1022) << 52) + q));
}

}  // namespace sflow
