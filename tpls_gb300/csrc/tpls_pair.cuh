// tpls_pair.cuh -- FP64 values as FP32 pairs by integer operations.
//
// On GB300 FP64 arithmetic and FP64<->FP32 conversions share a pipe 64x
// slower than FP32.  The FP32 parts of the FP32-mixed form therefore read
// FP64 values as a pair (hi = the value truncated to 24 significant bits,
// lo = the FP32 rounding of the remainder, hi + lo within 2^-47 of the
// value) built with integer instructions only, and form differences of
// nearby values as (hi_a - hi_b) + (lo_a - lo_b), which carries FP32
// precision relative to the difference itself rather than to the values.
#pragma once
#include "tpls_common.cuh"

namespace tpls {

struct F2 {
  float h, l;
};

__device__ __forceinline__ F2 split_bits(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned int top = (unsigned int)(b >> 32), sgn = top & 0x80000000u;
  const int e = (int)((top >> 20) & 0x7ffu);  // biased FP64 exponent
  const unsigned int m23 = (unsigned int)(b >> 29) & 0x7fffffu, rem = (unsigned int)b & 0x1fffffffu;
  F2 p;
  if (e >= 897 && e <= 1150) {  // 2^-126 <= |x| < 2^128: hi is an FP32 normal
    p.h = __uint_as_float(sgn | ((unsigned int)(e - 896) << 23) | m23);
    // lo = rem * 2^(e - 1075); that power of two is an FP32 normal for e >= 949
    const float sc = __uint_as_float((unsigned int)max(e - 948, 0) << 23);
    const float lo = (e >= 949) ? __uint2float_rn(rem) * sc : 0.0f;
    p.l = __uint_as_float(__float_as_uint(lo) | sgn);
  } else if (e == 2047) {  // inf / NaN stay inf / NaN
    p.h = __uint_as_float(sgn | 0x7f800000u | ((m23 | rem) ? 0x400000u : 0u));
    p.l = 0.0f;
  } else {  // |x| < 2^-126 (taken as zero) or beyond the FP32 range (inf)
    p.h = __uint_as_float(sgn | (e > 1150 ? 0x7f800000u : 0u));
    p.l = 0.0f;
  }
  return p;
}

// exact FP32 -> FP64 widening by integer operations (FP32 subnormals,
// never produced by these stencils' magnitudes, become signed zero)
__device__ __forceinline__ double widen_bits(float v) {
  const unsigned int b = __float_as_uint(v), e = (b >> 23) & 0xffu;
  const unsigned long long s = (unsigned long long)(b & 0x80000000u) << 32;
  const unsigned long long m = (unsigned long long)(b & 0x7fffffu) << 29;
  unsigned long long r;
  if (e == 0) r = s;
  else if (e == 255) r = s | 0x7ff0000000000000ull | m;
  else r = s | ((unsigned long long)(e + 896) << 52) | m;
  return __longlong_as_double((long long)r);
}

__device__ __forceinline__ float dif(F2 a, F2 b) { return (a.h - b.h) + (a.l - b.l); }

// the pair's value rounded to FP32 (hi alone is truncated, biased toward
// zero by up to an ulp: sums and products take the rounded value)
__device__ __forceinline__ float val(F2 a) { return a.h + a.l; }
__device__ __forceinline__ float round_bits(double x) { return val(split_bits(x)); }

// (float)x, round to nearest even, by operations on the two 32-bit words (a
// conversion instruction would hold the FP64 pipe); values outside FP32's
// normal range convert by the instruction
__device__ __forceinline__ float float_bits(double x) {
  const unsigned int hi = (unsigned int)__double2hiint(x), lo = (unsigned int)__double2loint(x);
  const unsigned int a = hi & 0x7fffffffu;
  if (a - 0x38100000u >= 0x47e00000u - 0x38100000u) return (a | lo) == 0 ? __uint_as_float(hi) : (float)x;
  const unsigned int m = __funnelshift_l(lo, a - 0x38000000u, 3), rem = lo & 0x1fffffffu;
  const unsigned int up = (rem > 0x10000000u || (rem == 0x10000000u && (m & 1u))) ? 1u : 0u;
  return __uint_as_float((m + up) | (hi & 0x80000000u));
}

// 1/d to about 2^-44 for 2^-100 < |d| < 2^100: FP32 reciprocal of the leading
// part and one Newton step in FP32 on the pair, joined by one FP64 addition.
__device__ __forceinline__ double rcp_seed(double d) {
  const F2 p = split_bits(d);
  const float r = __fdividef(1.0f, p.h);
  const float e = fmaf(-p.l, r, fmaf(-p.h, r, 1.0f));
  return widen_bits(r) + widen_bits(r * e);
}
// |d| within 2^-100 .. 2^100 (also excludes 0, infinities and NaN)
__device__ __forceinline__ bool rcp_range(double d) {
  const unsigned int a = (unsigned int)__double2hiint(d) & 0x7fffffffu;
  return a - (923u << 20) < (200u << 20);
}
// The quotient the hardware sequence would form, out of line: the callers'
// common path is four FP64 operations instead of about nine.
static __device__ __noinline__ double div_slow(double n, double d) { return n / d; }
// n/d to within one ulp: quotient from the seed, its remainder by an FMA
// (exact up to one rounding) and one correction.
__device__ __forceinline__ double div_fast(double n, double d) {
  if (!rcp_range(d)) return div_slow(n, d);
  const double r = rcp_seed(d);
  const double q = n * r;
  return fma(fma(-d, q, n), r, q);
}

// The same for any numerator: an infinite quotient is not corrected (its
// remainder would be NaN).
__device__ __forceinline__ double div_inf(double n, double d) {
  if (!rcp_range(d)) return div_slow(n, d);
  const double r = rcp_seed(d), q = n * r, v = fma(fma(-d, q, n), r, q);
  return (__double2hiint(q) & 0x7ff00000) == 0x7ff00000 ? q : v;
}

// sqrt(a), correctly rounded, with one FP64 operation: an FP32 pair (sh, sl)
// of the root to about 2^-43, joined to a double s0 by integer addition; the
// exact residual a - s0^2 by one FMA; the correction c = residual / (2 s0) in
// FP32, in units of s0's last place, rounded to an integer and added to the
// bits.  c is known to 2^-21.4 of itself (rsqrtf's two ulps and four FP32
// roundings), so where it lies that close to half-way between two integers,
// or a sum leaves the binade, the library's sqrt decides (about 1 in 3000).
// (a in 2^-60 .. 2^60; everything else goes there too.)
static __device__ __noinline__ double sqrt_slow(double a) { return sqrt(a); }
__device__ __forceinline__ double add_ulps(double x, int n) {
  unsigned lo, hi;
  asm("add.cc.u32 %0, %2, %4;\n\taddc.u32 %1, %3, %5;"
      : "=r"(lo), "=r"(hi)
      : "r"(__double2loint(x)), "r"(__double2hiint(x)), "r"(n), "r"(n >> 31));
  return __hiloint2double((int)hi, (int)lo);
}
__device__ __forceinline__ double sqrt_rn(double a) {
  if ((unsigned)__double2hiint(a) - (963u << 20) >= (120u << 20)) return sqrt_slow(a);
  const F2 p = split_bits(a);
  const float r = rsqrtf(p.h), hr = 0.5f * r;
  const float sh = p.h * r;
  const float sl = (fmaf(-sh, sh, p.h) + p.l) * hr;
  const unsigned eb = __float_as_uint(sh) >> 23;
  const float scale = __uint_as_float((306u - eb) << 23);  // 2^52 / 2^exponent(sh)
  const double s = widen_bits(sh);
  const double s0 = add_ulps(s, __float2int_rn(sl * scale));
  const float cu = float_bits(fma(-s0, s0, a)) * hr * scale;
  const float n = (cu + 12582912.0f) - 12582912.0f;  // nearest integer for |cu| < 2^22
  const double r0 = add_ulps(s0, (int)n);
  const int es = __double2hiint(s);
  const bool sure = fabsf(cu - n) <= 0.5f - fmaf(fabsf(cu), 9.5367431640625e-7f, 1.52587890625e-5f) &&
                    fabsf(cu) < 65536.0f && (((es ^ __double2hiint(s0)) | (es ^ __double2hiint(r0))) >> 20) == 0;
  return sure ? r0 : sqrt_slow(a);
}

// order of two pairs of the same normalisation (both from split_bits, or
// both from an error-free sum): by hi, then by lo
__device__ __forceinline__ F2 pmin(F2 a, F2 b) { return (b.h < a.h || (b.h == a.h && b.l < a.l)) ? b : a; }
__device__ __forceinline__ F2 pmax(F2 a, F2 b) { return (b.h > a.h || (b.h == a.h && b.l > a.l)) ? b : a; }

// FP64 min and max by integer operations.  The key maps the bit pattern of
// a double to a signed integer with the same order (negative values have
// their magnitude bits flipped), so for non-NaN a, b: a < b iff
// dkey(a) < dkey(b), with -0 just below +0.  That differs from fmin/fmax
// only in which zero a (+0, -0) tie returns; every use here squares the
// result or subtracts it from a value and squares that, where the sign of
// a zero does not survive.  The key and the sign tests work on the two
// 32-bit words of the double (no 64-bit integer shift).
__device__ __forceinline__ long long dkey(double a) {
  const int hi = __double2hiint(a), s = hi >> 31;
  return __double_as_longlong(__hiloint2double(hi ^ (s & 0x7fffffff), __double2loint(a) ^ s));
}
__device__ __forceinline__ double dmin_bits(double a, double b) { return (dkey(b) < dkey(a)) ? b : a; }
__device__ __forceinline__ double dmax_bits(double a, double b) { return (dkey(a) < dkey(b)) ? b : a; }
// max(a, 0) for a not NaN: +0 for a <= 0 (the sign bit decides)
__device__ __forceinline__ double dpos_bits(double a) { return (__double2hiint(a) < 0) ? 0.0 : a; }

}  // namespace tpls
