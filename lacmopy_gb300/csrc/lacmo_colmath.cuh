// Device math shared by the collision kernels: correctly rounded radius and
// kernel bin, integer-unit conversions, lower bounds of draws.  Included only
// by files compiled with -fmad=false.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

#include "lacmo_crmath.h"
#include "lacmo_internal.cuh"
#include "lacmo_physics.cuh"
#include "lacmo_thin.h"

namespace lacmo {

// x^(1/3 rounded to double) correctly rounded, fast path.  With c = double(1/3)
// = 1/3 - d, d = 2^-54/3, the value is cbrt(x) * exp(-d ln x).  y = cbrt(x)
// (faithful) is refined by one Newton step whose residual x - y^3 is formed in
// double-double, and exp(-d ln x) = 1 - d L + (d L)^2/2 to far below 2^-100.
// So z = y + t with t computed to ~2^-100 |y|.  The rounded sum y + t is the
// correctly-rounded result unless y + t lies within 2^-85 |y| of a rounding
// midpoint; then (or for non-normal x) the full routine decides.  The margin
// is wider than the full routine's own uncertainty, so both always agree.
__device__ __forceinline__ double cr_pow13_dd(double x) {
  if (!(x >= 0x1p-1000 && x <= 0x1p1000)) return lacmo_cr_pow(x, LC_ONE_THIRD);
  const double y = cbrt(x);
  const lacmo_dd y2 = lacmo_two_prod(y, y);
  const lacmo_dd y3 = lacmo_dd_mul_d(y2, y);
  const double r = (x - y3.hi) - y3.lo;           // x - y3.hi is exact (Sterbenz)
  const double corr = r / (3.0 * y2.hi);
  const double dL = 0x1.5555555555555p-56 * log(x);  // d * ln x, d = 2^-54 / 3
  const double t = corr - y * dL + y * (0.5 * dL * dL);
  const double s = y + t;
  const double e = (y - s) + t;                   // y + t = s + e exactly
  const uint64_t b = lacmo_as_u64(s);
  const int64_t ex = (int64_t)((b >> 52) & 0x7ff);
  double half_ulp = lacmo_as_f64((uint64_t)(ex - 53) << 52);
  if (e < 0.0 && (b & 0x000fffffffffffffULL) == 0) half_ulp *= 0.5;
  if (fabs(fabs(e) - half_ulp) <= 0x1p-85 * s) return lacmo_cr_pow(x, LC_ONE_THIRD);
  return s;
}

// The same value with most of the FP64 work moved to FP32 (GB300's FP64 pipe
// is narrow, and the collision events run on single lanes).  For x in
// [2^-40, 2^40] (every radius from 1 nm to 1 cm in micrometres):
//  - y: the FP32 cube root (a few ulp) refined by two Newton steps
//    y += (x - y^3) / (3 y^2), the residual in FP64 and the quotient in FP32:
//    the error goes 2^-21 -> 2^-43 -> within about an ulp (FP64 rounding of
//    the residual);
//  - t = r / (3 y^2) - y d ln x with r = x - y^3 in double-double as above,
//    both terms in FP32: |r / (3 y^2)| < 2^-50 y and |y d ln x| < 2^-46 y,
//    each within 2^-22 relative, their sum within 2^-24 of the larger, and the
//    neglected (d ln x)^2 / 2 below 2^-92: t is within 2^-67 y of its value;
//  - a flushed FP32 residual (|r| < 2^-126) changes t by less than
//    2^-126 / (3 x) <= 2^-86 y.
// s = y + t is then the correctly-rounded result unless it lies within
// 2^-62 s of a rounding midpoint (about one call in 500), where cr_pow13_dd
// decides.
__device__ __forceinline__ double cr_pow13(double x) {
  if (!(x >= 0x1p-40 && x <= 0x1p40)) return cr_pow13_dd(x);
  const float xf = d2f_int(x);
  double y = f2d_int(f_cbrt(xf));
#pragma unroll
  for (int it = 0; it < 2; ++it) {
    const float yf = d2f_int(y);
    const double r0 = x - (y * y) * y;
    y = y + f2d_int(d2f_int(r0) * f_rcp(3.0f * yf * yf));
  }
  const lacmo_dd y2 = lacmo_two_prod(y, y);
  const lacmo_dd y3 = lacmo_dd_mul_d(y2, y);
  const double r = (x - y3.hi) - y3.lo;
  const float yf = d2f_int(y);
  const float tf = d2f_int(r) * f_rcp(3.0f * yf * yf) -
                   yf * (0x1.555556p-56f * (f_lg2(xf) * 0.693147181f));
  const double t = f2d_int(tf);
  const double s = y + t;
  const double e = (y - s) + t;
  const uint64_t b = lacmo_as_u64(s);
  const int64_t ex = (int64_t)((b >> 52) & 0x7ff);
  double half_ulp = lacmo_as_f64((uint64_t)(ex - 53) << 52);
  if (e < 0.0 && (b & 0x000fffffffffffffULL) == 0) half_ulp *= 0.5;
  if (fabs(fabs(e) - half_ulp) <= 0x1p-62 * s) return cr_pow13_dd(x);
  return s;
}

__device__ __forceinline__ double col_radius(double m, double rho) {
  return cr_pow13(LC_FOUR_PI_OVER_THREE_INV * m / rho);
}
// collision/all_or_nothing.py:35-67; float -> int as x86-64 compiled code
// does it (NaN / out of range -> INT64_MIN -> bin 0).  The bin of the
// correctly-rounded log: with the hardware log the index value is within
// 1e-12 of it, so unless it lies within 1e-9 of an integer the truncation is
// the same; near a bin edge the correctly-rounded log decides.
__device__ __forceinline__ int32_t col_bin(double R, double lo, double bl, int64_t nb) {
  double v = (log(R) - lo) / bl + 0.5;
  const double fl = floor(v);
  if (!(v - fl > 1e-9 && (fl + 1.0) - v > 1e-9 && fabs(v) < 1e15))
    v = (lacmo_cr_log(R) - lo) / bl + 0.5;
  int64_t ind = (v > -9.2233720368547758e18 && v < 9.2233720368547758e18) ? (int64_t)v : INT64_MIN;
  if (ind < 0) ind = 0;
  else if (ind > nb - 1) ind = nb - 1;
  return (int32_t)ind;
}
// The same bin from an FP32 bin position first: lo_f, inv_bl_f are lo and 1/bl
// rounded to FP32 and margin bounds the error of the FP32 position (it is
// derived for radii within 1e-6; R is rounded to within 2^-24 here).  A
// position farther than margin from every bin edge gives the bin of the exact
// position; closer ones take col_bin.
__device__ __forceinline__ int32_t col_bin_f(double R, double lo, double bl, int64_t nb,
                                             float lo_f, float inv_bl_f, float margin) {
  const float Rf = d2f_int(R);
  const float v = (f_lg2(Rf) * 0.693147181f - lo_f) * inv_bl_f + 0.5f;
  const float fl = floorf(v);
  if (v - fl > margin && (fl + 1.0f) - v > margin && v > -1e6f && v < 1e6f && Rf > 1e-30f &&
      Rf < 1e30f) {
    int32_t kb = __float2int_rz(fl);
    return kb < 0 ? 0 : (kb > nb - 1 ? (int32_t)nb - 1 : kb);
  }
  return col_bin(R, lo, bl, nb);
}
__device__ __forceinline__ int64_t pair_rank(int64_t i, int64_t j, int64_t n) {
  return i * n - i * (i + 1) / 2 + (j - i - 1);
}

// integer-unit conversions (GB300 runs FP64 conversions on its narrow FP64
// pipe): round to nearest even, and truncation toward zero for r >= 0
static __device__ __noinline__ float d2f_rn_slow(double x) { return (float)x; }
__device__ __forceinline__ float d2f_rn(double x) {
  const uint64_t b = (uint64_t)__double_as_longlong(x);
  const uint32_t e = (uint32_t)(b >> 52) & 0x7ffu;
  if (e - 897u > 253u) return d2f_rn_slow(x);
  const uint32_t sign = (uint32_t)(b >> 32) & 0x80000000u;
  const uint64_t m = b & 0x000fffffffffffffull;
  const uint32_t fm = (uint32_t)(m >> 29), rem = (uint32_t)m & 0x1fffffffu;
  uint32_t fb = sign | ((e - 896u) << 23) | fm;
  fb += (rem > 0x10000000u) || (rem == 0x10000000u && (fm & 1u));
  return __int_as_float((int)fb);
}
// round to nearest even with zero/subnormal results flushed to zero and
// overflow (and NaN) to infinity: integer instructions only (screen inputs,
// where a flushed value makes the pair undecided or stays inside the bounds)
__device__ __forceinline__ float d2f_flush(double x) {
  const uint64_t b = (uint64_t)__double_as_longlong(x);
  const uint32_t e = (uint32_t)(b >> 52) & 0x7ffu;
  const uint32_t sign = (uint32_t)(b >> 32) & 0x80000000u;
  if (e < 897u) return __int_as_float((int)sign);
  if (e > 1150u) return __int_as_float((int)(sign | 0x7f800000u));
  const uint64_t m = b & 0x000fffffffffffffull;
  const uint32_t fm = (uint32_t)(m >> 29), rem = (uint32_t)m & 0x1fffffffu;
  uint32_t fb = sign | ((e - 896u) << 23) | fm;
  fb += (rem > 0x10000000u) || (rem == 0x10000000u && (fm & 1u));
  return __int_as_float((int)fb);
}
__device__ __forceinline__ float d2f_down_pos(double r) {  // r in [0, 1)
  const uint64_t b = (uint64_t)__double_as_longlong(r);
  const uint32_t e = (uint32_t)(b >> 52) & 0x7ffu;
  if (e < 897u) return 0.0f;
  return __int_as_float((int)(((e - 896u) << 23) | (uint32_t)((b >> 29) & 0x7fffffu)));
}

// the lower bound of a draw the first screens take: from the top word of a Philox
// draw (23 bits), or of an injected one
__device__ __forceinline__ float low_of_word(uint32_t x) {
  return __uint_as_float(0x3f800000u | (x >> 9)) - 1.0f;
}
__device__ __forceinline__ float low_of_double(double r) {
  const uint64_t b = (uint64_t)__double_as_longlong(r);
  return b < 0x3ff0000000000000ull && b >= 0x3e70000000000000ull ? d2f_down_pos(r) : 0.0f;
}

// Bound on the error of the FP32 bin position v = (__logf(Rf) - lo_f) *
// inv_bl_f + 0.5 against the exact (log R - lo) / bl + 0.5, doubled: Rf is
// within 1e-6 of R (relative), so log Rf within 1e-6; __logf within 2^-21.41
// absolute on [0.5, 2] and 3 ulp elsewhere (taken as 4 ulp of the largest
// |log R| a bin edge can have); lo_f and the subtraction round within one ulp
// of that value together; inv_bl_f, the product and the + 0.5 each within
// 2^-24 of v <= nb + 1.  Bins closer than this to an edge are taken from the
// exact FP64 path.
static inline float fp32_bin_margin(double lo, double bl, int64_t nb) {
  if (!(bl > 0.0) || nb <= 0) return 0.5f;
  const double lmax = fmax(fabs(lo), fabs(lo + (double)(nb + 1) * bl)) + 1.0;
  const double ulp = ldexp(1.0, (int)floor(log2(lmax)) - 23);
  const double log_err = fmax(ldexp(1.0, -21) , 4.0 * ulp);
  const double v_err = (1e-6 + log_err + ulp) / bl + 3.0 * (double)(nb + 1) * ldexp(1.0, -24);
  const double m = 2.0 * v_err;
  return (float)(m < 0.5 ? m : 0.5);
}

}  // namespace lacmo
