// mlc_scalar.cuh -- scalar functions of the kernels whose results rest on bit
// patterns or single instructions: the WAF limiter, the thresholds of the step
// end and the saturation mixing ratio (recip_d and div_d are in
// mlc_device.cuh).  In a header of their own so that a test can run them on
// arrays.
#pragma once
#include "mlc_device.cuh"

namespace mlc {

// The bit pattern of x through an opaque move, for the sign, region, range and
// upwind tests that run on the integer pipe: a plain reinterpretation lets the
// compiler turn an integer test of the pattern back into an FP64 comparison
// (an instruction of the 1/64-rate FP64 pipe on GB300).
__device__ __forceinline__ long long bits_of(double x) {
  long long b;
  asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
  return b;
}

// ---- the WAF limiter ----------------------------------------------------------
// WAF flux  hvel*((1+phi)*a + (1-phi)*c)  with  phi = is + zamu*b - is*b  and
// the limiter  b = max(0, min(2, max(r, min(2r, 1))))  of  r = num/den
// (local_flow_param, Main/mod_moloch.F90:1571-1590; the flux lines
// :877-883, :986-993, :1017-1024).  In every use den = c - a, so
//   (1+phi)*a + (1-phi)*c = (a + c) - phi*den,
//   phi*den = is*den + (zamu - is)*B,   B = b*den.
// With d = |den| > 0 and q = num*sign(den) (so r = q/d), multiplying the
// limiter by d > 0 gives
//   B = sign(den) * max(0, min(2d, max(q, min(2q, d)))),
// whose candidates 0, q, 2q, d, 2d are exact: B is one of 0, 2*num, den, num,
// 2*den exactly, the value of b*den in each region of r, ties included.  No
// division.

// FP32: |B| = max(0, min(|2 num|, |den|), min(|num|, |2 den|)), the two minima
// with num*den's sign (superbee in its other form, the same candidates in
// every region), B with den's: four instructions of the half-rate pipe instead
// of seven (moist 512x512x41, a step: vertical passes 0.227 -> 0.212 ms,
// increments 0.109 -> 0.094, horizontal 0.351 -> 0.338).  The reference's
// guard of tiny denominators is left out - it changes B only where
// |den| < 1e-15, by less than 2|den|, far below FP32 rounding of the flux.
__device__ __forceinline__ float waf_b(float den, float num) {
  float t1, t2, bd;
  asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(t1) : "f"(num + num), "f"(den));
  asm("min.xorsign.abs.f32 %0, %1, %2;" : "=f"(t2) : "f"(num), "f"(den + den));
  asm("max.f32 %0, %1, %2, 0f00000000;" : "=f"(bd) : "f"(t1), "f"(t2));
  return __uint_as_float(__float_as_uint(bd) ^ (__float_as_uint(den) & 0x80000000u));
}

// FP64: B = sel, or 2*sel where dbl is set.  The regions of r (0, 1/2, 1, 2)
// are tested in turn, which usually stops early, and on the integer pipe: on
// GB300 each FP64 min, max or compare is an instruction of the 1/64-rate FP64
// pipe.  Non-negative doubles order like their bit patterns read as integers,
// and for a normal d (d >= minden here) d/2 and 2d are d's pattern -/+ 2^52; q
// by a sign-bit XOR.  A NaN num fails every comparison and takes the last
// region; the reference's guard of denominators below minden (:1571-1590;
// minnum is the 4-byte real holding it) is kept exactly.
//
// The doubling stays out of the FP64 pipe too: in the regions where B is 2*num
// or 2*den the flux takes 2*zmih (an exponent's increment) as the factor of num
// or den instead, zmih*(2*sel) = (2*zmih)*sel exactly, so only the differences
// and one fused multiply-add are FP64 instructions.
__device__ __forceinline__ double waf_sel(double den, double num, bool &dbl) {
  const long long bden = bits_of(den), bnum = bits_of(num);
  const long long mag = 0x7fffffffffffffffLL, one_exp = 1LL << 52;
  const long long ad = bden & mag;            // |den|
  const long long bq = bnum ^ (bden & ~mag);  // q, as a signed pattern
  const long long eden = __double_as_longlong(1.0e-30);
  const long long enum_ = __double_as_longlong((double)1.0e-30f);
  dbl = false;
  if (ad < eden) return (bnum & mag) < enum_ ? den : 0.0;  // r = 1 or r = 0
  if ((bnum & mag) > 0x7ff0000000000000LL) { dbl = true; return den; }
  if (bq <= 0) return 0.0;                                 // q <= 0 (and -0)
  if (bq < ad - one_exp) { dbl = true; return num; }       // q < d/2
  if (bq <= ad) return den;                                // q <= d
  if (bq < ad + one_exp) return num;                       // q < 2d
  dbl = true;
  return den;
}
// 2x (if dbl) by the exponent, on the integer pipe; zeros, subnormals,
// infinities and NaN as they are
__device__ __forceinline__ double twice(double x, bool dbl) {
  const int h = __double2hiint(x), e = h & 0x7ff00000;
  return __hiloint2double(dbl && e && e != 0x7ff00000 ? h + 0x00100000 : h, __double2loint(x));
}

// ---- the step end -------------------------------------------------------------
// q < c for a positive finite threshold c, exactly as the comparison (false
// for a NaN q).  FP64 on the bit patterns: a negative q, -0 included, has the
// sign bit set and compares below every positive pattern as a signed integer.
// FP32 compares directly.
template <class R>
__device__ __forceinline__ bool below_pos(R q, double c) {
  if constexpr (sizeof(R) == sizeof(double)) {
    const long long b = bits_of(q);
    const bool nan = (b & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
    return !nan && b < __double_as_longlong(c);
  } else {
    return q < R(c);
  }
}

// pfwsat (Share/pfwsat.inc) of FP64 fields with few FP64 instructions: the
// range tests on the bit patterns, explicit fused multiply-adds, div_d.
__device__ __forceinline__ double pfwsat_d(double t, double p) {
  double td = t - kTzero;
  const long long b = bits_of(td), mag = b & 0x7fffffffffffffffLL;
  const bool num = mag <= 0x7ff0000000000000LL;
  if (num && b < 0 && mag > __double_as_longlong(75.0)) td = -75.0;
  if (num && b > __double_as_longlong(100.0)) td = 100.0;
  double es;
  if (num && b >= 0) {
    es = __fma_rn(td, 0.209339997e-13, -0.373208410e-10);
    es = __fma_rn(td, es, 0.892344772e-08);
    es = __fma_rn(td, es, 0.196237241e-05);
    es = __fma_rn(td, es, 0.305903558e-03);
    es = __fma_rn(td, es, 0.264461437e-01);
    es = __fma_rn(td, es, 0.143064234e+01);
    es = __fma_rn(td, es, 0.444007856e+02);
    es = __fma_rn(td, es, 0.611213476e+03);
  } else {
    es = __fma_rn(td, 0.262655803e-12, 0.149436277e-09);
    es = __fma_rn(td, es, 0.387940929e-07);
    es = __fma_rn(td, es, 0.602780717e-05);
    es = __fma_rn(td, es, 0.614396778e-03);
    es = __fma_rn(td, es, 0.420547422e-01);
    es = __fma_rn(td, es, 0.188369801e+01);
    es = __fma_rn(td, es, 0.503109514e+02);
    es = __fma_rn(td, es, 0.611123516e+03);
  }
  // (pressures and saturation pressures are positive, so they order like
  // their patterns; a NaN stays)
  const double cap = __dmul_rn(0.15, p);
  const long long be = bits_of(es);
  if (be <= 0x7ff0000000000000LL && bits_of(cap) < be) es = cap;
  return __dmul_rn(kEp2, div_d(es, p - es));
}

// x differs from c in its bits (-0 from 0 too), on the integer pipe
__device__ __forceinline__ bool bits_differ(double x, double c) { return bits_of(x) != __double_as_longlong(c); }
__device__ __forceinline__ bool bits_differ(float x, float c) { return __float_as_uint(x) != __float_as_uint(c); }

}  // namespace mlc
