// FP64 1 / d and d^-1/2 for the kernels that the FP64 pipe bounds: the hardware's
// estimate (rcp.approx.ftz.f64, rsqrt.approx.ftz.f64: a relative error e0 of about
// 2^-20) and one step of Householder's method of third order (A. S. Householder, The
// Numerical Treatment of a Single Nonlinear Equation, 1970; E. Halley's for the
// reciprocal).
//
//   e = 1 - d r,    1 / d  = r / (1 - e)      = r (1 + e + e^2 + O(e^3)),
//   e = 1 - d r^2,  d^-1/2 = r (1 - e)^(-1/2) = r (1 + e / 2 + 3 e^2 / 8 + O(e^3)),
//
// with e^3 below 2^-57.  The reciprocal's residual is one fused multiply-add, exact to
// 2^-53 e, so the last multiply-add's rounding remains: half a unit in the last place
// and 2^-4 for the rest.  The other residual takes d r rounded, 2^-53 of 1, half of it
// in the result: one unit altogether.  Zero, subnormal, infinite, NaN, (for the
// estimate's flush to zero) the ends of the exponent range, and for d^-1/2 negative
// arguments take the library's function.
#pragma once

namespace corr {

__device__ __forceinline__ bool fp64_approx_range(double d) {
  const int ex = (__double2hiint(d) >> 20) & 0x7FF;
  return ex >= 2 && ex <= 2044;
}

__device__ __forceinline__ double recip64(double d) {
  if (!fp64_approx_range(d)) return 1.0 / d;
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double e = fma(-d, r, 1.0);
  return fma(r, fma(e, e, e), r);
}

__device__ __forceinline__ double rsqrt64(double d) {
  if (__double2hiint(d) < 0 || !fp64_approx_range(d)) return rsqrt(d);
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(d));
  const double e = fma(-d * r, r, 1.0);
  return fma(r * e, fma(0.375, e, 0.5), r);
}

}  // namespace corr
