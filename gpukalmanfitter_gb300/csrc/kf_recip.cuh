// kf_recip.cuh — FP64 reciprocal and reciprocal square root of the fit kernels.
//
// The hardware's 20-bit estimate and one third-order step (Halley's family):
// three and four FP64 instructions.  The truncation, e^3 < 2^-57, lies below the
// rounding of the result, and in the root below that of a y as well: relative
// error below 2^-52 and 2^-51 (measured 1.0 and 1.24 times 2^-53).
//
// For normal arguments whose result is normal.  Denormal arguments count as
// zeros; a zero or an infinity gives an infinity or NaN, which no caller
// distinguishes from the exact result: a plane along the track is missed, a
// residual with an infinite covariance makes the track's chi2 NaN, as does a
// direction along the line's axis.
#pragma once

namespace kfd {

// with e = 1 - a y: 1/a = y (1 + e + e^2 + ...)
__device__ __forceinline__ double rcpFast(double a) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double e = fma(-a, y, 1.);
  return fma(fma(e, e, e), y, y);
}
// with e = 1 - a y^2: 1/sqrt(a) = y (1 + e/2 + 3/8 e^2 + ...)
__device__ __forceinline__ double rsqrtFast(double a) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
  const double e = fma(-a * y, y, 1.);
  return fma(fma(0.375, e, 0.5) * e, y, y);
}

} // namespace kfd
