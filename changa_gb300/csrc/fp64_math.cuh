/* FP64 helpers of the plain FP64 form. */
#pragma once

namespace chg {
namespace {

/* 1/sqrt(x) for positive normal x, from the hardware's approximation (some
 * 20 bits): with e = 1 - x y^2, 1/sqrt(x) = y (1 - e)^(-1/2), whose series
 * y (1 + e/2 + 3 e^2 / 8) is cut at 5 e^3 / 16, below 2^-58; the roundings of
 * x y, of e and of the last sum make at most 2^-52 of the root.  Five FP64
 * operations; NaN at infinity, for a zero and for a subnormal. */
__device__ __forceinline__ double rsqrt_normal(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(fma(e, 0.375, 0.5), e * y, y);
}

/* Whether x is not a number, on the integer pipe. */
__device__ __forceinline__ bool is_nan(double x) {
  return (__double_as_longlong(x) & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL;
}

/* The larger of a, not negative, and b, on the integer pipe; a NaN b of
 * positive sign is taken for the larger, so callers keep NaNs out. */
__device__ __forceinline__ double max_nonneg(double a, double b) {
  return __longlong_as_double(max(__double_as_longlong(a), __double_as_longlong(b)));
}

}  // namespace
}  // namespace chg
