// FP64 reciprocal and quotient in few FP64 operations (each warp-level FP64
// instruction holds an SM sub-partition's FP64 unit for 64 cycles).
#pragma once
#include <cuda_runtime.h>

namespace elfel {

__device__ __forceinline__ int exponent_of(double x) { return (int)((__double_as_longlong(x) >> 52) & 0x7ff); }

// Two steps of Newton's iteration y <- y + y (1 - x y) from the hardware's 20-bit
// estimate of 1 / x (x normal, its exponent and that of 1 / x not extreme).
__device__ __forceinline__ double newton_rcp(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// 1 / x in four FP64 operations after the estimate, at most one unit in the last place from
// the rounded 1 / x; x of extreme exponent (zero, infinity, NaN) goes through the division.
__device__ __forceinline__ double fast_rcp(double x) {
  const int e = exponent_of(x);
  if (e < 60 || e > 1980) return 1.0 / x;
  return newton_rcp(x);
}

// newton_rcp(x) here, ahead of where it is used (the compiler moves it there otherwise,
// behind the barrier of a sum: FP64 CG on 129,000 unknowns 1 % longer).
__device__ __forceinline__ double rcp_ahead(double x) {
  double y = newton_rcp(x);
  asm volatile("" : "+d"(y));
  return y;
}

// a / x from y = newton_rcp(x), formed ahead of a: a y, within two units in the last place; where
// the exponent of x is extreme the division (y is not used).
__device__ __forceinline__ double times_rcp(double a, double x, double y) {
  const int e = exponent_of(x);
  if (e < 60 || e > 1980) return a / x;
  return a * y;
}

// a / x: a y, y = newton_rcp(x), corrected by its remainder a - x q (Markstein 1990); at most one
// unit in the last place from the rounded quotient.  Where an exponent is extreme (of a, x or the
// quotient: a y overflows, the remainder underflows, zeros, infinities, NaN) the division.
__device__ __forceinline__ double fast_div(double a, double x) {
  const int e = exponent_of(x), f = exponent_of(a), d = f - e;
  if (e < 60 || e > 1980 || f < 60 || f == 0x7ff || d < -960 || d > 1020) return a / x;
  const double y = newton_rcp(x), q = a * y;
  return fma(fma(-x, q, a), y, q);
}

}  // namespace elfel
