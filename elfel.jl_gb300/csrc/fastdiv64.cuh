// FP64 reciprocal and quotient in few FP64 operations (each warp-level FP64
// instruction holds an SM sub-partition's FP64 unit for 64 cycles).
#pragma once
#include <cuda_runtime.h>

namespace elfel {

// 1 / x by Newton's iteration from the hardware's 20-bit estimate (four FP64
// operations; the compiler's division takes about twelve, 64 cycles each).
// x of extreme exponent goes through the division.
__device__ __forceinline__ double fast_rcp(double x) {
  const int e = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
  if (e < 60 || e > 1980) return 1.0 / x;
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}

// a / x, y = fast_rcp(x): the quotient corrected by its remainder.
__device__ __forceinline__ double fast_div(double a, double x, double y) {
  const double q = a * y;
  return fma(fma(-x, q, a), y, q);
}

}  // namespace elfel
