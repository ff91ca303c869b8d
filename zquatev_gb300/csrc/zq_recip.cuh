// Reciprocal and reciprocal square root of doubles for kernels that the FP64 pipe bounds.
//
// Method: functional iteration (M. J. Flynn, "On division by functional iteration",
// IEEE Trans. Computers C-19 (1970) 702-706): with an approximation y of 1 / d and
// e = 1 - d y, 1 / d = y (1 + e + e^2 + ...), cut after e^2; and likewise 1 / sqrt(q) =
// y (1 - h)^(-1/2) = y (1 + h / 2 + 3 h^2 / 8 + ...), h = 1 - q y^2. y comes from the
// documented approximation instructions (at least 20 correct bits), so the terms left
// out are below 2^-60 and 2^-58.
#pragma once

#include <cuda_runtime.h>

namespace zq {

// 1 / d in four instructions. Relative error at most (1 + 2^-6) 2^-53, that of a
// correctly rounded quotient but for the terms left out, where d and 1 / d are normal
// numbers (a subnormal d counts as zero); 0, Inf and NaN give NaN.
__device__ __forceinline__ double recip(double d) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

// 1 / sqrt(q) in six instructions, q in [2^-900, 2^900]: relative error at most
// (1 + 2^-6) 1.5 2^-53, below the one unit in the last place of rsqrt() (the rounding of
// q y gives the half).
__device__ __forceinline__ double recip_sqrt(double q) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(q));
  const double h = fma(-(q * y), y, 1.0);
  return fma(y * h, fma(0.375, h, 0.5), y);
}

}  // namespace zq
