// Reciprocal and reciprocal square root of a double for the FP64 sweeps: a
// hardware seed (~20 bits) and one third-order Householder step.  GB300's FP64
// unit takes a warp instruction every 16 cycles per SM, so their instruction
// count (3 and 5) is what matters.  The remainder of the step is far below a
// rounding, so 1/x is within 0.6 ulp and 1/sqrt(x) within 1.1 for arguments and
// results that are normal numbers (|x| up to 2^1021 for 1/x: the seed flushes
// subnormals), both without a bias.
#pragma once
#include <cuda_runtime.h>

namespace sph {
namespace dev {

// 1/sqrt(x), x normal and positive: y the hardware seed, e = 1 - x y^2,
// y (1 + e/2 + 3 e^2/8) (Householder's method of third order; the
// remainder is below 2^-56).
__device__ __forceinline__ double rsqrt64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = __fma_rn(-__dmul_rn(x, y), y, 1.0);
  return __fma_rn(__dmul_rn(e, y), __fma_rn(e, 0.375, 0.5), y);
}
// 1/x, x normal: r (1 + e + e^2) with e = 1 - x r (third order).
__device__ __forceinline__ double rcp64(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = __fma_rn(-x, r, 1.0);
  return __fma_rn(r, __fma_rn(e, e, e), r);
}

}  // namespace dev
}  // namespace sph
