// hb_fp64.cuh -- FP64 reciprocal and square root of the step and adjoint kernels.
#pragma once

namespace hb {

#ifdef __CUDACC__
// 1 / x for normal x: the hardware's seed r0 (relative error e; 2^-19.9 at most
// over 6e7 values of 2^-60..2^40) and the third-order iteration
// r0 (1 + e + e^2) (Householder's method for 1/r - x), remainder e^3.  Largest
// error over those values 2^-53 of the result.
__device__ __forceinline__ double rcp64(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = __fma_rn(-x, r, 1.0);
  return __fma_rn(r, __fma_rn(e, e, e), r);
}
// sqrt(x) for x >= 0: y0 ~ 1/sqrt(x) from the hardware, s0 = x y0, e = 1 - s0 y0, and
// sqrt(x) = s0 (1 - e)^(-1/2) by its binomial series to e^2 (remainder 5/16 e^3).
// Largest error over the same values 2^-52 of the result.  0 for x below the normal
// range (the seed flushes such x to 0; its root is at most 1.5e-154).
__device__ __forceinline__ double sqrt64(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double s0 = __dmul_rn(x, y);
  const double e = __fma_rn(-s0, y, 1.0);
  const double s = __fma_rn(__dmul_rn(s0, e), __fma_rn(0.375, e, 0.5), s0);
  return x >= 2.2250738585072014e-308 ? s : 0.0;
}
#endif

}  // namespace hb
