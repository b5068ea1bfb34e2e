// FP64 reciprocal and reciprocal square root for normal arguments, from the hardware's approximations
// (about 20 bits) and one third-order Newton-Householder step each.  A third to a fifth of the
// operations of the IEEE division and square root.  Largest errors over 4 M arguments: reciprocal 0.507
// ulp (the division 0.500), reciprocal square root 0.985 ulp (1 / sqrt(x) 1.487).  Zero, infinite and
// subnormal arguments give no finite result.  The functions stand where the division would have made
// the result NaN or infinite too; the sound speed, where a zero has a meaning, takes it apart
// (inviscid_pv.cuh).
#pragma once

namespace cb2 {

// y (1 + e + e^2), e = 1 - x y: the error e^3 is below half an ulp.
__device__ __forceinline__ double recip(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ float recip(float x) { return 1.0f / x; }

// y (1 + e/2 + 3 e^2/8), e = 1 - x y^2.
__device__ __forceinline__ double recip_sqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
__device__ __forceinline__ float recip_sqrt(float x) { return rsqrtf(x); }

}  // namespace cb2
