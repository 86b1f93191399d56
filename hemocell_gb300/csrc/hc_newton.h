// Reciprocal and reciprocal square root in FP64 from a coarse seed.
//
// The FP64 pipe (two lanes an SM and cycle on this GPU) bounds the plain form's
// kernels, and a division there is about ten of its instructions.  One step of
// Householder's third-order iteration takes a seed of relative error e0 to an
// error of e0^3, so a seed of about 20 bits (PTX rcp.approx.ftz.f64 and
// rsqrt.approx.ftz.f64) reaches full precision in three instructions for 1/x and
// seven for 1/sqrt(x) together with sqrt(x):
//   1/x:       e = 1 - x y,      y (1 + e + e^2)
//   1/sqrt(x): t = x y, e = 1 - t y,  p = 1/2 + 3/8 e,  y + (y e) p,  and
//              sqrt(x) = t + (t e) p
// (Householder, The Numerical Treatment of a Single Nonlinear Equation, 1970).
// For a seed within 2^-19 the relative error stays below 2^-52: 2^-53 of the last
// rounding, at most 2^-54 of t's, and e0^3 or 5/16 (2 e0)^3 of the iteration.  A
// CPU test checks that over random arguments and seeds, a GPU test with the
// hardware's seeds over all binades.  Host and device compile the same steps.
#pragma once
#include <math.h>
#include <stdint.h>

#ifdef __CUDACC__
#define HC_NEWTON_HD __host__ __device__ __forceinline__
#else
#define HC_NEWTON_HD inline
#endif

namespace hcnewton {

HC_NEWTON_HD double recip_from(double x, double y) {
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

HC_NEWTON_HD void rsqrt_from(double x, double y, double& inv, double& root) {
  const double t = x * y;
  const double e = fma(-t, y, 1.0);
  const double p = fma(0.375, e, 0.5);
  inv = fma(y * e, p, y);
  root = fma(t * e, p, t);
}

#ifdef __CUDACC__
// 1/x for a normal x (zero and infinity give NaN)
__device__ __forceinline__ double recip(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return recip_from(x, y);
}
__device__ __forceinline__ float recip(float x) { return 1.0f / x; }

// 1/sqrt(d) and sqrt(d); both 0 for a zero or subnormal d
__device__ __forceinline__ void inv_length(double d, double& inv, double& len) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  rsqrt_from(d, y, inv, len);
  if ((uint32_t)__double2hiint(d) < 0x00100000u) inv = len = 0.0;
}
__device__ __forceinline__ void inv_length(float d, float& inv, float& len) {
  inv = d == 0.f ? 0.f : rsqrtf(d);
  len = d * inv;
}
#endif

}  // namespace hcnewton
