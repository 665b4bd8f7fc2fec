// pmhd/fastmath.hpp -- reciprocal, reciprocal square root and square root of the
// performance builds (never the parity builds): binary32 by the hardware's
// approximate instructions (<= 1 ulp), binary64 by their seeds and one iteration.
// Host code (no device) uses the IEEE operations.
#ifndef PMHD_FASTMATH_HPP
#define PMHD_FASTMATH_HPP

#include <cmath>

#if defined(__CUDACC__)
#define PMHD_HD __host__ __device__ __forceinline__
#else
#define PMHD_HD inline
#endif

namespace pmhd {

#if defined(__CUDA_ARCH__)
__device__ __forceinline__ float fast_rcp(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float fast_rsqrt(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float fast_sqrt(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
#else
inline float fast_rcp(float x) { return 1.0f / x; }
inline float fast_rsqrt(float x) { return 1.0f / std::sqrt(x); }
inline float fast_sqrt(float x) { return std::sqrt(x); }
#endif
// Binary64 forms: the hardware's approximate seed (rcp / rsqrt.approx.ftz.f64,
// about 20 bits) and one third-order step of Householder's iteration (IEEE
// division and square root take a data-dependent slow path as well and about three
// times the instructions; the binary64 stage kernel is bound by instruction issue
// and dependent binary64 latency, not by a pipe).  With e = 1 - x r:  r + r (e +
// e^2); with h = x y, e = 1 - h y:  y + y t and h + h t, t = e/2 + 3 e^2/8, the root
// followed by one Newton correction by its residual.
//   Errors: the step leaves the cube of the seed's error, 2^-57 or less, before the
// last rounding: fast_rcp and the roots are within 0.6 ulp.  fast_rsqrt also carries
// half the rounding of h (2^-54): within 1.1 ulp.
//   Arguments: of either sign for fast_rcp, positive for the others, with argument
// and result of normal size (2^-1022 < |x| < 2^1022; the roots keep their bound from
// 2^-960 on, where the residual is representable).  fast_sqrt also returns 0 and +inf
// unchanged and NaN for negative arguments.  A subnormal argument gives NaN: its
// seed is infinite.  The callers' floors (1e-12) and degeneracy guards keep every
// argument far inside; the Euler forms, which have no floors, meet subnormal values
// only in states of that size, since a difference of normal values is zero or at
// least 2^-106 of them.
#if defined(__CUDA_ARCH__)
__device__ __forceinline__ double fast_rcp(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-x, r, 1.0);
  return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ double rsqrt_seed(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  return y;
}
__device__ __forceinline__ double fast_rsqrt(double x) {
  const double y = rsqrt_seed(x);
  const double e = fma(-(x * y), y, 1.0);
  return fma(y, e * fma(e, 0.375, 0.5), y);
}
// Root of a positive normal number (no zero, infinity or NaN to look after).
__device__ __forceinline__ double fast_sqrt_pos(double x) {
  const double y = rsqrt_seed(x);
  const double h = x * y;
  const double e = fma(-h, y, 1.0);
  const double s = fma(h, e * fma(e, 0.375, 0.5), h);
  return fma(fma(-s, s, x), 0.5 * y, s);
}
__device__ __forceinline__ double fast_sqrt(double x) {
  const double s = fast_sqrt_pos(x);
  return x + x == x ? x : s;
}
#else
inline double fast_rcp(double x) { return 1.0 / x; }
inline double fast_rsqrt(double x) { return 1.0 / std::sqrt(x); }
inline double fast_sqrt(double x) { return std::sqrt(x); }
inline double fast_sqrt_pos(double x) { return std::sqrt(x); }
#endif
PMHD_HD float fast_sqrt_pos(float x) { return fast_sqrt(x); }

}  // namespace pmhd

#endif  // PMHD_FASTMATH_HPP
