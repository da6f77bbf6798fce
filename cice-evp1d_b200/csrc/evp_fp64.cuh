// evp_fp64.cuh -- correctly rounded FP64 division and square root as
// straight-line code.
//
// The compiler's own FP64 `/` and sqrt are correctly rounded too, but each
// carries a branch to a slow path, so a point's several divisions and square
// roots run one after another however independent they are: four divisions
// took 501 cycles and four square roots 372 in one warp, 512 and 402 with two
// warps a scheduler; as below 103 and 119, 151 and 176.  These functions give
// the same bits for operands in a middle range of exponents, which the caller
// tests (fp64_mid) once for several operations, taking the plain operators
// where it fails.
//
// Methods, from the literature on division and square root with a fused
// multiply-add:
//  - P. W. Markstein, "Computation of elementary functions on the IBM RISC
//    System/6000 processor", IBM J. Res. Dev. 34 (1990);
//  - M. Cornea, J. Harrison, P. T. P. Tang, "Scientific Computing on
//    Itanium-based Systems", Intel Press (2002).
// Reciprocal: the seed (PTX rcp.approx.ftz.f64, measured error below 2^-19.9)
// takes one cubic step, which leaves it within 0.52 ulp, and one Newton step
// with the exact residual, which rounds it correctly for every b whose
// significand is not all ones (Markstein).
// Quotient: a*y1, corrected once by its residual, is within one ulp; the
// residual of that is exact, and adding residual times the correctly rounded
// reciprocal rounds a/b correctly (Markstein).  With an all-ones b the
// reciprocal may come out as the power of two below; working the sum through,
// the quotient is then still right unless a is a power of two itself.  So the
// caller also makes sure that either b's significand is not all ones or a's
// is not 1.
// Square root: the seed y of 1/sqrt(x) (PTX rsqrt.approx.ftz.f64, |y*y*x - 1|
// measured below 2^-19) takes a cubic step, relative error then below
// 1.6*2^-53; g = x*y is corrected by its residual, g + (y/2)*(x - g*g).
// Before its one rounding that sum is within 9.6*2^-53 ulp of sqrt(x), so it
// can only be rounded to the wrong side where sqrt(x) lies that close to the
// middle of two doubles; with x = X*2^e, X in [2^104, 2^106) a multiple of
// 2^52 (2^53 above 2^105), and the midpoint n + 1/2, that means
// |n*n + n + 1/4 - X| <= 19.3: a few dozen significands, each of which the
// tests try on the device.
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#include <cuda_runtime.h>

namespace evp {

__host__ __device__ __forceinline__ uint32_t fp64_hi(double x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2hiint(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return (uint32_t)(b >> 32);
#endif
}

__host__ __device__ __forceinline__ uint32_t fp64_lo(double x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__double2loint(x);
#else
  uint64_t b;
  std::memcpy(&b, &x, 8);
  return (uint32_t)b;
#endif
}

// x > 0 with an exponent of -500..499: no step below can overflow, underflow
// or meet a zero, an infinity or a NaN.
__host__ __device__ __forceinline__ bool fp64_mid(double x) {
  return fp64_hi(x) - (523u << 20) < (1000u << 20);
}

// The same for |x|.
__host__ __device__ __forceinline__ bool fp64_mid_abs(double x) {
  return (fp64_hi(x) & 0x7fffffffu) - (523u << 20) < (1000u << 20);
}

// A dividend for divisors whose significand may be all ones: in range and no
// power of two, or +0 (every step then gives +0).
__host__ __device__ __forceinline__ bool fp64_dividend(double a) {
  const uint32_t h = fp64_hi(a), l = fp64_lo(a);
  return (fp64_mid(a) && ((h & 0xfffffu) | l) != 0u) || (h | l) == 0u;
}

// A divisor that any dividend of middle range may have.
__host__ __device__ __forceinline__ bool fp64_divisor(double b) {
  return fp64_mid(b) && fp64_lo(b) != 0xffffffffu;
}

// 1/b within 0.52 ulp (y1) and correctly rounded (y2).
struct Recip {
  double y1, y2;
};

__host__ __device__ __forceinline__ Recip fp64_recip(double b) {
  Recip r;
#if defined(__CUDA_ARCH__)
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  const double e = __fma_rn(-b, y, 1.0);
  r.y1 = __fma_rn(y, __fma_rn(e, e, e), y);
  r.y2 = __fma_rn(r.y1, __fma_rn(-b, r.y1, 1.0), r.y1);
#else
  r.y1 = r.y2 = 1.0 / b;
#endif
  return r;
}

// a/b, correctly rounded, from b's reciprocal.
__host__ __device__ __forceinline__ double fp64_quot(double a, double b, const Recip &r) {
#if defined(__CUDA_ARCH__)
  double q = __dmul_rn(a, r.y1);
  q = __fma_rn(__fma_rn(-b, q, a), r.y1, q);
  return __fma_rn(__fma_rn(-b, q, a), r.y2, q);
#else
  (void)r;
  return a / b;
#endif
}

// The operand of fp64_sqrt: in range, or +0.
__host__ __device__ __forceinline__ bool fp64_radicand(double x) {
  return fp64_mid(x) | ((fp64_hi(x) | fp64_lo(x)) == 0u);
}

// sqrt(x), correctly rounded.
__host__ __device__ __forceinline__ double fp64_sqrt(double x) {
#if defined(__CUDA_ARCH__)
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  // from a seed of 0, x = 0 gives 0 (ice beside the coast, where no corner
  // moves, has Delta = 0)
  y = (fp64_hi(x) | fp64_lo(x)) == 0u ? 0.0 : y;
  const double r = __fma_rn(-__dmul_rn(x, y), y, 1.0);
  y = __fma_rn(__dmul_rn(y, r), __fma_rn(r, 0.375, 0.5), y);
  const double g = __dmul_rn(x, y);
  return __fma_rn(__dmul_rn(0.5, y), __fma_rn(-g, g, x), g);
#else
  return std::sqrt(x);
#endif
}

}  // namespace evp
