// GELU of the FNO layers, x Phi(x), and its BF16 rounding.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace huv_dev {

__device__ __forceinline__ float gelu_erf(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }

// (bf16(gelu_erf(a)), bf16(gelu_erf(b))), exactly, at less than half of two
// erff: an approximation g of x Phi(x) whose distance to gelu_erf is below
// e = 2^-20 |x|, then both ends of [g - e, g + e] rounded; where they agree,
// every value between them rounds the same way, and where they do not (about
// one pair in 500; also for NaN, infinities and zeros) gelu_erf decides.
// g = max(x, 0) - |x| erfc(|x| / sqrt 2) / 2 with Abramowitz and Stegun's
// rational approximation 7.1.26 of erfc (absolute error below 1.5e-7, so that
// |x| times half of it stays below e / 10).
__device__ __forceinline__ void gelu_bounds(float x, float& lo, float& hi) {
  const float ax = fabsf(x);
  float t, ex;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(t) : "f"(fmaf(ax, 0.3275911f * 0.70710678f, 1.f)));
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(ex) : "f"(x * x * -0.72134752f));
  float p = fmaf(t, 0.5f * 1.061405429f, 0.5f * -1.453152027f);
  p = fmaf(t, p, 0.5f * 1.421413741f);
  p = fmaf(t, p, 0.5f * -0.284496736f);
  p = fmaf(t, p, 0.5f * 0.254829592f);
  const float g = fmaf(-ax, p * t * ex, fmaxf(x, 0.f));
  const float e = fmaf(ax, 9.5367431640625e-7f, 1e-30f);
  lo = g - e;
  hi = g + e;
}
__device__ __forceinline__ __nv_bfloat162 gelu_bf16x2(float a, float b) {
  float la, ha, lb, hb;
  gelu_bounds(a, la, ha);
  gelu_bounds(b, lb, hb);
  const __nv_bfloat162 lo = __floats2bfloat162_rn(la, lb), hi = __floats2bfloat162_rn(ha, hb);
  if (__hbeq2(lo, hi)) return lo;
  return __floats2bfloat162_rn(gelu_erf(a), gelu_erf(b));
}

}  // namespace huv_dev
