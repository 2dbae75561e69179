// Gaussian CDF for GELU without the library erff: Abramowitz & Stegun 7.1.26,
//   erf(x) = 1 - (a1 t + a2 t^2 + a3 t^3 + a4 t^4 + a5 t^5) exp(-x^2),  t = 1 / (1 + 0.3275911 x),  x >= 0,
// absolute error below 1.5e-7 (plus ~1e-6 relative from the fast exponential): two orders of magnitude inside the float32
// tolerance of the model outputs (1e-4) and far below bfloat16 resolution.  `e` = exp(-a^2 / 2) is passed in because the
// backward pass needs the same exponential for the density.
// About 18 instructions, two of them on the special-function unit (16 results per clock and SM): the arithmetic of 32 Mi elements
// takes about as long as their bfloat16 traffic.  The library's correctly rounded reciprocal took a dozen instructions more and
// bound the row kernels: bias + GELU of 8192 x 4096 50 -> 40 us, 3072 x 3072
// 16.6 -> 12.5 us.  The Newton step below gives the same bits for every float from
// 1 to 64, so the results did not change.
#pragma once
#include <cuda_runtime.h>

namespace ob200 {

// 1 / x for x >= 1: the special-function unit's approximation and one Newton step.  For x = infinity the step would be
// infinity * 0; the approximation, zero, stands.
__device__ __forceinline__ float reciprocal_from_1(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    const float e = fmaf(-x, r, 1.0f);
    return x < 1e30f ? fmaf(r, e, r) : r;
}
__device__ __forceinline__ float gauss_exp(float a) { return __expf(-0.5f * a * a); }
__device__ __forceinline__ float gauss_cdf_with_exp(float a, float e) {
    const float ax = fabsf(a) * 0.70710678118654752f;
    const float t = reciprocal_from_1(fmaf(0.3275911f, ax, 1.0f));
    float poly = fmaf(0.5f * 1.061405429f, t, 0.5f * -1.453152027f);   // halved: 0.5 * (1 - erf(|a| / sqrt 2))
    poly = fmaf(poly, t, 0.5f * 1.421413741f);
    poly = fmaf(poly, t, 0.5f * -0.284496736f);
    poly = fmaf(poly, t, 0.5f * 0.254829592f);
    const float half_tail = poly * t * e;
    return a >= 0.f ? 1.0f - half_tail : half_tail;
}
__device__ __forceinline__ float gauss_cdf(float a) { return gauss_cdf_with_exp(a, gauss_exp(a)); }

}  // namespace ob200
