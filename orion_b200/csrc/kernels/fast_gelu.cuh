// Gaussian CDF for GELU without the library erff: Abramowitz & Stegun 7.1.26,
//   erf(x) = 1 - (a1 t + a2 t^2 + a3 t^3 + a4 t^4 + a5 t^5) exp(-x^2),  t = 1 / (1 + 0.3275911 x),  x >= 0,
// absolute error below 1.5e-7 (plus ~1e-6 relative from the fast exponential): two orders of magnitude inside the float32
// tolerance of the model outputs (1e-4) and far below bfloat16 resolution.  `e` = exp(-a^2 / 2) is passed in because the
// backward pass needs the same exponential for the density.
// About 14 instructions, two of them on the special-function unit (16 results per clock and SM): at 8 elements per clock and SM
// the arithmetic of 32 Mi elements takes as long as their bfloat16 traffic.  The correctly rounded reciprocal that stood here
// (its error, half an ulp, is as far below the formula's own 1.5e-7 as the approximate one's single ulp) took a dozen
// instructions more and bound the row kernels: bias + GELU of 8192 x 4096 50 -> 33 us (4.1 TB/s), error unchanged (4.2e-7).
#pragma once
#include <cuda_runtime.h>

namespace ob200 {

__device__ __forceinline__ float rcp_approx(float x) {   // 1 / x, one ulp; x >= 1 here
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float gauss_exp(float a) {    // exp(-a^2 / 2)
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a * a * -0.72134752044448170f));
    return y;
}
__device__ __forceinline__ float gauss_cdf_with_exp(float a, float e) {
    const float t = rcp_approx(fmaf(0.3275911f * 0.70710678118654752f, fabsf(a), 1.0f));
    float poly = fmaf(0.5f * 1.061405429f, t, 0.5f * -1.453152027f);
    poly = fmaf(poly, t, 0.5f * 1.421413741f);
    poly = fmaf(poly, t, 0.5f * -0.284496736f);
    poly = fmaf(poly, t, 0.5f * 0.254829592f);
    const float half_tail = poly * t * e;                 // 0.5 * (1 - erf(|a| / sqrt 2))
    return a >= 0.f ? 1.0f - half_tail : half_tail;
}
__device__ __forceinline__ float gauss_cdf(float a) { return gauss_cdf_with_exp(a, gauss_exp(a)); }

}  // namespace ob200
