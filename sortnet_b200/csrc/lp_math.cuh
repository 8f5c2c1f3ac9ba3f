// Powers by the special-function unit, shared by the dense (norm_dist_lp.cu) and the sparse (lp_skip.cu) l-p kernels.
#pragma once
#include "common.cuh"

namespace snb {

// Special-function-unit exp2 / log2.  The .ftz forms skip the denormal fix-up code: a denormal
// argument of log2 reads as 0 (its power is 0 to fp32 anyway) and results below 2^-126 flush to 0.
__device__ __forceinline__ float ex2_approx(float z) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(z));
    return r;
}
__device__ __forceinline__ float lg2_approx(float a) {
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
    return r;
}

// log2(a) by a degree-8 series in d = a - 1 (exact subtraction), for |d| <= 0.125.  The hardware
// approximation has an absolute error of 2^-22, i.e. no relative accuracy near a = 1; the series
// keeps the relative error of log2 at fp32 level there, so that a^e for large e is as accurate as
// the fp32 rounding of a allows.
__device__ __forceinline__ float log2_series(float a) {
    const float d = a - 1.0f;
    float s = fmaf(d, -0.125f, 1.0f / 7.0f);
    s = fmaf(d, s, -1.0f / 6.0f);
    s = fmaf(d, s, 0.2f);
    s = fmaf(d, s, -0.25f);
    s = fmaf(d, s, 1.0f / 3.0f);
    s = fmaf(d, s, -0.5f);
    s = fmaf(d, s, 1.0f);
    return d * 1.4426950408889634f * s;
}
__device__ __forceinline__ bool near_one(float a) { return fabsf(a - 1.0f) <= 0.125f; }

// a^e for a >= 0, accurate per value (used once per output and in the backward).
__device__ __forceinline__ float pow_pos(float a, float e) {
    return ex2_approx(e * (near_one(a) ? log2_series(a) : lg2_approx(a)));
}
// a^e where only the *sum* of many such terms matters (forward): the absolute error of the
// hardware log2 perturbs the sum by ~1.7e-7 * e relative, and the e-th root taken afterwards
// divides that by e.
__device__ __forceinline__ float pow_pos_sum(float a, float e) { return ex2_approx(e * lg2_approx(a)); }

}  // namespace snb
