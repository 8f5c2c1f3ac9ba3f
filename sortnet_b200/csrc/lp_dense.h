// Operands of the dense l-p kernels (norm_dist_lp.cu: any exponent; lp_power.cu: whole ones up to 8).
#pragma once
#include <cuda_runtime.h>

namespace snb {

struct LpFwdParams {
    const float* x;
    const float* w;
    float* y;
    const float* m;  // NORMALISED: the maxima M (may be y itself when direct)
    const int* ci;
    const int* co;
    int B, CO, CI, W_CI;
    float p;
    int direct;      // 1: one CTA per output tile, finished in the kernel; 0: shared tiles, lp_finish_kernel follows
};

struct LpBwdParams {
    const float* g;
    const float* x;
    const float* w;
    const float* y;
    float* gx;
    float* gw;  // may be null: grad_x only
    const int* ci;
    const int* co;
    int B, CO, CI, W_CI;
    float pm1;  // p - 1
};

enum { MODE_VEC = 0, MODE_SCALAR = 1, MODE_GATHER = 2 };   // how W is copied: 16 bytes, 4 bytes, through the lists

// sums -> distances: y = M S^(1/p), or max(S, FLT_MIN)^(1/p) without maxima (norm_dist_lp.cu)
cudaError_t lp_finish(float* y, const float* m, long long n, float p, cudaStream_t st);

// Whole p in 1 .. 8 (lp_power.cu); gw of the backward may be null and is zero-filled otherwise.
cudaError_t lp_power_forward(const LpFwdParams& p, cudaStream_t st);
cudaError_t lp_power_backward(const LpBwdParams& p, cudaStream_t st);

}  // namespace snb
