// l-p distance for large p over the terms that can matter (lp_skip.cu).
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace snb {

struct LpProblem {
    const float* x;     // [B, CI]
    const float* w;     // [W_CO, W_CI]
    const int* ci;      // [S, CI] kept columns per sub-batch, or null
    const int* co;      // [S, CO] kept rows of W per sub-batch, or null
    int B, CO, CI, W_CO, W_CI;
    float p;
};

// Scratch of the sparse form in bytes; 0 where the dense kernels are the better ones (sizes and p only).
size_t lp_skip_forward_bytes(const LpProblem& q);
size_t lp_skip_backward_bytes(const LpProblem& q);
// The forward without what only makes it faster, the pruned evaluation of the maxima.
size_t lp_skip_forward_least_bytes(const LpProblem& q);
// ws: that many bytes, 16-byte aligned; the forward takes the least or more.
cudaError_t lp_skip_forward(const LpProblem& q, float* y, void* ws, size_t ws_bytes, cudaStream_t st);
// gw may be null; otherwise it has been zero-filled.
cudaError_t lp_skip_backward(const LpProblem& q, const float* g, const float* y, float* gx, float* gw, void* ws, cudaStream_t st);

}  // namespace snb
