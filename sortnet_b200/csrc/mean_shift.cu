// Mean-shift normalisation that follows every hidden norm-distance layer.
//
// Replaces the ~12 PyTorch element-wise / scatter launches of MeanShiftDropout.forward in
// zbh2047/SortNet core/models/bound_basic_module.py:123-157 (no native counterpart there).
//
//   stats : mean[c] = sum over rows b whose 32-row sub-batch kept channel c of x[b, slot(c)]
//                     / max(number of such rows, 1e-10)           (0 for never-kept channels)
//           running_mean = (1 - momentum) * running_mean + momentum * mean      (optional)
//   apply : y[b, j] = x[b, j] - mean[index[s_b][j]]                (index NULL = identity)
//
// The training-mode backward is the same pair applied to the incoming gradient, because the
// reference differentiates through the batch mean.  Both kernels are deterministic: sums run
// in a fixed order (rows ascending inside a sub-batch, sub-batches combined in a fixed tree).
#include "common.cuh"
#include "launch.h"

namespace snb {

// CTA = 16 channels x 16 sub-batch lanes.  Lane (cx, sg) sums channel c over the sub-batches
// sg, sg + 16, ...; the 16 partial sums are then added in index order.  The kernel is bound by the
// latency of each lane's chain (a binary search in the sorted list, then 32 rows), hence many short
// chains.
__global__ void __launch_bounds__(256) mean_shift_stats_kernel(const float* __restrict__ x,
                                                               const int* __restrict__ index, int B,
                                                               int C, int C_full, float* __restrict__ mean,
                                                               float* __restrict__ running_mean,
                                                               float momentum) {
    __shared__ float ssum[16][17];
    __shared__ float scnt[16][17];
    const int cx = threadIdx.x & 15, sg = threadIdx.x >> 4;
    const int c = blockIdx.x * 16 + cx;
    const int S = (B + SNB_SUB_BATCH - 1) / SNB_SUB_BATCH;
    float sum = 0.f, cnt = 0.f;
    if (c < C_full) {
        for (int s = sg; s < S; s += 16) {
            int slot = c;
            if (index) {
                // lower bound of c in the sorted kept-channel list of sub-batch s
                const int* idx = index + (size_t)s * C;
                int lo = 0, hi = C;
                while (lo < hi) {
                    const int mid = (lo + hi) >> 1;
                    if (idx[mid] < c) lo = mid + 1;
                    else hi = mid;
                }
                slot = (lo < C && idx[lo] == c) ? lo : -1;
            } else if (c >= C) {
                slot = -1;
            }
            if (slot < 0) continue;
            const int b0 = s * SNB_SUB_BATCH, b1 = min(B, b0 + SNB_SUB_BATCH);
            float part = 0.f;
            for (int b = b0; b < b1; b++) part += x[(size_t)b * C + slot];
            sum += part;
            cnt += (float)(b1 - b0);
        }
    }
    ssum[sg][cx] = sum;
    scnt[sg][cx] = cnt;
    __syncthreads();
    if (sg == 0 && c < C_full) {
        float t = 0.f, n = 0.f;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            t += ssum[k][cx];
            n += scnt[k][cx];
        }
        const float m = t / fmaxf(n, 1e-10f);
        mean[c] = m;
        if (running_mean) running_mean[c] = running_mean[c] * (1.0f - momentum) + momentum * m;
    }
}

__global__ void __launch_bounds__(256) mean_shift_apply_kernel(const float* __restrict__ x,
                                                               const float* __restrict__ mean,
                                                               const int* __restrict__ index, int B,
                                                               int C, float* __restrict__ y) {
    const int j = blockIdx.x * 256 + threadIdx.x;
    if (j >= C) return;
    const int s = blockIdx.y;
    const float m = mean[index ? index[(size_t)s * C + j] : j];
    const int b0 = s * SNB_SUB_BATCH, b1 = min(B, b0 + SNB_SUB_BATCH);
    for (int b = b0; b < b1; b++) y[(size_t)b * C + j] = x[(size_t)b * C + j] - m;
}

// The same over rows and positions of x [B, n, HW] (n kept channels of G groups, lists of within-group channels): a warp per channel, which
// walks the channel's HW neighbouring floats of every row that kept it twice, for the sum and for the result; the second time they come from L1
// or L2.  The slot of the channel in 32 sub-batches' lists is searched for by 32 lanes at once.  SHIFT: the mean into `out`, x minus it into y;
// otherwise the sums alone.  Bound by latency: 128 x 1024 x 4 with lists 8.4 us, against 8.2 + 3.2 for the same plane as 4096 channels and six
// launches for its lists, the average over positions, its expansion and the running mean; a forward and backward of two convolutions, which
// the host issues, 1050 -> 740 us (58 -> 39 launches).
template <bool SHIFT>
__global__ void __launch_bounds__(256) plane_shift_kernel(const float* __restrict__ x, const int* __restrict__ index, int B, int G,
                                                          int kept, int HW, int C, float* __restrict__ out,
                                                          float* __restrict__ running_mean, float momentum, float* __restrict__ y) {
    const int lane = threadIdx.x & 31, c = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (c >= C) return;
    const int S = (B + SNB_SUB_BATCH - 1) / SNB_SUB_BATCH, per = C / G, g = c / per, inside = c % per, n = G * kept;
    // Place of channel `want` in list g of sub-batch s: that of the first entry that is not smaller, if the list ascends.
    auto place = [&](int s, int g, int want) {
        const int* list = index + ((size_t)s * G + g) * kept;
        int lo = 0, hi = kept;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (list[mid] < want) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    };
    auto slot_in = [&](int s, int g, int inside) {
        if (!index) return inside;
        const int at = place(s, g, inside);
        return at < kept && index[((size_t)s * G + g) * kept + at] == inside ? g * kept + at : -1;
    };
    // body(offset of the element) for this lane's elements of slot `slot` of sub-batch s
    auto walk = [&](int s, int slot, auto&& body) {
        const int b0 = s * SNB_SUB_BATCH, items = min(SNB_SUB_BATCH, B - b0) * HW;
#pragma unroll 4
        for (int i = lane; i < items; i += 32) {
            const int b = i / HW;
            body(((size_t)(b0 + b) * n + slot) * HW + (i - b * HW));
        }
    };
    auto walk_all = [&](int s0, int mine, auto&& body) {
        for (int t = 0; t < min(32, S - s0); t++) {
            const int slot = __shfl_sync(0xffffffffu, mine, t);
            if (slot >= 0) walk(s0 + t, slot, body);
        }
    };
    int first = -1;                                          // the slots of the first 32 sub-batches
    float cnt;
    // Sum and number of the elements of a channel.
    auto total = [&](int g, int inside) {
        double sum = 0.;                                     // a lane's chain grows with rows x HW: in fp32 its rounding showed (1.4e-7 -> 1.6e-7 of the mean)
        cnt = 0.f;
        for (int s0 = 0; s0 < S; s0 += 32) {
            const int mine = s0 + lane < S ? slot_in(s0 + lane, g, inside) : -1;
            if (s0 == 0) first = mine;
            if (mine >= 0) cnt += (float)(min(SNB_SUB_BATCH, B - (s0 + lane) * SNB_SUB_BATCH) * HW);
            walk_all(s0, mine, [&](size_t o) { sum += (double)x[o]; });
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            sum += __shfl_xor_sync(0xffffffffu, sum, d);
            cnt += __shfl_xor_sync(0xffffffffu, cnt, d);
        }
        return sum;
    };
    // Whether slot c of the list of sub-batch s0 + lane was found by its channel's warp (`entry`: the channel).  In a list that does not ascend, or names a
    // channel twice, some are not.
    const int gj = c / kept;
    auto lost_in = [&](int s0, int& entry) {
        const int s = s0 + lane;
        entry = s < S ? index[(size_t)s * n + c] : -1;
        return __ballot_sync(0xffffffffu, entry >= 0 && entry < per && place(s, gj, entry) != c - gj * kept);
    };
    const double sum = total(g, inside);
    if (!SHIFT) {
        if (lane == 0 && !index) out[c] = (float)sum;
        else if (lane == 0 && cnt > 0.f) atomicAdd(out + c, (float)sum);
        if (!index || c >= n) return;
        // What was not found is added here.  Lists that ascend end in one addition to zero per channel.
        for (int s0 = 0; s0 < S; s0 += 32) {
            int entry;
            unsigned lost = lost_in(s0, entry);
            for (; lost; lost &= lost - 1) {
                const int t = __ffs(lost) - 1;
                double part = 0.;
                walk(s0 + t, c, [&](size_t o) { part += (double)x[o]; });
#pragma unroll
                for (int d = 16; d > 0; d >>= 1) part += __shfl_xor_sync(0xffffffffu, part, d);
                const int channel = gj * per + __shfl_sync(0xffffffffu, entry, t);
                if (lane == 0) atomicAdd(out + channel, (float)part);
            }
        }
        return;
    }
    const float m = (float)(sum / fmaxf(cnt, 1e-10f));
    if (lane == 0) {
        out[c] = m;
        if (running_mean) running_mean[c] = running_mean[c] * (1.0f - momentum) + momentum * m;
    }
    for (int s0 = 0; s0 < S; s0 += 32) {
        const int mine = s0 == 0 ? first : s0 + lane < S ? slot_in(s0 + lane, g, inside) : -1;
        walk_all(s0, mine, [&](size_t o) { y[o] = x[o] - m; });
    }
    if (!index || c >= n) return;
    // The lists are to ascend; where one does not, what was not found is left out of the means, but every element of y is written.
    for (int s0 = 0; s0 < S; s0 += 32) {
        int entry;
        unsigned lost = lost_in(s0, entry);
        for (; lost; lost &= lost - 1) {
            const int t = __ffs(lost) - 1;
            const double its = total(gj, __shfl_sync(0xffffffffu, entry, t));
            const float mean = (float)(its / fmaxf(cnt, 1e-10f));
            walk(s0 + t, c, [&](size_t o) { y[o] = x[o] - mean; });
        }
    }
}

// y[b, j, :] = x[b, j, :] + v[channel j of b's list] (NaN where the list holds no channel).  Bound by the traffic of x and y.
__global__ void __launch_bounds__(256) plane_add_kernel(const float* __restrict__ x, const int* __restrict__ index, int G, int kept,
                                                        int HW, int C, const float* __restrict__ v, long long total, float* __restrict__ y) {
    const int n = G * kept, per = C / G;
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
        const long long row = i / HW;
        const int j = (int)(row % n), g = j / kept;
        const int s = (int)(row / n) / SNB_SUB_BATCH;
        const int inside = index ? index[(size_t)s * n + j] : j - g * kept;
        y[i] = (unsigned)inside < (unsigned)per ? x[i] + v[g * per + inside] : __int_as_float(0x7fc00000);
    }
}

static int check_plane(int B, int G, int kept, int hw, int channels, bool lists) {
    if (B <= 0 || G <= 0 || kept <= 0 || hw <= 0 || channels < (long long)G * kept || channels % G || (!lists && channels != G * kept))
        return SNB_ERR_BAD_SHAPE;
    return (long long)B * G * kept * hw >= (1ll << 31) ? SNB_ERR_TOO_LARGE : SNB_OK;
}

}  // namespace snb

using namespace snb;

extern "C" int snb_mean_shift_stats(const float* x, const int* index, int B, int C, int C_full,
                                    float* mean, float* running_mean, float momentum, void* stream) {
    if (!x || !mean) return SNB_ERR_NULL_POINTER;
    if (B <= 0 || C <= 0 || C_full < C || (!index && C_full != C)) return SNB_ERR_BAD_SHAPE;
    if ((long long)B * C >= (1ll << 31)) return SNB_ERR_TOO_LARGE;
    mean_shift_stats_kernel<<<(C_full + 15) / 16, 256, 0, (cudaStream_t)stream>>>(
        x, index, B, C, C_full, mean, running_mean, momentum);
    SNB_CUDA(launched());
    return SNB_OK;
}

extern "C" int snb_mean_shift_apply(const float* x, const float* mean, const int* index, int B, int C,
                                    float* y, void* stream) {
    if (!x || !mean || !y) return SNB_ERR_NULL_POINTER;
    if (B <= 0 || C <= 0) return SNB_ERR_BAD_SHAPE;
    if ((long long)B * C >= (1ll << 31)) return SNB_ERR_TOO_LARGE;
    dim3 grid((C + 255) / 256, (B + SNB_SUB_BATCH - 1) / SNB_SUB_BATCH);
    mean_shift_apply_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>(x, mean, index, B, C, y);
    SNB_CUDA(launched());
    return SNB_OK;
}

extern "C" int snb_plane_shift(const float* x, const int* index, int B, int G, int kept, int hw, int channels, float* mean,
                               float* running_mean, float momentum, float* y, void* stream) {
    if (!x || !mean || !y) return SNB_ERR_NULL_POINTER;
    const int rc = check_plane(B, G, kept, hw, channels, index != nullptr);
    if (rc) return rc;
    plane_shift_kernel<true><<<(channels + 7) / 8, 256, 0, (cudaStream_t)stream>>>(x, index, B, G, kept, hw, channels, mean, running_mean,
                                                                                   momentum, y);
    SNB_CUDA(launched());
    return SNB_OK;
}

extern "C" int snb_plane_sum(const float* x, const int* index, int B, int G, int kept, int hw, int channels, float* sum, void* stream) {
    if (!x || !sum) return SNB_ERR_NULL_POINTER;
    const int rc = check_plane(B, G, kept, hw, channels, index != nullptr);
    if (rc) return rc;
    if (index) SNB_CUDA(cudaMemsetAsync(sum, 0, sizeof(float) * channels, (cudaStream_t)stream));
    plane_shift_kernel<false><<<(channels + 7) / 8, 256, 0, (cudaStream_t)stream>>>(x, index, B, G, kept, hw, channels, sum, nullptr, 0.f,
                                                                                    nullptr);
    SNB_CUDA(launched());
    return SNB_OK;
}

extern "C" int snb_plane_add(const float* x, const int* index, int B, int G, int kept, int hw, int channels, const float* v, float* y,
                             void* stream) {
    if (!x || !v || !y) return SNB_ERR_NULL_POINTER;
    const int rc = check_plane(B, G, kept, hw, channels, index != nullptr);
    if (rc) return rc;
    const long long total = (long long)B * G * kept * hw, blocks = (total + 255) / 256, most = 16ll * sm_count();
    plane_add_kernel<<<(unsigned)(blocks < most ? blocks : most), 256, 0, (cudaStream_t)stream>>>(x, index, G, kept, hw, channels, v, total, y);
    SNB_CUDA(launched());
    return SNB_OK;
}
