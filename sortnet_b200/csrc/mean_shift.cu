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
#include <cooperative_groups.h>

#include <type_traits>

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

// The same over rows and positions of x [B, n, HW] (n kept channels of G groups, lists of within-group channels): a channel's HW neighbouring
// floats of every row that kept it are walked twice, for the sum and for the result; the second time they come from L1 or L2.  SHIFT: the mean into
// `out`, x minus it into y; otherwise the sums alone.  Bound by latency, four loads in flight per thread and 22 % of the warps that fit: 512 x 64 x 1024 92 us, DRAM at 47 %
// of its peak (the sums alone 49 us, 34 %); 128 x 1024 x 4 4.6 us, most of it the start and the two dependent searches and walks.
struct PlaneArgs {
    const float* x;
    const int* index;
    int B, G, kept, HW, C;
    float* out;
    float* running_mean;
    float momentum;
    float* y;
};

constexpr int PLANE_THREADS = 256;

// WIDE: a cluster of CTAs per channel, else a warp.  V: floats per load (HW is a multiple of it).
template <bool SHIFT, bool WIDE, int V>
__global__ void __launch_bounds__(PLANE_THREADS) plane_shift_kernel(const PlaneArgs a) {
    namespace cg = cooperative_groups;
    using Vec = std::conditional_t<V == 4, float4, float>;
    constexpr int MINE = WIDE ? PLANE_THREADS : 32, LOADS = 4;   // threads of this CTA per channel, loads in flight per thread
    __shared__ int table[PLANE_THREADS / MINE][MINE];        // slots of a channel in the lists of MINE sub-batches
    __shared__ double part[PLANE_THREADS / 32], whole;
    __shared__ int rows_part[PLANE_THREADS / 32], entry_of[WIDE ? MINE : 1];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, me = WIDE ? threadIdx.x : lane;
    const unsigned ranks = WIDE ? cg::this_cluster().num_blocks() : 1, rank = WIDE ? cg::this_cluster().block_rank() : 0;
    const int c = WIDE ? (int)(blockIdx.x / ranks) : (int)blockIdx.x * 8 + warp;
    if (c >= a.C) return;
    int* const slots = table[WIDE ? 0 : warp];
    const int B = a.B, kept = a.kept, n = a.G * kept, per = a.C / a.G, S = (B - 1) / SNB_SUB_BATCH + 1;
    // unit: V neighbouring positions of a row.  This thread's first unit and its step, as rows and units within a row.
    const unsigned units = a.HW / V, first_unit = rank * MINE + me, threads = ranks * MINE;
    const unsigned row0 = first_unit / units, pos0 = first_unit % units, row_step = threads / units, pos_step = threads % units;
    auto sync = [&]() {
        if (WIDE) __syncthreads();
        else __syncwarp();
    };
    // Place of channel `want` in list g of sub-batch s: that of the first entry that is not smaller, if the list ascends.
    auto place = [&](int s, int g, int want) {
        const int* list = a.index + ((size_t)s * a.G + g) * kept;
        int lo = 0, hi = kept;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (list[mid] < want) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    };
    auto slot_in = [&](int s, int g, int inside) {
        if (!a.index) return inside;
        const int at = place(s, g, inside);
        return at < kept && a.index[((size_t)s * a.G + g) * kept + at] == inside ? g * kept + at : -1;
    };
    auto load = [&](size_t o) { return *reinterpret_cast<const Vec*>(a.x + o); };
    // body(offsets, which of them are there) for this thread's units of the rows [from, to); slot(row): -1 for rows that dropped the channel
    auto walk = [&](unsigned from, unsigned to, auto&& slot, auto&& body) {
        unsigned row = from + row0, pos = pos0;
        while (row < to) {
            size_t o[LOADS];
            bool here[LOADS];
#pragma unroll
            for (int q = 0; q < LOADS; q++) {
                const int at = row < to ? slot(row) : -1;
                here[q] = at >= 0;
                o[q] = ((size_t)row * n + at) * a.HW + (size_t)pos * V;
                row += row_step, pos += pos_step;
                if (pos >= units) pos -= units, row++;
            }
            body(o, here);
        }
    };
    auto add_up = [&](double& sum) {
        return [&](const size_t(&o)[LOADS], const bool(&here)[LOADS]) {
            Vec v[LOADS];
#pragma unroll
            for (int q = 0; q < LOADS; q++) v[q] = here[q] ? load(o[q]) : Vec{};
#pragma unroll
            for (int q = 0; q < LOADS; q++) {
                if constexpr (V == 4) sum += ((double)v[q].x + (double)v[q].y) + ((double)v[q].z + (double)v[q].w);
                else sum += (double)v[q];
            }
        };
    };
    auto subtract = [&](float m) {
        return [&, m](const size_t(&o)[LOADS], const bool(&here)[LOADS]) {
            Vec v[LOADS];
#pragma unroll
            for (int q = 0; q < LOADS; q++)
                if (here[q]) v[q] = load(o[q]);
#pragma unroll
            for (int q = 0; q < LOADS; q++)
                if (here[q]) {
                    if constexpr (V == 4) v[q].x -= m, v[q].y -= m, v[q].z -= m, v[q].w -= m;
                    else v[q] -= m;
                    *reinterpret_cast<Vec*>(a.y + o[q]) = v[q];
                }
        };
    };
    // Sums over the threads of the channel, in a fixed order; rows: the same in every CTA.
    auto over_all = [&](double& sum, int& rows) {
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            sum += __shfl_xor_sync(0xffffffffu, sum, d);
            rows += __shfl_xor_sync(0xffffffffu, rows, d);
        }
        if constexpr (WIDE) {
            if (lane == 0) part[warp] = sum, rows_part[warp] = rows;
            __syncthreads();
            sum = 0., rows = 0;
#pragma unroll
            for (int w = 0; w < PLANE_THREADS / 32; w++) sum += part[w], rows += rows_part[w];
            if (ranks > 1) {
                if (threadIdx.x == 0) whole = sum;
                cg::this_cluster().sync();
                sum = 0.;
                for (unsigned r = 0; r < ranks; r++) sum += *cg::this_cluster().map_shared_rank(&whole, r);
                cg::this_cluster().sync();                   // before `whole` is written again, or its CTA ends
            }
            __syncthreads();
        }
    };
    auto put_slots = [&](int s0, int g, int inside) {
        const int s = s0 + me, slot = s < S ? slot_in(s, g, inside) : -1;
        sync();                                              // the readers of the slots before are done
        slots[me] = slot;
        sync();
        return slot >= 0 ? min(SNB_SUB_BATCH, B - s * SNB_SUB_BATCH) : 0;
    };
    auto walk_slots = [&](int s0, auto&& body) {
        const long long end = (long long)(s0 + MINE) * SNB_SUB_BATCH;
        walk((unsigned)s0 * SNB_SUB_BATCH, end < B ? (unsigned)end : (unsigned)B, [&](unsigned row) { return slots[row / SNB_SUB_BATCH - s0]; }, body);
    };
    int rows;
    auto total = [&](int g, int inside) {
        double sum = 0.;                                     // in 64 bits: a thread's chain grows with rows x HW
        rows = 0;
        for (int s0 = 0; s0 < S; s0 += MINE) {
            rows += put_slots(s0, g, inside);
            walk_slots(s0, add_up(sum));
        }
        over_all(sum, rows);
        return sum;
    };
    auto mean_of = [&](double sum) { return rows ? (float)(sum / ((double)rows * a.HW)) : 0.f; };
    // Calls body(s, channel) for every list in which slot c was not found by its channel's threads.  In a list that does not ascend, or names a
    // channel twice, some are not.
    auto each_lost = [&](auto&& body) {
        if (!a.index || c >= n) return;
        const int gj = c / kept;
        for (int s0 = 0; s0 < S; s0 += MINE) {
            const int s = s0 + me;
            int entry = s < S ? a.index[(size_t)s * n + c] : -1;
            if (entry >= per || (entry >= 0 && place(s, gj, entry) == c - gj * kept)) entry = -1;
            if (!WIDE) {
                for (unsigned lost = __ballot_sync(0xffffffffu, entry >= 0); lost; lost &= lost - 1) {
                    const int t = __ffs(lost) - 1;
                    body(s0 + t, gj, __shfl_sync(0xffffffffu, entry, t));
                }
            } else if (__syncthreads_or(entry >= 0)) {
                entry_of[WIDE ? me : 0] = entry;
                __syncthreads();
                for (int t = 0; t < min(MINE, S - s0); t++)
                    if (const int lost = entry_of[WIDE ? t : 0]; lost >= 0) body(s0 + t, gj, lost);
                __syncthreads();
            }
        }
    };
    auto rows_of = [&](int s, auto&& body) {                 // slot c of one sub-batch
        const unsigned from = (unsigned)s * SNB_SUB_BATCH;
        walk(from, from + min(SNB_SUB_BATCH, B - s * SNB_SUB_BATCH), [&](unsigned) { return c; }, body);
    };

    const int g = c / per, inside = c - g * per;
    const bool writer = me == 0 && rank == 0;
    const double sum = total(g, a.index ? inside : c);
    if (!SHIFT) {
        if (writer && !a.index) a.out[c] = (float)sum;
        else if (writer && rows) atomicAdd(a.out + c, (float)sum);
        // What was not found is added here.  Lists that ascend end in one addition to zero per channel.
        each_lost([&](int s, int g, int inside) {
            double its = 0.;
            int none = 0;
            rows_of(s, add_up(its));
            over_all(its, none);
            if (writer) atomicAdd(a.out + g * per + inside, (float)its);
        });
        return;
    }
    const float m = mean_of(sum);
    if (writer) {
        a.out[c] = m;
        if (a.running_mean) a.running_mean[c] = a.running_mean[c] * (1.0f - a.momentum) + a.momentum * m;
    }
    for (int s0 = 0; s0 < S; s0 += MINE) {
        if (S > MINE) put_slots(s0, g, a.index ? inside : c);
        walk_slots(s0, subtract(m));
    }
    // The lists are to ascend; where one does not, what was not found is left out of the means, but every element of y is written.
    each_lost([&](int s, int g, int inside) {
        const double its = total(g, inside);
        rows_of(s, subtract(mean_of(its)));
    });
}

// y[b, j, :] = x[b, j, :] + v[channel j of b's list] (NaN where the list holds no channel).  Bound by the traffic of x and y (512 x 64 x 1024 39 us, DRAM at
// 69 % of its peak).  A thread goes through the units (V floats) in strides and keeps row, slot and position of the next one, so that nothing is divided per unit.
template <int V>
__global__ void __launch_bounds__(PLANE_THREADS) plane_add_kernel(const PlaneArgs a, const float* __restrict__ v) {
    using Vec = std::conditional_t<V == 4, float4, float>;
    constexpr int LOADS = 4;
    const int n = a.G * a.kept, per = a.C / a.G;
    const unsigned units = a.HW / V, stride = gridDim.x * PLANE_THREADS;
    const unsigned long long first = (unsigned long long)blockIdx.x * PLANE_THREADS + threadIdx.x;
    unsigned pos = first % units, slot = first / units % n, row = (unsigned)(first / units / n);
    const unsigned pos_step = stride % units, slot_step = stride / units % n, row_step = stride / units / n;
    while (row < (unsigned)a.B) {
        size_t o[LOADS];
        bool here[LOADS];
        Vec x[LOADS];
        float add[LOADS];
#pragma unroll
        for (int q = 0; q < LOADS; q++) {
            here[q] = row < (unsigned)a.B;
            o[q] = ((size_t)row * n + slot) * a.HW + (size_t)pos * V;
            if (here[q]) {
                x[q] = *reinterpret_cast<const Vec*>(a.x + o[q]);
                int channel = (int)slot;
                bool ok = true;
                if (a.index) {
                    const int inside = a.index[(size_t)(row / SNB_SUB_BATCH) * n + slot];
                    ok = (unsigned)inside < (unsigned)per;
                    channel = a.G == 1 ? inside : (int)slot / a.kept * per + inside;
                }
                add[q] = ok ? v[channel] : __int_as_float(0x7fc00000);
            }
            pos += pos_step, slot += slot_step, row += row_step;
            if (pos >= units) pos -= units, slot++;
            if (slot >= (unsigned)n) slot -= n, row++;
        }
#pragma unroll
        for (int q = 0; q < LOADS; q++)
            if (here[q]) {
                if constexpr (V == 4) x[q].x += add[q], x[q].y += add[q], x[q].z += add[q], x[q].w += add[q];
                else x[q] += add[q];
                *reinterpret_cast<Vec*>(a.y + o[q]) = x[q];
            }
    }
}

static int check_plane(int B, int G, int kept, int hw, int channels, bool lists) {
    if (B <= 0 || G <= 0 || kept <= 0 || hw <= 0 || channels < (long long)G * kept || channels % G || (!lists && channels != G * kept))
        return SNB_ERR_BAD_SHAPE;
    return SNB_OK;
}

template <bool SHIFT, bool WIDE, int V>
static cudaError_t launch_plane(const PlaneArgs& a, int ranks, cudaStream_t st) {
    cudaLaunchAttribute cluster;
    cluster.id = cudaLaunchAttributeClusterDimension;
    cluster.val.clusterDim.x = (unsigned)ranks, cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
    cudaLaunchConfig_t config = {};
    config.gridDim = WIDE ? (unsigned)a.C * ranks : (a.C + 7) / 8, config.blockDim = PLANE_THREADS, config.stream = st;
    config.attrs = &cluster, config.numAttrs = WIDE && ranks > 1 ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&config, plane_shift_kernel<SHIFT, WIDE, V>, a);
    const cudaError_t last = launched();                     // takes a failed launch's error away, so that no later call reports it
    return e != cudaSuccess ? e : last;
}

// A warp per channel where there are many channels and little to walk for each, a cluster of 1 to 8 CTAs where it is the other way round: CTAs that are not there
// leave SMs idle, CTAs with little to do cost their start.  The lines: a unit per thread of a CTA and more units per channel than channels; two, four, eight CTAs
// while a thread has more than 16 units and the device 1.25 CTAs per SM at most.  B200, inside a graph, mean shift in us (rows x channels x positions; "m": of 4/3 as many
// channels, with lists):
//                        warp   1 CTA     2     4     8                         warp   1 CTA     2     4     8
//     128 x 1024 x 4      4.6     9.3  21.2  38.0  72.6    128 x 64 x 64        19.5     4.5   4.8   5.4   9.4
//     128 x 1024 x 4 m    8.1    18.1  41.0  80.8   169    8192 x 64 x 1 m       121    20.5  20.6  18.6  20.1
//     512 x 1024 x 4     10.7    13.4  24.5  42.8  80.8    128 x 128 x 225       137    22.7  16.3  16.2  18.5
//     300 x 5000 x 4 m   38.2    99.1   229   468   988    128 x 256 x 256      69.1    14.4  18.8  20.2  28.9
//     1024 x 1000 x 1 m  20.9    25.2  38.2  57.8   109    128 x 64 x 1024       274    37.8  22.0  15.5  21.1
//     4096 x 1024 x 4    98.7    83.8  87.0   102   139    512 x 64 x 1024      1886     279   154  96.2  98.9
//     192 x 512 x 9      11.4     7.6  11.3  16.7  28.7    128 x 16 x 1024       265    37.1  21.5  12.5   9.7
//     128 x 256 x 16      6.6     4.3   8.7  11.9  21.4    512 x 3 x 1024        923     138  71.7  37.8  21.1
// As launches over (channel, position) columns with their lists, averages and running mean apart (11 to 13 of them), kernels alone: 128 x 1024 x 4 16 to 19, 128 x 64 x
// 1024 75 to 84, 512 x 64 x 1024 114 to 130, 4096 x 1024 x 4 125 to 146, 1024 x 1000 x 1 m 20.
template <bool SHIFT>
static cudaError_t run_plane(const PlaneArgs& a, cudaStream_t st) {
    const bool four = a.HW % 4 == 0 && aligned16(a.x) && (!SHIFT || aligned16(a.y));
    const long long units = (long long)a.B * (four ? a.HW / 4 : a.HW);
    int ranks = 0;                                           // a warp per channel
    if (units >= 256 && units >= a.C)
        for (ranks = 1; ranks < 8 && units > 4096ll * ranks && 4ll * a.C * ranks <= 5ll * sm_count();) ranks *= 2;
    if (ranks == 0) return four ? launch_plane<SHIFT, false, 4>(a, 1, st) : launch_plane<SHIFT, false, 1>(a, 1, st);
    return four ? launch_plane<SHIFT, true, 4>(a, ranks, st) : launch_plane<SHIFT, true, 1>(a, ranks, st);
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
    SNB_CUDA(run_plane<true>({x, index, B, G, kept, hw, channels, mean, running_mean, momentum, y}, (cudaStream_t)stream));
    return SNB_OK;
}

extern "C" int snb_plane_sum(const float* x, const int* index, int B, int G, int kept, int hw, int channels, float* sum, void* stream) {
    if (!x || !sum) return SNB_ERR_NULL_POINTER;
    const int rc = check_plane(B, G, kept, hw, channels, index != nullptr);
    if (rc) return rc;
    if (index) SNB_CUDA(cudaMemsetAsync(sum, 0, sizeof(float) * channels, (cudaStream_t)stream));
    SNB_CUDA(run_plane<false>({x, index, B, G, kept, hw, channels, sum, nullptr, 0.f, nullptr}, (cudaStream_t)stream));
    return SNB_OK;
}

extern "C" int snb_plane_add(const float* x, const int* index, int B, int G, int kept, int hw, int channels, const float* v, float* y,
                             void* stream) {
    if (!x || !v || !y) return SNB_ERR_NULL_POINTER;
    const int rc = check_plane(B, G, kept, hw, channels, index != nullptr);
    if (rc) return rc;
    const PlaneArgs a{x, index, B, G, kept, hw, channels, nullptr, nullptr, 0.f, y};
    const bool four = hw % 4 == 0 && aligned16(x) && aligned16(y);
    const long long units = (long long)B * G * kept * (four ? hw / 4 : hw), blocks = (units + 4 * PLANE_THREADS - 1) / (4 * PLANE_THREADS), most = 8ll * sm_count();
    const unsigned grid = (unsigned)(blocks < most ? blocks : most);
    if (four) plane_add_kernel<4><<<grid, PLANE_THREADS, 0, (cudaStream_t)stream>>>(a, v);
    else plane_add_kernel<1><<<grid, PLANE_THREADS, 0, (cudaStream_t)stream>>>(a, v);
    SNB_CUDA(launched());
    return SNB_OK;
}
