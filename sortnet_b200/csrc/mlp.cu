// A whole SortNet-MLP in one call per direction: the p = infinity training pass (masked forward, margin and mixture loss,
// sparse backward) and the evaluation pass (point value and interval bounds, l-inf or sort neuron per layer).
//
// The layers are those of layer.cu, with the same arithmetic in the same order; what differs is what moves
// between them.  Activations stay in the form in which the pruned evaluation reads its input (prune.cuh:
// [sub-batch][channel][32 rows], full width, NaN in dropped channels), so a layer is filter + walk (+ redo of rejected outputs)
// + one pass that takes the batch mean off; nothing is gathered through index lists.  The backward keeps that form: one launch
// per layer adds to the gradient of the layer below, makes grad_w (rows cleared and added to in place) and takes the mean shift's
// backward on the way.  The host issues the launches of a whole direction from C.
#include "../../include/sortnet_b200.h"
#include "prune.cuh"

namespace snb {
namespace {

// Index lists [S][count] of the hidden layers -> flags [S][channels], one CTA per list.
constexpr int MAX_DEPTH = 16;
struct KeepJobs {
    const int* list[MAX_DEPTH];
    unsigned char* flags[MAX_DEPTH];
    int count[MAX_DEPTH], channels[MAX_DEPTH];
};
__global__ void __launch_bounds__(1024) keep_flags_kernel(const KeepJobs jobs) {
    const int* list = nullptr;
    unsigned char* flags = nullptr;
    int count = 0, channels = 0;
#pragma unroll
    for (int j = 0; j < MAX_DEPTH; j++)                      // compile-time indices keep the table in the parameter bank
        if (j == (int)blockIdx.y) list = jobs.list[j], flags = jobs.flags[j], count = jobs.count[j], channels = jobs.channels[j];
    if (!list) return;
    const int s = blockIdx.x;
    unsigned char* f = flags + (size_t)s * channels;
    for (int c = threadIdx.x; c < channels; c += 1024) f[c] = 0;
    __syncthreads();
#pragma unroll 4
    for (int k = threadIdx.x; k < count; k += 1024) {
        const int c = list[(size_t)s * count + k];
        if ((unsigned)c < (unsigned)channels) f[c] = 1;      // the lists are the caller's: an entry out of range keeps nothing
    }
}

// Training mean shift in the chain form: the batch mean of every channel from the sub-batches' row sums (in the order of
// mean_shift_stats_kernel, bit for bit), running mean, y - mean in place, and the column ranges of the result.
// CTA = 8 channels, lane = row.  Bound by latency: the first rows of y are fetched together with the sums, before the mean is known.
// 512 rows x 5120 channels: 12.6 us with 16 channels and y read after the mean, 10.3 with 8; with both a training pass of six layers
// 764 -> 733 us (4 channels: 743).  No __restrict__: no load may be moved ahead of after_previous().
constexpr int SHIFT_C = 8, SHIFT_S = 64;                     // sub-batches whose sums fit shared memory
__global__ void __launch_bounds__(256) chain_shift_kernel(float* yt, const float* part, const unsigned char* keep, int B, int S, int C,
                                                          float* running_mean, float momentum, float* rows_kept, unsigned* hi_out,
                                                          unsigned* nlo_out) {
    __shared__ float sums[SHIFT_S][SHIFT_C];                 // NaN: dropped
    __shared__ float mean[SHIFT_C];
    __shared__ unsigned hi[SHIFT_C], nlo[SHIFT_C];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c0 = blockIdx.x * SHIFT_C, n = min(SHIFT_C, C - c0);
    const int cx = tid & (SHIFT_C - 1), c = c0 + cx;
    after_previous();
    let_next();
    auto fetch = [&](int s) {
        const bool kept = cx < n && (!keep || keep[(size_t)s * C + c]);
        return kept ? part[(size_t)s * C + c] : __int_as_float(0x7fc00000);
    };
    const int items = S * SHIFT_C;                           // (sub-batch, channel) rows of 32
    float v[8];
    auto rows = [&](int i0) {
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int i = i0 + 8 * u, ch = i % SHIFT_C;
            v[u] = i < items && ch < n ? yt[((size_t)(i / SHIFT_C) * C + c0 + ch) * 32 + lane] : 0.f;
        }
    };
    rows(warp);
    for (int s = tid / SHIFT_C; s < min(S, SHIFT_S); s += 256 / SHIFT_C) sums[s][cx] = fetch(s);
    __syncthreads();
    if (tid < SHIFT_C) {
        hi[tid] = nlo[tid] = 0u;
        float t = 0.f, cnt = 0.f;
        for (int k = 0; k < 16; k++) {
            float sum = 0.f;
            for (int s = k; s < S; s += 16) {
                const float v = s < SHIFT_S ? sums[s][cx] : fetch(s);
                if (v == v) {
                    sum += v;
                    cnt += (float)(min(B, s * 32 + 32) - s * 32);
                }
            }
            t += sum;
        }
        const float m = t / fmaxf(cnt, 1e-10f);
        mean[tid] = m;
        if (tid < n) {
            rows_kept[c] = cnt;
            if (running_mean) running_mean[c] = running_mean[c] * (1.0f - momentum) + momentum * m;
        }
    }
    __syncthreads();
    for (int i0 = warp; i0 < items; i0 += 64) {
        if (i0 != warp) rows(i0);
#pragma unroll
        for (int u = 0; u < 8; u++) {
            const int i = i0 + 8 * u, ch = i % SHIFT_C;
            if (i >= items || ch >= n) continue;
            const float y = v[u] - mean[ch];
            yt[((size_t)(i / SHIFT_C) * C + c0 + ch) * 32 + lane] = y;
            const unsigned h = __reduce_max_sync(0xffffffffu, order_code(y)), l = __reduce_max_sync(0xffffffffu, order_code(-y));
            if (lane == 0) {
                atomicMax(&hi[ch], h);
                atomicMax(&nlo[ch], l);
            }
        }
    }
    __syncthreads();
    if (tid < n) hi_out[c] = hi[tid], nlo_out[c] = nlo[tid];
}

// Gradient of the head's outputs: g [B][C] * *scale -> gt [S][C][32], and its column sums (the bias gradient).
// CTA = 32 channels, warp = row of every sub-batch.  Bound by latency.
__global__ void __launch_bounds__(1024) head_gradient_kernel(const float* __restrict__ g, const float* __restrict__ scale, int B,
                                                             int S, int C, float* __restrict__ gt, float* __restrict__ col_sum) {
    __shared__ float tile[2][32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, c = blockIdx.x * 32 + lane, ch = blockIdx.x * 32 + warp;
    const float f = *scale;
    float sum = 0.f;
    for (int s = 0; s < S; s++) {
        const int b = s * 32 + warp;
        const float x = b < B && c < C ? g[(size_t)b * C + c] * f : 0.f;
        sum += x;
        tile[s & 1][warp][lane] = x;
        __syncthreads();                                     // the other buffer's readers are past their previous barrier
        if (ch < C) gt[((size_t)s * C + ch) * 32 + lane] = tile[s & 1][lane][warp];
    }
    if (!col_sum) return;
    __syncthreads();
    tile[0][warp][lane] = sum;
    __syncthreads();
    sum = tile[0][lane][warp];                               // the sums of channel `warp`
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if (lane == 0 && ch < C) col_sum[ch] = sum;
}

// Sparse l-inf backward of one layer, gradients in the form [sub-batch][channel][32 rows] like the words: two warps per output j,
// lane = row, up to CHAIN_S sub-batches at a time in registers.  The backward of the mean shift is taken on the way: g minus its mean
// over the rows that kept output j (g is 0 where it was dropped; rows_kept null: the head).  grad_x is added to the zeroed
// gradient of the layer below by reductions in L2, one per row, whose addresses share sectors (the rows of a sub-batch share a handful of
// argmax columns).  The row of grad_w is cleared by plain stores, and behind a barrier the few columns that occur get their sums over
// the rows, each column's over all sub-batches of the warp before it leaves it.  512 x 5120 x 5120: 31 us, bound by latency and the
// write of grad_w (16 us); the former kernels (grad_x in shared memory by a CTA per row, rows of grad_w too, the mean in a pass of
// its own) took 37 + 20 us.
constexpr int CHAIN_THREADS = 256, CHAIN_ROWS = CHAIN_THREADS / 64, CHAIN_S = 8;
struct ChainBwd {
    const float* gt;            // [S][CO][32]
    const int* post;            // [S][CO][32]
    const float* rows_kept;     // [CO] or null
    int S, CO, CI;
    float* gxt;                 // [S][CI][32], zeroed before, or null
    float* gx;                  // instead of gxt: [B][CI], zeroed before
    float* gw;                  // [CO][CI], or null
};
__global__ void __launch_bounds__(CHAIN_THREADS) chain_bwd_kernel(const ChainBwd a) {
    __shared__ float sums[CHAIN_ROWS][2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, group = warp >> 1, half = warp & 1, t64 = threadIdx.x & 63;
    const int j = (int)blockIdx.x * CHAIN_ROWS + group, CO = a.CO, CI = a.CI, S = a.S;
    after_previous();
    let_next();
    if (j >= CO) return;
    const int each = min(CHAIN_S, (S + 1) / 2);              // sub-batches per warp and turn
    uint32_t word[CHAIN_S];
    float v[CHAIN_S];
    auto fetch = [&](int s0) {
#pragma unroll
        for (int u = 0; u < CHAIN_S; u++) {
            const bool ok = u < each && s0 + u < S;
            const size_t o = ((size_t)(ok ? s0 + u : 0) * CO + j) * 32 + lane;
            word[u] = ok ? (uint32_t)a.post[o] : SNB_NO_GRAD_ID;
            v[u] = ok ? a.gt[o] : 0.f;
        }
    };
    float sum = 0.f;
    if (a.rows_kept)
        for (int s = 2 * each + half * each; s < S; s += 2 * each)                   // the turns after the first one
            for (int u = 0; u < each && s + u < S; u++) sum += a.gt[((size_t)(s + u) * CO + j) * 32 + lane];
    fetch(half * each);
    float* dst = a.gw + (size_t)j * CI;
    if (a.gw) {
        if ((CI & 3) == 0 && (reinterpret_cast<uintptr_t>(a.gw) & 15u) == 0)
            for (int c = t64; c < CI / 4; c += 64) reinterpret_cast<float4*>(dst)[c] = make_float4(0.f, 0.f, 0.f, 0.f);
        else
            for (int c = t64; c < CI; c += 64) dst[c] = 0.f;
    }
#pragma unroll
    for (int u = 0; u < CHAIN_S; u++) sum += v[u];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, d);
    if (lane == 0) sums[group][half] = sum;
    asm volatile("bar.sync %0, 64;" ::"r"(1 + group) : "memory");                    // sums, and the row of grad_w is cleared
    const float mean = a.rows_kept ? (sums[group][0] + sums[group][1]) / fmaxf(a.rows_kept[j], 1e-10f) : 0.f;
    for (int s0 = half * each;;) {
#pragma unroll
        for (int u = 0; u < CHAIN_S; u++) {
            if (word[u] == SNB_NO_GRAD_ID) continue;
            v[u] = (word[u] & SNB_SIGN_BIT) ? v[u] - mean : mean - v[u];             // into grad_w; grad_x gets the opposite
            word[u] &= ~SNB_SIGN_BIT;
            if (a.gxt) atomicAdd(a.gxt + ((size_t)(s0 + u) * CI + word[u]) * 32 + lane, -v[u]);
            else if (a.gx) atomicAdd(a.gx + (size_t)((s0 + u) * 32 + lane) * CI + word[u], -v[u]);
        }
        if (a.gw) {
#pragma unroll
            for (int u = 0; u < CHAIN_S; u++) {
                unsigned todo = __ballot_sync(0xffffffffu, word[u] != SNB_NO_GRAD_ID);
                while (todo) {
                    const uint32_t one = __shfl_sync(0xffffffffu, word[u], __ffs(todo) - 1);
                    float part = 0.f;
#pragma unroll
                    for (int k = u; k < CHAIN_S; k++)
                        if (word[k] == one) {
                            part += v[k];
                            word[k] = SNB_NO_GRAD_ID;
                        }
                    todo = __ballot_sync(0xffffffffu, word[u] != SNB_NO_GRAD_ID);
#pragma unroll
                    for (int d = 16; d > 0; d >>= 1) part += __shfl_xor_sync(0xffffffffu, part, d);
                    if (lane == 0) atomicAdd(dst + one, part);
                }
            }
        }
        s0 += 2 * each;
        if (s0 >= S) break;
        fetch(s0);
    }
}

// Scores and margins of the evaluation pass from the head's outputs (ell_inf_models.py:45-50): score = -y * scale,
// margin[b, c] = ((-yl[b, c]) - (-yu[b, t])) / (2 eps), 0 at the target.  A label outside [0, K) gives NaN.
__global__ void __launch_bounds__(256) scores_kernel(const float* __restrict__ y, const float* __restrict__ yl,
                                                     const float* __restrict__ yu, const long long* __restrict__ target, int B,
                                                     int K, float inv_two_eps, float scale, float* __restrict__ score,
                                                     float* __restrict__ margin) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= B * K) return;
    const int b = i / K, c = i % K;
    const long long t = target[b];
    score[i] = -y[i] * scale;
    if (t < 0 || t >= K) margin[i] = __int_as_float(0x7fc00000);
    else margin[i] = c == t ? 0.f * inv_two_eps : (-yl[i] - -yu[(size_t)b * K + t]) * inv_two_eps;
}

size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }

struct Cursor {
    char* base;
    size_t off = 0;
    template <class T>
    T* take(size_t n) {
        char* at = base + off;
        off += up256(sizeof(T) * n);
        return reinterpret_cast<T*>(at);
    }
};

// What the backward needs from the forward.
struct Saved {
    unsigned char* keep[MAX_DEPTH];
    int* post[MAX_DEPTH];
    float* rows_kept[MAX_DEPTH];
    float* grad_d;
};
size_t saved_layout(const snb_mlp_layer* l, int depth, int B, char* base, Saved* out) {
    const size_t S = (B + 31) / 32;
    Cursor at{base};
    Saved v{};
    for (int k = 0; k < depth; k++) {
        const size_t C = l[k].out;
        v.keep[k] = at.take<unsigned char>(l[k].kept_list ? S * C : 0);
        v.post[k] = at.take<int>(S * C * 32);
        v.rows_kept[k] = at.take<float>(C);
    }
    v.grad_d = at.take<float>((size_t)B * l[depth - 1].out);
    if (out) *out = v;
    return at.off;
}

int widest(const snb_mlp_layer* l, int depth) {
    int c = l[0].in;
    for (int k = 0; k < depth; k++) c = l[k].out > c ? l[k].out : c;
    return c;
}

PruneProblem layer_problem(const snb_mlp_layer* l, int k, int B, int tensors) {
    static const float some = 0.f;
    PruneProblem p;
    if (tensors != 2) p.x = &some;
    if (tensors != 1) p.xl = p.xu = &some;
    p.w = l[k].w;
    p.B = B, p.CO = p.W_CO = l[k].out, p.CI = p.W_CI = l[k].in;
    p.K = l[k].K, p.q = l[k].q;
    if (k > 0 && l[k - 1].kept_list) p.kept = l[k - 1].kept, p.kept_list = l[k - 1].kept_list;
    return p;
}

struct Scratch {
    char* zeroed;                  // fail counters and input ranges of every layer, one memset
    size_t zero_bytes;
    unsigned* counters[MAX_DEPTH];
    unsigned* hi[MAX_DEPTH];       // ranges of layer k's input
    unsigned* nlo[MAX_DEPTH];
    float* xt[2];
    float* part;
    float* d;
    float* row_loss;
    char* prune;
};
size_t scratch_layout(const snb_mlp_layer* l, int depth, int B, int tensors, bool training, char* base, Scratch* out) {
    const size_t S = (B + 31) / 32, W = widest(l, depth);
    Cursor at{base};
    Scratch v{};
    v.zeroed = base;
    for (int k = 0; k < depth; k++) {
        v.counters[k] = at.take<unsigned>(4);
        v.hi[k] = at.take<unsigned>(l[k].in);
        v.nlo[k] = at.take<unsigned>(l[k].in);
    }
    v.zero_bytes = at.off;
    for (int i = 0; i < 2; i++) v.xt[i] = at.take<float>(S * W * tensors * 32);
    v.part = at.take<float>(training ? S * W : 0);
    v.d = at.take<float>((size_t)tensors * B * l[depth - 1].out);
    v.row_loss = at.take<float>(B);
    size_t most = 0;
    static const float some = 0.f;
    static unsigned none = 0;
    static int word = 0;
    for (int k = 0; k < depth; k++) {
        PruneProblem p = layer_problem(l, k, B, tensors);
        p.xt = &some, p.hi = p.nlo = &none, p.counters = &none;
        if (training) p.post = &word;
        const size_t n = prune_workspace_bytes(p);
        most = n > most ? n : most;
    }
    v.prune = at.take<char>(most);
    if (out) *out = v;
    return at.off;
}

int check_layers(const snb_mlp_layer* l, int depth, int B) {
    if (!l) return SNB_ERR_NULL_POINTER;
    if (depth < 1 || B <= 0) return SNB_ERR_BAD_SHAPE;
    if (depth > MAX_DEPTH) return SNB_ERR_UNSUPPORTED;
    for (int k = 0; k < depth; k++) {
        if (l[k].in <= 0 || l[k].out <= 0 || (k > 0 && l[k].in != l[k - 1].out)) return SNB_ERR_BAD_SHAPE;
        if (l[k].kept_list && (l[k].kept <= 0 || l[k].kept > l[k].out)) return SNB_ERR_BAD_SHAPE;
        if (l[k].K < 1 || l[k].K > 25 || l[k].K > l[k].in) return SNB_ERR_UNSUPPORTED;
        if ((long long)l[k].in * l[k].out >= (1ll << 31) || (long long)B * l[k].in >= (1ll << 31) ||
            (long long)B * l[k].out >= (1ll << 31))
            return SNB_ERR_TOO_LARGE;
    }
    return SNB_OK;
}

}  // namespace
}  // namespace snb

using namespace snb;

// 1 when the calls below take these layers: rows of W within the filter's width, and enough work that nothing is lost on small
// nets.  Wall time of five-layer MNIST nets on a B200, by layers / whole: training 945 / 653 us at 3 M terms per layer, 1093 / 539 at 25 M,
// 1200 / 596 at 50 M; certification 693 / 272, 889 / 331, 911 / 346.
extern "C" int snb_mlp_applies(const snb_mlp_layer* l, int depth, int B) {
    if (check_layers(l, depth, B) != SNB_OK || (B + 31) / 32 > 65535) return 0;
    long long work = 0;
    for (int k = 0; k < depth; k++) {
        if (l[k].in > 12288 || l[k].in < 64) return 0;
        work += (long long)B * l[k].in * l[k].out;
    }
    return work >= (16ll << 20) * depth;
}

extern "C" size_t snb_mlp_saved_bytes(const snb_mlp_layer* l, int depth, int B) {
    return check_layers(l, depth, B) == SNB_OK ? saved_layout(l, depth, B, nullptr, nullptr) : 0;
}
extern "C" size_t snb_mlp_scratch_bytes(const snb_mlp_layer* l, int depth, int B, int tensors, int training) {
    return check_layers(l, depth, B) == SNB_OK ? scratch_layout(l, depth, B, tensors, training != 0, nullptr, nullptr) : 0;
}
// backward: the gradients of all layers' outputs
extern "C" size_t snb_mlp_backward_scratch_bytes(const snb_mlp_layer* l, int depth, int B) {
    if (check_layers(l, depth, B) != SNB_OK) return 0;
    size_t n = 0;
    for (int k = 0; k < depth; k++) n += up256(sizeof(float) * (size_t)((B + 31) / 32) * 32 * l[k].out);
    return n;
}

extern "C" int snb_mlp_train_forward(const snb_mlp_layer* l, int depth, const float* x, int B, const long long* targets, float eps,
                                     float clip, float lam, float scale, void* saved, void* scratch, float* loss, int* launches,
                                     void* stream) {
    int rc = check_layers(l, depth, B);
    if (rc) return rc;
    if (!x || !targets || !saved || !scratch || !loss) return SNB_ERR_NULL_POINTER;
    cudaStream_t st = (cudaStream_t)stream;
    const int S = (B + 31) / 32;
    Saved sv;
    Scratch sc;
    saved_layout(l, depth, B, static_cast<char*>(saved), &sv);
    scratch_layout(l, depth, B, 1, true, static_cast<char*>(scratch), &sc);
    int count = 0;
    SNB_CUDA(cudaMemsetAsync(sc.zeroed, 0, sc.zero_bytes, st));
    KeepJobs jobs{};
    int masked = 0;
    for (int k = 0; k < depth; k++)
        if (l[k].kept_list) {
            jobs.list[masked] = l[k].kept_list, jobs.flags[masked] = sv.keep[k];
            jobs.count[masked] = l[k].kept, jobs.channels[masked] = l[k].out;
            masked++;
        }
    if (masked) {
        keep_flags_kernel<<<dim3(S, masked), 1024, 0, st>>>(jobs);
        SNB_CUDA(launched());
        count++;
    }
    PrunePrep prep;
    prep.x = x, prep.B = B, prep.CI = prep.W_CI = l[0].in;
    prep.xt = sc.xt[0], prep.hi = sc.hi[0], prep.nlo = sc.nlo[0];
    SNB_CUDA(prune_prepare(prep, st));
    count++;
    for (int k = 0; k < depth; k++) {
        const bool head = k == depth - 1;
        const int C = l[k].out;
        PruneProblem p = layer_problem(l, k, B, 1);
        p.xt = sc.xt[k & 1], p.hi = sc.hi[k], p.nlo = sc.nlo[k], p.counters = sc.counters[k];
        p.post = sv.post[k];
        if (l[k].kept_list) p.keep = sv.keep[k], p.out_list = l[k].kept_list, p.out_kept = l[k].kept;
        if (head) {
            p.y = sc.d;
            p.bias = l[k].bias;
        } else {
            p.yt = sc.xt[(k + 1) & 1];
            p.part = sc.part;
        }
        SNB_CUDA(prune_forward(p, sc.prune, st));
        count += 3;
        if (!head) {
            SNB_CUDA(launch_next(chain_shift_kernel, (C + SHIFT_C - 1) / SHIFT_C, 256, 0, st, p.yt, p.part, p.keep, B, S, C, l[k].running_mean,
                                 l[k].momentum, sv.rows_kept[k], sc.hi[k + 1], sc.nlo[k + 1]));
            count++;
        }
    }
    rc = snb_margin_loss(sc.d, targets, B, l[depth - 1].out, eps, clip, lam, scale, nullptr, sc.row_loss, loss, sv.grad_d, stream);
    if (rc) return rc;
    if (launches) *launches = count + 2;
    return SNB_OK;
}

// grad_w [depth] (entries may be null), grad_bias of the head and grad_x [B, in] optional; grad_loss: device scalar.
extern "C" int snb_mlp_train_backward(const snb_mlp_layer* l, int depth, int B, const float* grad_loss, const void* saved,
                                      void* scratch, float* const* grad_w, float* grad_bias, float* grad_x, int* launches,
                                      void* stream) {
    int rc = check_layers(l, depth, B);
    if (rc) return rc;
    if (!grad_loss || !saved || !scratch || !grad_w) return SNB_ERR_NULL_POINTER;
    cudaStream_t st = (cudaStream_t)stream;
    const int S = (B + 31) / 32;
    Saved sv;
    saved_layout(l, depth, B, const_cast<char*>(static_cast<const char*>(saved)), &sv);
    Cursor at{static_cast<char*>(scratch)};
    float* gt[MAX_DEPTH];
    for (int k = 0; k < depth; k++) gt[k] = at.take<float>((size_t)S * 32 * l[k].out);
    int lowest = 0;                                          // deepest layer that anybody wants a gradient from
    while (!grad_x && lowest < depth && !grad_w[lowest]) lowest++;
    if (lowest == depth && grad_bias) lowest = depth - 1;
    if (lowest == depth) {
        if (launches) *launches = 0;
        return SNB_OK;
    }
    const int classes = l[depth - 1].out;
    if (lowest < depth - 1)
        SNB_CUDA(cudaMemsetAsync(gt[lowest], 0, (char*)gt[depth - 1] - (char*)gt[lowest], st));
    if (grad_x) SNB_CUDA(cudaMemsetAsync(grad_x, 0, sizeof(float) * (size_t)B * l[0].in, st));
    head_gradient_kernel<<<(classes + 31) / 32, 1024, 0, st>>>(sv.grad_d, grad_loss, B, S, classes, gt[depth - 1], grad_bias);
    SNB_CUDA(launched());
    int count = 1;
    for (int k = depth - 1; k >= lowest; k--) {
        ChainBwd a{};
        a.gt = gt[k], a.post = sv.post[k], a.rows_kept = k < depth - 1 ? sv.rows_kept[k] : nullptr;
        a.S = S, a.CO = l[k].out, a.CI = l[k].in;
        if (k > lowest) a.gxt = gt[k - 1];
        else if (k == 0) a.gx = grad_x;
        a.gw = grad_w[k];
        if (!a.gxt && !a.gx && !a.gw) continue;
        SNB_CUDA(launch_next(chain_bwd_kernel, (a.CO + CHAIN_ROWS - 1) / CHAIN_ROWS, CHAIN_THREADS, 0, st, a));
        count++;
    }
    if (launches) *launches = count;
    return SNB_OK;
}

// Evaluation pass.  tensors = 1: y only; 3: y, yl, yu for the box xl, xu, or (xl null) [max(x - eps, down), min(x + eps, up)].
// y, yl, yu [B, classes] are the head's outputs; score / margin optional (tensors = 3, targets given).
extern "C" int snb_mlp_eval_forward(const snb_mlp_layer* l, int depth, const float* x, const float* xl, const float* xu, int B,
                                    int tensors, float box_eps, float down, float up, void* scratch, float* y, float* yl,
                                    float* yu, const long long* targets, float inv_two_eps, float scale, float* score,
                                    float* margin, int* launches, void* stream) {
    int rc = check_layers(l, depth, B);
    if (rc) return rc;
    if (!x || !scratch || !y || (tensors == 3 && (!yl || !yu)) || ((xl != nullptr) != (xu != nullptr))) return SNB_ERR_NULL_POINTER;
    if (tensors != 1 && tensors != 3) return SNB_ERR_UNSUPPORTED;
    if (score && (tensors != 3 || !targets || !margin)) return SNB_ERR_NULL_POINTER;
    cudaStream_t st = (cudaStream_t)stream;
    Scratch sc;
    scratch_layout(l, depth, B, tensors, false, static_cast<char*>(scratch), &sc);
    int count = 0;
    SNB_CUDA(cudaMemsetAsync(sc.zeroed, 0, sc.zero_bytes, st));
    PrunePrep prep;
    prep.x = x, prep.B = B, prep.CI = prep.W_CI = l[0].in;
    if (tensors == 3) prep.xl = xl, prep.xu = xu, prep.box = !xl, prep.eps = box_eps, prep.down = down, prep.up = up;
    prep.xt = sc.xt[0], prep.hi = sc.hi[0], prep.nlo = sc.nlo[0];
    SNB_CUDA(prune_prepare(prep, st));
    for (int k = 0; k < depth; k++) {
        PruneProblem p = layer_problem(l, k, B, tensors);
        p.xt = sc.xt[k & 1], p.hi = sc.hi[k], p.nlo = sc.nlo[k], p.counters = sc.counters[k];
        p.mean = l[k].running_mean, p.bias = l[k].bias;
        if (k == depth - 1) {
            p.y = y;
            if (tensors == 3) p.yl = yl, p.yu = yu;
        } else {
            p.yt = sc.xt[(k + 1) & 1], p.yhi = sc.hi[k + 1], p.ynlo = sc.nlo[k + 1];
        }
        SNB_CUDA(prune_forward(p, sc.prune, st));
        count += 3;
    }
    if (score) {
        const int n = B * l[depth - 1].out;
        scores_kernel<<<(n + 255) / 256, 256, 0, st>>>(y, yl, yu, targets, B, l[depth - 1].out, inv_two_eps, scale, score, margin);
        SNB_CUDA(launched());
        count++;
    }
    if (launches) *launches = count + 1;
    return SNB_OK;
}
