// l-p distance neuron for whole p in 1 .. 8: dense forward and backward.
//
// Replaces zbh2047/SortNet core/cuda/norm_dist_cuda.cu (forward kernels :36-160, backward kernels :269-504) for the exponents
// that its dispatch (core/cuda/norm_dist.cpp:43-129) gives multiply chains of their own.
//
//   y = max(sum_c |x - w|^p, FLT_MIN)^(1/p);    term = g sgn(t) (|t| / y)^(p-1),  t = x - w
//   grad_x[b,c] = sum_j term;    grad_w[co[s][j], ci[s][c]] -= sum_{b in sub-batch s} term
//
// Both are bound by the fp32 pipe: subtract, multiply chain and fma, for p = 8 four operations per term of the forward and seven of
// the backward.  Everything is done on pairs of values (sub / mul / fma .f32x2: two operations per issued instruction, at the
// pipe's full rate), which leaves half of the issue slots for loads and addresses.  B200, 512 x 5120 x 5120, scalar kernels with four
// lanes per column -> these: p = 8 forward 1.74 -> 1.61 ms, backward 4.46 -> 3.56; p = 2 0.99 -> 0.95, 2.94 -> 2.14; p = 5 backward
// 3.88 -> 3.3.  Cycles in which the pipe is busy at p = 8 (256 x 3840 x 5120): forward 91 %, backward 76 % (7 operations per term: 2.6 ms
// of the 3.56 above; the reductions into grad_w are 4 % of it).
#include <float.h>
#include "launch.h"
#include "lp_dense.h"
#include "lp_math.cuh"
#include "tile.cuh"

namespace snb {

namespace {

// Two values per 64-bit register pair.  Where a magnitude enters, the two halves are taken one by one: |.| is free as an operand of
// scalar instructions, and none of the packed ones (p = 3, 512 x 5120 x 5120 forward: 1.47 ms scalar, 1.68 ms with |t| made by
// logic instructions).
__device__ __forceinline__ uint64_t mul_abs(uint64_t t, uint64_t a) {    // |t| a
    float t0, t1, a0, a1;
    unpack2(t, t0, t1), unpack2(a, a0, a1);
    return pack2(fabsf(t0) * a0, fabsf(t1) * a1);
}
__device__ __forceinline__ uint64_t fma_abs(uint64_t t, uint64_t a, uint64_t c) {   // |t| a + c
    float t0, t1, a0, a1, c0, c1;
    unpack2(t, t0, t1), unpack2(a, a0, a1), unpack2(c, c0, c1);
    return pack2(fmaf(fabsf(t0), a0, c0), fmaf(fabsf(t1), a1, c1));
}
__device__ __forceinline__ uint64_t with_sign(uint64_t a, uint64_t t) {  // a >= 0 with the sign of t
    return a | (t & 0x8000000080000000ull);
}

// acc + |t|^IP, IP = 1 .. 8.
template <int IP>
__device__ __forceinline__ uint64_t add_pow(uint64_t t, uint64_t acc) {
    if (IP == 1) return fma_abs(t, pack2(1.0f, 1.0f), acc);
    if (IP == 2) return fma2(t, t, acc);
    const uint64_t a = mul2(t, t);
    if (IP == 3) return fma_abs(t, a, acc);
    if (IP == 4) return fma2(a, a, acc);
    const uint64_t b = mul2(a, a);
    if (IP == 5) return fma_abs(t, b, acc);
    if (IP == 6) return fma2(a, b, acc);
    if (IP == 7) return fma2(mul_abs(t, a), b, acc);
    return fma2(b, b, acc);
}

// sgn(t) * |t|^IP, IP = 0 .. 7; sgn(0) = 1 and sgn(NaN) = -1 as a comparison with 0 gives them.
template <int IP>
__device__ __forceinline__ uint64_t signed_pow(uint64_t t) {
    if (IP == 0) {
        float lo, hi;
        unpack2(t, lo, hi);
        return pack2(lo >= 0.f ? 1.0f : -1.0f, hi >= 0.f ? 1.0f : -1.0f);
    }
    if (IP == 1) return t;
    if (IP == 2) return mul_abs(t, t);
    const uint64_t a = mul2(t, t);
    if (IP == 3) return mul2(a, t);
    if (IP == 4) return mul2(a, with_sign(a, t));
    const uint64_t b = mul2(a, a);
    if (IP == 5) return mul2(b, t);
    if (IP == 6) return mul2(b, with_sign(a, t));
    return mul2(b, mul2(a, t));
}
// r^IP for r >= 0
template <int IP>
__device__ __forceinline__ float whole_pow(float r) {
    if constexpr (IP == 0) {
        return 1.0f;
    } else {
        const float half = whole_pow<IP / 2>(r);
        return IP % 2 ? r * half * half : half * half;
    }
}

// ---- forward ------------------------------------------------------------------------------------------
// Tile: one sub-batch of 32 rows x 128 outputs, warp = 32 x 32, thread = 8 rows x 4 outputs, each with two sums (even and odd
// columns).  The (tile, k-tile) pairs of the whole problem form one sequence that is cut into gridDim.x equal ranges (StreamK);
// with `direct` the grid has one CTA per tile and the kernel takes the root itself.
constexpr int FWD_WARPS = 4, FWD_NT = FWD_WARPS * 32, FWD_BM = 32, FWD_BN = 32 * FWD_WARPS;

template <int MODE, int IP>
__global__ void __launch_bounds__(FWD_NT, 3) lp_power_fwd_kernel(const LpFwdParams p) {
    constexpr int BM = FWD_BM, BN = FWD_BN, NT = FWD_NT;
    extern __shared__ __align__(16) float smem[];
    float* xs = smem;                                       // [2][BM][LDS]
    float* ws = smem + 2 * BM * LDS;                        // [2][BN][LDS]
    const int tid = threadIdx.x, lane = tid & 31, wn = tid >> 5, tb = lane >> 3, tj = lane & 7;
    const int nk = (p.CI + BK - 1) / BK;
    const StreamK sk{(p.B + BM - 1) / BM, (p.CO + BN - 1) / BN, nk};
    long long u, u_end;
    sk.range(u, u_end);
    while (u < u_end) {
        const int tile = (int)(u / nk), kt_begin = (int)(u % nk);
        const int kt_end = (int)min((long long)nk, kt_begin + (u_end - u));
        const int m0 = (tile / sk.tiles_n) * BM, n0 = (tile % sk.tiles_n) * BN;
        GatherW<BN, NT> gw;
        const int* ci_s = nullptr;
        if (MODE == MODE_GATHER) {
            const int s = m0 / SNB_SUB_BATCH;
            ci_s = p.ci ? p.ci + (size_t)s * p.CI : nullptr;
            gw.init_rows(p.co ? p.co + (size_t)s * p.CO : nullptr, n0, p.CO, p.W_CI, tid);
            gw.fetch_cols(ci_s, kt_begin * BK, p.CI, tid);
        }
        auto stage = [&](int kt, int st) {
            float* xd = xs + st * BM * LDS;
            float* wd = ws + st * BN * LDS;
            if (MODE == MODE_VEC) {
                stage_dense_vec<BM, NT>(xd, p.x, m0, p.B, p.CI, kt * BK, p.CI, tid);
                stage_dense_vec<BN, NT>(wd, p.w, n0, p.CO, p.W_CI, kt * BK, p.CI, tid);
            } else if (MODE == MODE_SCALAR) {
                stage_dense_scalar<BM, NT>(xd, p.x, m0, p.B, p.CI, kt * BK, p.CI, tid);
                stage_dense_scalar<BN, NT>(wd, p.w, n0, p.CO, p.W_CI, kt * BK, p.CI, tid);
            } else {
                stage_dense_scalar<BM, NT>(xd, p.x, m0, p.B, p.CI, kt * BK, p.CI, tid);
                gw.stage(wd, p.w, tid);
            }
        };
        uint64_t acc[8][4];
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) acc[i][j] = 0ull;

        __syncthreads();                                    // everyone is done with the previous range's tiles
        stage(kt_begin, 0);
        cp_async_commit();
        if (MODE == MODE_GATHER && kt_begin + 1 < kt_end) gw.fetch_cols(ci_s, (kt_begin + 1) * BK, p.CI, tid);
        for (int kt = kt_begin; kt < kt_end; kt++) {
            const int cur = (kt - kt_begin) & 1;
            cp_async_wait<0>();
            __syncthreads();
            if (kt + 1 < kt_end) {
                stage(kt + 1, cur ^ 1);
                if (MODE == MODE_GATHER && kt + 2 < kt_end) gw.fetch_cols(ci_s, (kt + 2) * BK, p.CI, tid);
            }
            cp_async_commit();
            const float* xr = xs + cur * BM * LDS + tb * LDS;
            const float* wr = ws + cur * BN * LDS + (wn * 32 + tj) * LDS;
            // zero-filled padding (x = w = 0) contributes |0|^p = 0
            // (p = 3, unrolled by four: 512 x 2048 x 2048 256 -> 251 us, 16 x 5120 x 5120 106 -> 103, 512 x 3072 x 5120 908 -> 892)
            constexpr int UNROLL = IP == 3 ? 4 : 2;
#pragma unroll UNROLL
            for (int kk = 0; kk < BK; kk += 4) {
                ulonglong2 xf[8], wf[4];
#pragma unroll
                for (int j = 0; j < 4; j++) wf[j] = *reinterpret_cast<const ulonglong2*>(wr + j * 8 * LDS + kk);
#pragma unroll
                for (int i = 0; i < 8; i++) xf[i] = *reinterpret_cast<const ulonglong2*>(xr + i * 4 * LDS + kk);
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        acc[i][j] = add_pow<IP>(sub2(xf[i].x, wf[j].x), acc[i][j]);
                        acc[i][j] = add_pow<IP>(sub2(xf[i].y, wf[j].y), acc[i][j]);
                    }
            }
        }
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const int m = m0 + tb + 4 * i;
            if (m >= p.B) continue;
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int n = n0 + wn * 32 + tj + 8 * j;
                if (n >= p.CO) continue;
                float even, odd;
                unpack2(acc[i][j], even, odd);
                float* dst = p.y + (size_t)m * p.CO + n;
                if (p.direct) *dst = pow_pos(fmaxf(even + odd, FLT_MIN), 1.0f / p.p);
                else atomicAdd(dst, even + odd);
            }
        }
        u += kt_end - kt_begin;
    }
}

// ---- backward -----------------------------------------------------------------------------------------
// Work unit: one sub-batch of 32 rows x 128 compact columns x eight outputs j.  The units of the whole problem form one sequence
// (sub-batch, column tile, outputs) that is cut into gridDim.x equal ranges; a range that covers all outputs of a (sub-batch,
// column tile) pair stores its grad_x block, a partial one adds it with atomics into the zero-filled grad_x.
// Thread = one column, all 32 rows: x and grad_x stay in registers as 16 pairs of rows, the sum of a column over the rows needs
// no other lane, a weight is used by one thread only and comes straight from global memory (eight outputs ahead),
// and a warp's reduction into grad_w covers 32 neighbouring kept columns.  (g, y) of the next 32 outputs are copied to shared memory
// [j][row] meanwhile; each thread turns the elements that it copied into g / y^(p-1) before the barrier, so that a term is one
// subtract, the multiply chain and two fmas, and reads them back four rows at a time (all lanes the same words: broadcast).
// Four CTAs per SM, and three for p = 1, whose selected signs take 168 registers: with 128 it spills (67 x 1000 x 1000 37.0 -> 34.6 us, 16 x
// 5120 x 5120 227 -> 220, 512 x 2048 x 2048 505 -> 506).
constexpr int BWD_NT = 128, BWD_JT = 32, BWD_LD = 36, BWD_AHEAD = 8;

template <int IP>
__global__ void __launch_bounds__(BWD_NT, IP == 0 ? 3 : 4) lp_power_bwd_kernel(const LpBwdParams p) {
    constexpr int NT = BWD_NT, JT = BWD_JT, LD = BWD_LD, AHEAD = BWD_AHEAD;
    __shared__ __align__(16) float gt[2][JT * LD], yt[2][JT * LD];
    const int tid = threadIdx.x, lane = tid & 31;
    const int parts = (p.CO + AHEAD - 1) / AHEAD, col_tiles = (p.CI + NT - 1) / NT;
    const long long total = (long long)((p.B + SNB_SUB_BATCH - 1) / SNB_SUB_BATCH) * col_tiles * parts;
    long long u = total * blockIdx.x / gridDim.x;
    const long long u_end = total * (blockIdx.x + 1) / gridDim.x;
    while (u < u_end) {
        const int unit = (int)(u / parts), part0 = (int)(u % parts);
        const int part1 = (int)min((long long)parts, part0 + (u_end - u));
        const int j_begin = part0 * AHEAD, j_end = min(part1 * AHEAD, p.CO), t_begin = j_begin / JT, t_end = (j_end + JT - 1) / JT;
        const int s = unit / col_tiles, b0 = s * SNB_SUB_BATCH, c = (unit % col_tiles) * NT + tid;
        const int* co_s = p.co ? p.co + (size_t)s * p.CO : nullptr;
        const bool cok = c < p.CI;
        const int col = cok ? (p.ci ? p.ci[(size_t)s * p.CI + c] : c) : 0;
        const float* wcol = p.w + col;
        float* gwcol = p.gw + col;
        // Element r of this thread in the 32 x 32 (g, y) tiles: a warp takes eight neighbouring j of four rows, whole sectors in
        // memory and 32 different banks in shared memory.
        auto element = [&](int r, int& jj, int& bb) {
            const int e = tid + NT * r;
            jj = (e & 7) + 8 * ((e >> 5) & 3);
            bb = ((e >> 3) & 3) + 4 * (e >> 7);
        };
        auto stage = [&](int t, int st) {
#pragma unroll
            for (int r = 0; r < 1024 / NT; r++) {
                int jj, bb;
                element(r, jj, bb);
                const int b = b0 + bb, j = t * JT + jj;
                const bool ok = b < p.B && j < p.CO;
                const size_t o = ok ? (size_t)b * p.CO + j : 0;
                cp_async4(smem_u32(gt[st] + jj * LD + bb), p.g + o, ok ? 4 : 0);
                cp_async4(smem_u32(yt[st] + jj * LD + bb), p.y + o, ok ? 4 : 0);
            }
        };
        // row of W of output t * JT + lane; past the last output: the last one, whose weights are fetched and not used
        auto rows_of = [&](int t) {
            const int j = min(t * JT + lane, p.CO - 1);
            return co_s ? co_s[j] : j;
        };
        __syncthreads();                                    // everyone is done with the previous range's tiles
        stage(t_begin, 0);
        cp_async_commit();
        int row = rows_of(t_begin);
        float ahead[AHEAD];
#pragma unroll
        for (int k = 0; k < AHEAD; k++) {
            const int r = __shfl_sync(0xffffffffu, row, (j_begin + k) & 31);
            ahead[k] = cok ? wcol[(size_t)r * p.W_CI] : 0.f;
        }
        uint64_t xv[16], gx[16];
#pragma unroll
        for (int i = 0; i < 16; i++) {
            float v[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int b = b0 + 2 * i + h;
                v[h] = b < p.B && cok ? p.x[(size_t)b * p.CI + c] : 0.f;
            }
            xv[i] = pack2(v[0], v[1]);
            gx[i] = 0ull;
        }
        for (int t = t_begin; t < t_end; t++) {
            const int st = (t - t_begin) & 1;
            cp_async_wait<0>();
#pragma unroll
            for (int r = 0; r < 1024 / NT; r++) {
                int jj, bb;
                element(r, jj, bb);
                const float v = yt[st][jj * LD + bb];
                gt[st][jj * LD + bb] *= whole_pow<IP>(v > 0.f ? 1.0f / v : 0.f);
            }
            __syncthreads();                                // tile t is ready; everyone is done with tile t - 1
            if (t + 1 < t_end) stage(t + 1, st ^ 1);
            cp_async_commit();
            const int next_row = t + 1 < t_end ? rows_of(t + 1) : row;
            const int jn = min(JT, j_end - t * JT);
#pragma unroll 1
            for (int j0 = max(0, j_begin - t * JT); j0 < jn; j0 += AHEAD) {
                float w[AHEAD];
#pragma unroll
                for (int k = 0; k < AHEAD; k++) w[k] = ahead[k];
#pragma unroll
                for (int k = 0; k < AHEAD; k++) {
                    const int r = __shfl_sync(0xffffffffu, j0 + AHEAD < JT ? row : next_row, (j0 + AHEAD + k) & 31);
                    ahead[k] = cok ? wcol[(size_t)r * p.W_CI] : 0.f;
                }
#pragma unroll
                for (int k = 0; k < AHEAD; k++) {
                    const int jj = j0 + k;
                    if (jj >= jn) break;
                    const uint64_t ww = pack2(w[k], w[k]);
                    const ulonglong2* g4 = reinterpret_cast<const ulonglong2*>(gt[st] + jj * LD);
                    uint64_t sum[2] = {0ull, 0ull};
#pragma unroll
                    for (int i = 0; i < 8; i++) {
                        const ulonglong2 g = g4[i];
                        const uint64_t pa = signed_pow<IP>(sub2(xv[2 * i], ww)), pb = signed_pow<IP>(sub2(xv[2 * i + 1], ww));
                        gx[2 * i] = fma2(g.x, pa, gx[2 * i]);
                        sum[0] = fma2(g.x, pa, sum[0]);
                        gx[2 * i + 1] = fma2(g.y, pb, gx[2 * i + 1]);
                        sum[1] = fma2(g.y, pb, sum[1]);
                    }
                    const int r = __shfl_sync(0xffffffffu, row, jj);
                    if (p.gw && cok) {
                        float lo, hi;
                        unpack2(add2(sum[0], sum[1]), lo, hi);
                        atomicAdd(gwcol + (size_t)r * p.W_CI, -(lo + hi));
                    }
                }
            }
            row = next_row;
        }
        const bool whole = part0 == 0 && part1 == parts;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            float v[2];
            unpack2(gx[i], v[0], v[1]);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int b = b0 + 2 * i + h;
                if (b >= p.B || !cok) continue;
                float* dst = p.gx + (size_t)b * p.CI + c;
                if (whole) *dst = v[h];
                else atomicAdd(dst, v[h]);
            }
        }
        u += part1 - part0;
    }
}

// ---- host side ----------------------------------------------------------------------------------------

// CTAs of KERN that fit the device at once.
template <auto KERN, int NT, int BYTES>
cudaError_t resident(long long* slots) {
    static std::atomic<int> cached[64];
    int dev = 0;
    cudaGetDevice(&dev);
    std::atomic<int>& slot = cached[dev & 63];
    int per_sm = slot.load(std::memory_order_acquire);
    if (per_sm == 0) {
        cudaError_t e = BYTES > 48 * 1024 ? allow_smem<KERN, BYTES>() : cudaSuccess;
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KERN, NT, BYTES);
        if (e != cudaSuccess) return e;
        if (per_sm < 1) per_sm = 1;
        slot.store(per_sm, std::memory_order_release);
    }
    *slots = (long long)sm_count() * per_sm;
    return cudaSuccess;
}

// CTAs for `units` of work when `slots` fit at once.  Of the warps of a scheduler the oldest goes first, so CTAs with equal shares
// end one after the other and leave the last ones alone on their SM (512 x 2048 x 2048 backward: 3.0 of 4 warps per scheduler);
// several shares per slot keep the slots filled to the end (512 x 5120 x 5120, p = 8: backward 3.81 -> 3.56 ms, forward
// 1.67 -> 1.61).  Not below `least` units, where loading and storing a share's operands counts, and whole multiples only.
// Where that leaves one share per slot, p = 8, forward and backward, scalar kernels -> these: 33 x 784 x 500 13.1 -> 10.8 and 21.0 -> 19.7 us, 67 x 1000 x
// 1000 28.3 -> 21.6 and 46.9 -> 43.0, 200 x 1503 x 777 63 -> 51 and 102 -> 89, 16 x 5120 x 5120 117 -> 113 and 311 -> 268.  Slower: 128 x 5120 x 200 with lists
// of three quarters, forward 29.7 -> 30.9 (p = 3 26.7 -> 28.8): up to three steps of 128 outputs one after the other instead of two of 256.  Fewer shares, all
// equal, give 30.3 there and 30.6 instead of 32.5 at 200 x 1503 x 777 with lists, but 55 instead of 51 without.
unsigned shares(long long units, long long slots, int most, int least) {
    long long per_slot = units / (slots * least);
    per_slot = per_slot < 1 ? 1 : per_slot < most ? per_slot : most;
    const long long n = slots * per_slot;
    return (unsigned)(n < units ? n : units);
}

template <int MODE, int IP>
cudaError_t forward(LpFwdParams p, cudaStream_t st) {
    constexpr int SMEM = 2 * (FWD_BM + FWD_BN) * LDS * (int)sizeof(float);
    constexpr auto kern = lp_power_fwd_kernel<MODE, IP>;
    long long slots = 0;
    cudaError_t e = resident<kern, FWD_NT, SMEM>(&slots);
    if (e != cudaSuccess) return e;
    const long long tiles = (long long)((p.B + FWD_BM - 1) / FWD_BM) * ((p.CO + FWD_BN - 1) / FWD_BN);
    p.direct = tiles % slots == 0;                          // whole tiles per CTA fill the slots evenly anyway
    if (p.direct) {
        kern<<<(unsigned)tiles, FWD_NT, SMEM, st>>>(p);
        return launched();
    }
    const size_t n = (size_t)p.B * p.CO;
    if ((e = cudaMemsetAsync(p.y, 0, sizeof(float) * n, st)) != cudaSuccess) return e;
    const long long units = tiles * ((p.CI + BK - 1) / BK);
    kern<<<shares(units, slots, 4, 8), FWD_NT, SMEM, st>>>(p);
    if ((e = launched()) != cudaSuccess) return e;
    return lp_finish(p.y, nullptr, (long long)n, p.p, st);
}

template <int IP>
cudaError_t forward_mode(const LpFwdParams& p, cudaStream_t st) {
    if (p.ci || p.co) return forward<MODE_GATHER, IP>(p, st);
    const bool vec = (p.CI % 4 == 0) && (p.W_CI % 4 == 0) && aligned16(p.x) && aligned16(p.w);
    return vec ? forward<MODE_VEC, IP>(p, st) : forward<MODE_SCALAR, IP>(p, st);
}

template <int IP>
cudaError_t backward(const LpBwdParams& p, cudaStream_t st) {
    constexpr auto kern = lp_power_bwd_kernel<IP>;
    long long slots = 0;
    cudaError_t e = resident<kern, BWD_NT, 0>(&slots);
    if (e != cudaSuccess) return e;
    const long long total =
        (long long)((p.B + 31) / 32) * ((p.CI + BWD_NT - 1) / BWD_NT) * ((p.CO + BWD_AHEAD - 1) / BWD_AHEAD);
    if ((e = cudaMemsetAsync(p.gx, 0, sizeof(float) * (size_t)p.B * p.CI, st)) != cudaSuccess) return e;
    kern<<<shares(total, slots, 8, 32), BWD_NT, 0, st>>>(p);
    return launched();
}

}  // namespace

cudaError_t lp_power_forward(const LpFwdParams& p, cudaStream_t st) {
    switch ((int)p.p) {
        case 1: return forward_mode<1>(p, st);
        case 2: return forward_mode<2>(p, st);
        case 3: return forward_mode<3>(p, st);
        case 4: return forward_mode<4>(p, st);
        case 5: return forward_mode<5>(p, st);
        case 6: return forward_mode<6>(p, st);
        case 7: return forward_mode<7>(p, st);
        case 8: return forward_mode<8>(p, st);
    }
    return cudaErrorInvalidValue;
}

cudaError_t lp_power_backward(const LpBwdParams& p, cudaStream_t st) {
    switch ((int)p.pm1) {
        case 0: return backward<0>(p, st);
        case 1: return backward<1>(p, st);
        case 2: return backward<2>(p, st);
        case 3: return backward<3>(p, st);
        case 4: return backward<4>(p, st);
        case 5: return backward<5>(p, st);
        case 6: return backward<6>(p, st);
        case 7: return backward<7>(p, st);
    }
    return cudaErrorInvalidValue;
}

}  // namespace snb
