// Outputs whose list of columns did not do (included by prune.cu, after its list walks).
//
// Two cases.  A few outputs here and there (a mask that took all the columns of a threshold, a row of W unlike the
// others): prune_max / prune_sort record them, and they are evaluated one by one.  Or the data cannot be pruned at all (inputs
// spread as wide as the weights: every column can matter): prune_filter counts the rows of W whose list overflowed, and above
// a share of them (prune_gives_up) nothing is walked; the whole layer is evaluated by register tiles like those of inf_dist.cu,
// split over all CTAs along (tile, k-tile) pairs.  Columns come in the order of W, or, where lists are in another order (position,
// not column, decides their ties), in that of the list; a list that names a column twice is always evaluated like that.
#pragma once
#include <type_traits>

#include "tile.cuh"

namespace snb {
namespace {

constexpr int FIX_K = 32;           // columns per stage
constexpr int FIX_FEW = 4;
constexpr int REDO_THREADS = 128;   // prune_redo_max

// v[t], words of one output of sub-batch s, lane = row; all lanes of a warp.
template <int NX, bool TRACK>
__device__ __forceinline__ void store_output(const PruneProblem& p, int s, int n, const float (&v)[NX],
                                             const uint32_t (&word)[TRACK ? NX : 1]) {
    const int lane = threadIdx.x & 31, b = s * 32 + lane;
    if (p.yt || p.post) emit_chain<NX>(p, s, n, v, TRACK ? word[0] : 0u);
    if (p.part) {
        float sum = 0.f;
        for (int r = 0; r < min(32, p.B - s * 32); r++) sum += __shfl_sync(0xffffffffu, v[0], r);
        if (lane == 0) p.part[(size_t)s * p.CO + n] = sum;
    }
    if (b >= p.B) return;
    const size_t o = (size_t)b * p.CO + n;
    if (NX != 2 && p.y) p.y[o] = shifted<NX>(p, v[0], n);
    if (NX >= 2 && p.yl) p.yl[o] = shifted<NX>(p, v[NX - 2], n), p.yu[o] = shifted<NX>(p, v[NX - 1], n);
    if (TRACK && NX == 1 && p.pos) p.pos[o] = (int)word[0];
    if (TRACK && NX == 2) p.posl[o] = (int)word[0], p.posu[o] = (int)word[TRACK ? NX - 1 : 0];
}

// ---- a whole layer: maxima --------------------------------------------------------------------------
// Rows of W of a tile of 16 RPT outputs -> shared memory, by 128 threads: 16 bytes at a time along the row where alignment
// allows, else (and for columns picked through a list) 4.  Eight lanes per row; the rows of a warp's four groups lie two apart,
// which keeps the 4-byte writes free of bank conflicts.
template <int RPT>
struct DenseW {
    int rowoff[RPT];                // first element of the row in W, -1 past the last output
    int col[4];                     // columns of the next k-tile, -1 past the last (4-byte copies)
    __device__ __forceinline__ static int first_row() {
        const int w = threadIdx.x >> 5, g = (threadIdx.x >> 3) & 3;
        return 2 * g + (w & 1) + 8 * (w >> 1);
    }
    __device__ __forceinline__ void columns(const int* list, int k0, int K) {
#pragma unroll
        for (int m = 0; m < 4; m++) {
            const int k = k0 + (threadIdx.x & 7) + 8 * m;
            col[m] = k < K ? (list ? list[k] : k) : -1;
        }
    }
    __device__ __forceinline__ void copy16(float* dst, const float* w, int k0, int K) const {
        const int kc = (threadIdx.x & 7) * 4, r0 = first_row();
#pragma unroll
        for (int i = 0; i < RPT; i++) {
            const bool ok = rowoff[i] >= 0 && k0 + kc < K;
            cp_async16(smem_u32(dst + (r0 + 16 * i) * LDS + kc), ok ? w + rowoff[i] + k0 + kc : w, ok ? 16 : 0);
        }
    }
    __device__ __forceinline__ void copy4(float* dst, const float* w) const {
        const int r0 = first_row(), l8 = threadIdx.x & 7;
#pragma unroll
        for (int i = 0; i < RPT; i++)
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const bool ok = rowoff[i] >= 0 && col[m] >= 0;
                cp_async4(smem_u32(dst + (r0 + 16 * i) * LDS + l8 + 8 * m), ok ? w + rowoff[i] + col[m] : w, ok ? 4 : 0);
            }
    }
};

struct DenseLayer {
    int N, K, blocks;               // outputs to do per sub-batch, columns, blocks of 128 outputs
    bool gather, vec;
    __device__ __forceinline__ explicit DenseLayer(const PruneArgs& a) {
        gather = a.p.ci && a.counters[GENERAL] != 0u;
        N = a.p.out_list ? a.p.out_kept : a.p.CO;
        K = gather ? a.p.CI : a.p.W_CI;
        blocks = (N + 127) / 128;
        vec = !gather && (a.p.W_CI & 3) == 0 && (reinterpret_cast<uintptr_t>(a.p.w) & 15u) == 0;
    }
};
// A CTA's share of `tiles` x nk k-tiles: whole tiles, and of the rest an equal part.  Half of the CTAs do that part first: a tile
// is stored (a latency-bound time) by whoever completes it, and so the two CTAs of an SM do not store at the same time.
struct DenseWork {
    int nk, next, tiles;
    long long u0, u1;
    __device__ __forceinline__ DenseWork(int all, int nk_) : nk(nk_), next(blockIdx.x) {
        tiles = all / (int)gridDim.x * (int)gridDim.x;
        const long long rest = (long long)(all - tiles) * nk;
        u0 = rest * blockIdx.x / gridDim.x, u1 = rest * (blockIdx.x + 1) / gridDim.x;
    }
    __device__ __forceinline__ bool take(int& tile, int& ka, int& kb) {
        if (u0 < u1 && (next >= tiles || blockIdx.x >= gridDim.x / 2)) {
            tile = tiles + (int)(u0 / nk), ka = (int)(u0 % nk), kb = (int)min((long long)nk, ka + (u1 - u0));
            u0 += kb - ka;
            return true;
        }
        if (next >= tiles) return false;
        tile = next, ka = 0, kb = nk;
        next += gridDim.x;
        return true;
    }
};
// n-th output of sub-batch s, and its row of W
__device__ __forceinline__ int dense_output(const PruneProblem& p, int s, int n) {
    return p.out_list ? p.out_list[(size_t)s * p.out_kept + n] : n;
}
__device__ __forceinline__ int dense_row(const PruneProblem& p, int s, int out) {
    return p.co ? p.co[(size_t)s * p.CO + out] : out;
}

// Partial results of one tensor, [s][n][row]: maxima, or (value, chunk of 32 columns) with the lowest chunk of equal values.
template <bool TRACK>
__device__ __forceinline__ void merge(void* part, size_t at, float v, uint32_t chunk, bool whole) {
    if (TRACK) {
        const unsigned long long key = (unsigned long long)__float_as_uint(v) << 32 | (chunk == 0xffffu ? 0u : 0xffffffffu - chunk);
        unsigned long long* k = static_cast<unsigned long long*>(part) + at;
        if (whole) *k = key;
        else atomicMax(k, key);
    } else {
        float* k = static_cast<float*>(part) + at;
        if (whole) *k = v;
        else atomic_max_nonneg(k, v);
    }
}
template <bool TRACK>
__device__ __forceinline__ void* part_of(const PruneArgs& a, int t) {
    return a.partial + (size_t)t * a.S * a.p.CO * 32 * (TRACK ? 8 : 4);
}

// Which column of its chunk of 32 gave a row's value: place in the chunk | sign, for one output, lane = row.  low: the low
// halves of the keys (0: at the floor).
template <int NX>
struct Rescan {
    const float* xs[NX];            // rows of the sub-batch
    int stride, rows, last;         // last: the last column
    const int* list;                // columns of W, or null
    template <int T>
    __device__ __forceinline__ static bool holds(float x, float u, float w, float want, bool* negative) {
        if (NX == 1) {
            *negative = x - w < 0.f;
            return fabsf(x - w) == want;
        }
        const float t1 = w - x, t2 = u - w;
        *negative = !(t1 <= t2);
        return (T == 0 ? fmaxf(-t1, -t2) : fmaxf(t1, t2)) == want;
    }
    // four lanes per row, eight columns each by 16-byte loads: rows 8 e + lane / 4 of SETS e at a time
    template <int T, int SETS>
    __device__ __forceinline__ uint32_t vectors(const float* wr, float value, uint32_t low) const {
        const int lane = threadIdx.x & 31;
        uint32_t found = 0u;
#pragma unroll 1
        for (int e0 = 0; e0 < 4; e0 += SETS) {
            float4 x[SETS][NX][2], w[SETS][2];
            int at[SETS][2];
#pragma unroll
            for (int e = 0; e < SETS; e++) {
                const int r = 8 * (e0 + e) + (lane >> 2);
                const unsigned q = __shfl_sync(0xffffffffu, low, r);
                const int c = (q ? (int)(0xffffffffu - q) * 32 : 0) + 8 * (lane & 3);
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    at[e][h] = min(c + 4 * h, last - 3);             // past the end: the last columns once more
                    w[e][h] = *reinterpret_cast<const float4*>(wr + at[e][h]);
#pragma unroll
                    for (int u = 0; u < NX; u++)
                        x[e][u][h] = *reinterpret_cast<const float4*>(xs[u] + (size_t)min(r, rows - 1) * stride + at[e][h]);
                }
            }
#pragma unroll
            for (int e = 0; e < SETS; e++) {
                const float want = __shfl_sync(0xffffffffu, value, 8 * (e0 + e) + (lane >> 2));
                unsigned best = 0xffffffffu;                         // column << 1 | negative
#pragma unroll
                for (int k = 7; k >= 0; k--) {
                    auto of = [&](const float4& v) { return (k & 3) == 0 ? v.x : (k & 3) == 1 ? v.y : (k & 3) == 2 ? v.z : v.w; };
                    bool negative;
                    if (holds<T>(of(x[e][0][k >> 2]), of(x[e][NX - 1][k >> 2]), of(w[e][k >> 2]), want, &negative))
                        best = (unsigned)(at[e][k >> 2] + (k & 3)) << 1 | (negative ? 1u : 0u);
                }
                best = min(best, __shfl_xor_sync(0xffffffffu, best, 1));
                best = min(best, __shfl_xor_sync(0xffffffffu, best, 2));
                best = __shfl_sync(0xffffffffu, best, 4 * (lane & 7));
                if ((lane >> 3) == e0 + e) found = ((best >> 1) & 31u) | (best & 1u ? SNB_SIGN_BIT : 0u);
            }
        }
        return found;
    }
    // a lane per column, AHEAD rows at a time
    template <int T, int AHEAD>
    __device__ __forceinline__ uint32_t columns(const float* wr, float value, uint32_t low) const {
        const int lane = threadIdx.x & 31;
        uint32_t found = 0u;
#pragma unroll 1
        for (int r0 = 0; r0 < rows; r0 += AHEAD) {
            float x[AHEAD][NX], w[AHEAD];
#pragma unroll
            for (int e = 0; e < AHEAD; e++) {                        // past the end: the last column once more
                const unsigned q = __shfl_sync(0xffffffffu, low, r0 + e);
                const int c = min(q ? (int)(0xffffffffu - q) * 32 + lane : 0, last);
                w[e] = wr[list ? list[c] : c];
#pragma unroll
                for (int u = 0; u < NX; u++) x[e][u] = xs[u][(size_t)min(r0 + e, rows - 1) * stride + c];
            }
#pragma unroll
            for (int e = 0; e < AHEAD; e++) {
                bool negative;
                const bool hit = holds<T>(x[e][0], x[e][NX - 1], w[e], __shfl_sync(0xffffffffu, value, r0 + e), &negative);
                const unsigned hits = __ballot_sync(0xffffffffu, hit), signs = __ballot_sync(0xffffffffu, negative);
                const int k = (__ffs(hits) - 1) & 31;
                if (lane == r0 + e) found = (uint32_t)k | ((signs >> k) & 1u ? SNB_SIGN_BIT : 0u);
            }
        }
        return found;
    }
};

// Words and stores of 128 outputs whose partial results are complete, 32 at a time through shared memory `sm`.  Warp = eight of
// the 32 outputs, lane = row; the words of an output: the chunks of its rows are read once more, by four lanes per row where
// 16-byte loads are allowed, else by a lane per column.  Bound by the loads in flight (512 x 5120 x 5120: a lane per column
// 0.6 ms, four lanes per row 0.25 ms on top of 0.84).
template <int NX, bool TRACK>
__device__ __noinline__ void dense_emit(const PruneArgs& a, const DenseLayer& d, int s, int block, float* sm) {
    constexpr int SLOTS = 32 / (REDO_THREADS / 32), NW = TRACK ? NX : 0;
    const PruneProblem& p = a.p;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, C = p.W_CI, rows = min(32, p.B - s * 32);
    float(*tile)[32][33] = reinterpret_cast<float(*)[32][33]>(sm);           // [NX values, NW words][row][output]
    for (int base = block * 128; base < min(d.N, block * 128 + 128); base += 32) {
        __syncthreads();
#pragma unroll
        for (int t = 0; t < NX; t++)
#pragma unroll
            for (int i = 0; i < SLOTS; i++) {
                const int slot = warp * SLOTS + i;
                const size_t at = ((size_t)s * p.CO + min(base + slot, d.N - 1)) * 32 + lane;
                if (TRACK) {
                    const unsigned long long key = __ldcg(static_cast<const unsigned long long*>(part_of<TRACK>(a, t)) + at);
                    tile[t][lane][slot] = __uint_as_float((unsigned)(key >> 32));
                    tile[NX + t][lane][slot] = __uint_as_float((unsigned)key);
                } else {
                    tile[t][lane][slot] = __ldcg(static_cast<const float*>(part_of<TRACK>(a, t)) + at);
                }
            }
        if constexpr (TRACK) {
            const int* inv = p.ci && !d.gather ? a.inv + (size_t)s * C : nullptr;
            Rescan<NX> scan;
            scan.stride = d.gather ? p.CI : a.ldr, scan.rows = rows, scan.last = d.K - 1;
            scan.list = d.gather ? p.ci + (size_t)s * p.CI : nullptr;
#pragma unroll
            for (int u = 0; u < NX; u++)
                scan.xs[u] = d.gather ? p.x + (size_t)s * 32 * p.CI : a.xr + (size_t)(u * a.S + s) * 32 * a.ldr;
            auto words = [&](auto which, int slot) {
                constexpr int T = decltype(which)::value;
                const float* wr = p.w + (size_t)dense_row(p, s, dense_output(p, s, min(base + slot, d.N - 1))) * C;
                const float value = tile[T][lane][slot];
                const uint32_t low = __float_as_uint(tile[NX + T][lane][slot]);
                const uint32_t place = d.vec ? scan.template vectors<T, NX == 1 ? 4 : 2>(wr, value, low)
                                             : scan.template columns<T, 16>(wr, value, low);
                uint32_t word = NX == 1 ? first_kept(p, s) : T == 0 ? SNB_NO_GRAD_ID : 0u;       // at its floor
                if (low) {
                    const int col = min((int)(0xffffffffu - low) * 32 + (int)(place & 31u), d.K - 1);
                    word = (uint32_t)(inv ? inv[col] : col) | (place & SNB_SIGN_BIT);
                }
                tile[NX + T][lane][slot] = __uint_as_float(word);
            };
#pragma unroll 1
            for (int i = 0; i < SLOTS; i++) {
                words(std::integral_constant<int, 0>(), warp * SLOTS + i);
                if constexpr (NX == 2) words(std::integral_constant<int, 1>(), warp * SLOTS + i);
            }
        }
        __syncthreads();
        // rows: lane = output
        const int n = base + lane, out = dense_output(p, s, min(n, d.N - 1));
        for (int r = warp; r < rows; r += REDO_THREADS / 32) {
            if (n >= d.N) continue;
            const size_t o = (size_t)(s * 32 + r) * p.CO + out;
            if (NX != 2 && p.y) p.y[o] = shifted<NX>(p, tile[0][r][lane], out);
            if (NX >= 2 && p.yl) p.yl[o] = shifted<NX>(p, tile[NX - 2][r][lane], out), p.yu[o] = shifted<NX>(p, tile[NX - 1][r][lane], out);
            if (NW == 1 && p.pos) p.pos[o] = __float_as_int(tile[NX][r][lane]);
            if (NW == 2) p.posl[o] = __float_as_int(tile[NX][r][lane]), p.posu[o] = __float_as_int(tile[NX + NW - 1][r][lane]);
        }
        if (p.yt || p.post)                                  // lane = row
            for (int i = 0; i < SLOTS; i++) {
                const int slot = warp * SLOTS + i;
                if (base + slot >= d.N) break;
                float u[NX];
#pragma unroll
                for (int t = 0; t < NX; t++) u[t] = tile[t][lane][slot];
                emit_chain<NX>(p, s, dense_output(p, s, base + slot), u, NW ? __float_as_uint(tile[NW ? NX : 0][lane][slot]) : 0u);
            }
        if (p.part && warp == 0 && n < d.N) {
            float sum = 0.f;
            for (int r = 0; r < rows; r++) sum += tile[0][r][lane];
            p.part[(size_t)s * p.CO + out] = sum;
        }
    }
    __syncthreads();
}

// The CTA has merged `amount` k-tiles of `count` blocks from `first` on, in sub-batches s0 ..; whoever completes a block stores it.
template <int NX, bool TRACK>
__device__ __forceinline__ void dense_finish(const PruneArgs& a, const DenseLayer& d, int s0, int subs, int first, int count, int amount,
                                             float* sm) {
    __shared__ bool last;
    const unsigned need = (unsigned)((d.K + BK - 1) / BK) * (NX == 3 ? 2u : 1u);
    __threadfence();
    __syncthreads();
    for (int s = s0; s < s0 + subs; s++)
        for (int k = first; k < min(d.blocks, first + count); k++) {
            if (threadIdx.x == 0) {
                const unsigned before = atomicAdd(a.tile_done + (size_t)s * ((a.p.CO + 127) / 128) + k, (unsigned)amount);
                last = before + (unsigned)amount == need;
            }
            __syncthreads();
            if (last) {
                __threadfence();
                dense_emit<NX, TRACK>(a, d, s, k, sm);
            }
            __syncthreads();
        }
}

// max |x - w| : CTA tile of WM sub-batches x 256 / WM outputs, thread 8 x 8 (rows tb + 4 i, outputs tj + 8 j of its warp's
// 32 x 64).  Bound by the issue of subtract and max, two cycles per element.  Two sub-batches where all have the same
// outputs (fewer bytes of W per element), one where lists pick them.
template <int NX, bool TRACK, int WM>
__device__ void dense_point(const PruneArgs& a, const DenseLayer& d, float* smem) {
    const PruneProblem& p = a.p;
    constexpr int WN = 4 / WM, BM = 32 * WM, BN = 64 * WN, NT = REDO_THREADS;
    float* xs = smem;                                        // [2][BM][LDS]
    float* ws = smem + 2 * BM * LDS;                         // [2][BN][LDS]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wm = warp / WN, wn = warp % WN, tb = lane >> 3, tj = lane & 7;
    const int tiles_m = (a.S + WM - 1) / WM;
    const int nk = (d.K + BK - 1) / BK;
    DenseWork work(tiles_m * ((d.N + BN - 1) / BN), nk);
    for (int tile, ka, kb; work.take(tile, ka, kb);) {
        const int s0 = tile % tiles_m * WM, s = s0 + wm, n0 = tile / tiles_m * BN;
        const int* list = d.gather ? p.ci + (size_t)s0 * p.CI : nullptr;
        DenseW<BN / 16> rw;
#pragma unroll
        for (int i = 0; i < BN / 16; i++) {
            const int n = n0 + rw.first_row() + 16 * i;
            rw.rowoff[i] = n < d.N ? dense_row(p, s0, dense_output(p, s0, n)) * p.W_CI : -1;
        }
        auto stage = [&](int kt) {
            float *xd = xs + (kt & 1) * BM * LDS, *wd = ws + (kt & 1) * BN * LDS;
            if (d.gather) stage_dense_scalar<BM, NT>(xd, p.x, s0 * 32, p.B, p.CI, kt * BK, d.K, tid);
            else stage_dense_vec<BM, NT>(xd, a.xr, s0 * 32, a.S * 32, a.ldr, kt * BK, a.ldr, tid);
            if (d.vec) rw.copy16(wd, p.w, kt * BK, d.K);
            else rw.copy4(wd, p.w);
        };
        float acc[8][8], prev[TRACK ? 8 : 1][TRACK ? 8 : 1];
        uint32_t q[TRACK ? 8 : 1][TRACK ? 4 : 1];            // two 16-bit chunk ids per word, 0xffff = none
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) {
                acc[i][j] = SNB_EPS;
                if (TRACK) prev[TRACK ? i : 0][TRACK ? j : 0] = SNB_EPS, q[TRACK ? i : 0][TRACK ? j >> 1 : 0] = 0xffffffffu;
            }
        __syncthreads();                                     // the previous tile's readers are done with both stages
        if (!d.vec) rw.columns(list, ka * BK, d.K);
        stage(ka);
        cp_async_commit();
        for (int kt = ka; kt < kb; kt++) {
            if (!d.vec && kt + 1 < kb) rw.columns(list, (kt + 1) * BK, d.K);
            cp_async_wait<0>();
            __syncthreads();
            if (kt + 1 < kb) stage(kt + 1);
            cp_async_commit();
            const float* xr = xs + (kt & 1) * BM * LDS + (wm * 32 + tb) * LDS;
            const float* wr = ws + (kt & 1) * BN * LDS + (wn * 64 + tj) * LDS;
#pragma unroll 2
            for (int kk = 0; kk < BK / 4; kk++) {
                ulonglong2 xf[8], wf[8];
#pragma unroll
                for (int i = 0; i < 8; i++) xf[i] = *reinterpret_cast<const ulonglong2*>(xr + i * 4 * LDS + kk * 4);
#pragma unroll
                for (int j = 0; j < 8; j++) wf[j] = *reinterpret_cast<const ulonglong2*>(wr + j * 8 * LDS + kk * 4);
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        float u, v;
                        unpack2(sub2(xf[i].x, wf[j].x), u, v);
                        acc[i][j] = max3abs(acc[i][j], u, v);
                        unpack2(sub2(xf[i].y, wf[j].y), u, v);
                        acc[i][j] = max3abs(acc[i][j], u, v);
                    }
            }
            if (TRACK) {
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int j = 0; j < 8; j++) {
                        uint32_t& id = q[TRACK ? i : 0][TRACK ? j >> 1 : 0];
                        float& old = prev[TRACK ? i : 0][TRACK ? j : 0];
                        if (acc[i][j] > old) id = __byte_perm(id, (uint32_t)kt, (j & 1) ? 0x5410 : 0x3254);
                        old = acc[i][j];
                    }
            }
        }
        const bool whole = ka == 0 && kb == nk;
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const int n = n0 + wn * 64 + tj + 8 * j;
                const uint32_t id = q[TRACK ? i : 0][TRACK ? j >> 1 : 0];
                if (n < d.N && s < a.S)
                    merge<TRACK>(part_of<TRACK>(a, 0), ((size_t)s * p.CO + n) * 32 + tb + 4 * i, acc[i][j],
                                 (j & 1) ? id >> 16 : id & 0xffffu, whole);
            }
        dense_finish<NX, TRACK>(a, d, s0, min(WM, a.S - s0), n0 / 128, BN / 128, kb - ka, smem);
    }
}

// Both bounds of a box: CTA tile 32 rows x 128 outputs, thread 8 x 4.  Bound by the issue of two subtracts and two
// three-input maxima per element (5.8 cycles).
template <int NX, bool TRACK>
__device__ void dense_box(const PruneArgs& a, const DenseLayer& d, float* smem) {
    const PruneProblem& p = a.p;
    constexpr int BN = 128, NT = REDO_THREADS;
    float* ls = smem;                                        // [2][32][LDS]
    float* us = ls + 2 * 32 * LDS;                           // [2][32][LDS]
    float* ws = us + 2 * 32 * LDS;                           // [2][BN][LDS]
    const float* xl = a.xr + (size_t)(NX - 2) * a.S * 32 * a.ldr;
    const float* xu = a.xr + (size_t)(NX - 1) * a.S * 32 * a.ldr;
    const int tid = threadIdx.x, lane = tid & 31, wn = tid >> 5, tb = lane >> 3, tj = lane & 7;
    const int nk = (d.K + BK - 1) / BK;
    DenseWork work(a.S * ((d.N + BN - 1) / BN), nk);
    for (int tile, ka, kb; work.take(tile, ka, kb);) {
        const int s = tile % a.S, n0 = tile / a.S * BN;
        DenseW<BN / 16> rw;
#pragma unroll
        for (int i = 0; i < BN / 16; i++) {
            const int n = n0 + rw.first_row() + 16 * i;
            rw.rowoff[i] = n < d.N ? dense_row(p, s, dense_output(p, s, n)) * p.W_CI : -1;
        }
        auto stage = [&](int kt) {
            stage_dense_vec<32, NT>(ls + (kt & 1) * 32 * LDS, xl, s * 32, a.S * 32, a.ldr, kt * BK, a.ldr, tid);
            stage_dense_vec<32, NT>(us + (kt & 1) * 32 * LDS, xu, s * 32, a.S * 32, a.ldr, kt * BK, a.ldr, tid);
            float* wd = ws + (kt & 1) * BN * LDS;
            if (d.vec) {
                rw.copy16(wd, p.w, kt * BK, d.K);
            } else {
                rw.columns(nullptr, kt * BK, d.K);
                rw.copy4(wd, p.w);
            }
        };
        float lo[8][4], hi[8][4], pl[TRACK ? 8 : 1][TRACK ? 4 : 1], ph[TRACK ? 8 : 1][TRACK ? 4 : 1];
        uint32_t q[TRACK ? 8 : 1][TRACK ? 4 : 1];            // chunk ids: lower bound in the low half, upper in the high half
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                lo[i][j] = hi[i][j] = SNB_EPS;
                if (TRACK) {
                    pl[TRACK ? i : 0][TRACK ? j : 0] = ph[TRACK ? i : 0][TRACK ? j : 0] = SNB_EPS;
                    q[TRACK ? i : 0][TRACK ? j : 0] = 0xffffffffu;
                }
            }
        __syncthreads();
        stage(ka);
        cp_async_commit();
        for (int kt = ka; kt < kb; kt++) {
            cp_async_wait<0>();
            __syncthreads();
            if (kt + 1 < kb) stage(kt + 1);
            cp_async_commit();
            const float* lr = ls + (kt & 1) * 32 * LDS + tb * LDS;
            const float* ur = us + (kt & 1) * 32 * LDS + tb * LDS;
            const float* wr = ws + (kt & 1) * BN * LDS + (wn * 32 + tj) * LDS;
#pragma unroll 1
            for (int kk = 0; kk < BK / 4; kk++) {
                ulonglong2 wf[4];
#pragma unroll
                for (int j = 0; j < 4; j++) wf[j] = *reinterpret_cast<const ulonglong2*>(wr + j * 8 * LDS + kk * 4);
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    const ulonglong2 lf = *reinterpret_cast<const ulonglong2*>(lr + i * 4 * LDS + kk * 4);
                    const ulonglong2 uf = *reinterpret_cast<const ulonglong2*>(ur + i * 4 * LDS + kk * 4);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        float e1, e2, f1, f2;
                        unpack2(sub2(wf[j].x, lf.x), e1, f1);
                        unpack2(sub2(uf.x, wf[j].x), e2, f2);
                        hi[i][j] = max3(max3(hi[i][j], e1, e2), f1, f2);
                        lo[i][j] = max3(max3(lo[i][j], -e1, -e2), -f1, -f2);
                        unpack2(sub2(wf[j].y, lf.y), e1, f1);
                        unpack2(sub2(uf.y, wf[j].y), e2, f2);
                        hi[i][j] = max3(max3(hi[i][j], e1, e2), f1, f2);
                        lo[i][j] = max3(max3(lo[i][j], -e1, -e2), -f1, -f2);
                    }
                }
            }
            if (TRACK) {
#pragma unroll
                for (int i = 0; i < 8; i++)
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        uint32_t& id = q[TRACK ? i : 0][TRACK ? j : 0];
                        float &ol = pl[TRACK ? i : 0][TRACK ? j : 0], &oh = ph[TRACK ? i : 0][TRACK ? j : 0];
                        if (lo[i][j] > ol) id = __byte_perm(id, (uint32_t)kt, 0x3254);
                        if (hi[i][j] > oh) id = __byte_perm(id, (uint32_t)kt, 0x5410);
                        ol = lo[i][j], oh = hi[i][j];
                    }
            }
        }
        const bool whole = ka == 0 && kb == nk;
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const int n = n0 + wn * 32 + tj + 8 * j;
                if (n >= d.N) continue;
                const size_t at = ((size_t)s * p.CO + n) * 32 + tb + 4 * i;
                const uint32_t id = q[TRACK ? i : 0][TRACK ? j : 0];
                merge<TRACK>(part_of<TRACK>(a, NX - 2), at, lo[i][j], id & 0xffffu, whole);
                merge<TRACK>(part_of<TRACK>(a, NX - 1), at, hi[i][j], id >> 16, whole);
            }
        dense_finish<NX, TRACK>(a, d, s, 1, n0 / 128, 1, kb - ka, smem);
    }
}

// ---- a few outputs: maxima ---------------------------------------------------------------------------
template <int NX, int NT>
__device__ __forceinline__ void fix_stage(const float* xt_s, float* sm, int k0, int C) {
    const int n = min(FIX_K, C - k0) * NX * 8;               // 16-byte pieces; the columns of a sub-batch are contiguous
    const float* src = xt_s + (size_t)k0 * NX * 32;
    for (int k = threadIdx.x; k < n; k += NT) cp_async16(smem_u32(sm + k * 4), src + k * 4, 16);
}

template <int NX, bool TRACK>
constexpr int redo_max_smem() {
    const int point = 2 * (32 + 256) * LDS, box = 2 * (64 + 128) * LDS, few = 2 * FIX_K * NX * 32;
    const int tiles = NX == 1 ? point : NX == 2 ? box : (point > box ? point : box);
    return (tiles > few ? tiles : few) * (int)sizeof(float);
}

// Persistent CTAs over the recorded units (32 outputs of one sub-batch, a mask of those to redo).  A few outputs of a
// unit: the warps share the columns of one output.  Many: warp = four outputs side by side over all columns, xt staged in
// shared memory, W read along rows by uniform 16-byte loads.
// LEAVE: a layer that would be evaluated as a whole is left to the caller.  A form of its own, as asking for it in the other's way cost the tiles 4 %
// (values of 512 x 5120 x 5120 that cannot be pruned 930 -> 966 us).
template <int NX, bool TRACK, bool LEAVE = false>
__global__ void __launch_bounds__(REDO_THREADS, 2) prune_redo_max(const __grid_constant__ PruneArgs a) {
    constexpr int WARPS = REDO_THREADS / 32;
    extern __shared__ __align__(16) float redo_smem[];
    after_previous();
    let_next();
    if (dense_mode(a)) {
        if constexpr (!LEAVE) {
            const DenseLayer d(a);
            if constexpr (NX != 2) {
                if (a.p.co || a.p.ci || a.p.out_list || a.S == 1) dense_point<NX, TRACK, 1>(a, d, redo_smem);
                else dense_point<NX, TRACK, 2>(a, d, redo_smem);
            }
            if constexpr (NX >= 2) dense_box<NX, TRACK>(a, d, redo_smem);
        }
        return;
    }
    const PruneProblem& p = a.p;
    const int count = (int)a.counters[FAILED];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, C = p.W_CI;
    float* const sm = redo_smem;                             // [2][FIX_K * NX * 32]
    constexpr int STAGE = FIX_K * NX * 32;
    for (int unit = blockIdx.x; unit < count; unit += gridDim.x) {
        const int4 f = a.fail[unit];
        const int s = f.x, n0 = f.y;
        const unsigned mask = (unsigned)f.z;
        const float* xs = a.xt + (size_t)s * C * NX * 32;
        const int* inv = p.ci ? a.inv + (size_t)s * C : nullptr;
        const uint32_t floor_word = first_kept(p, s);
        if (__popc(mask) <= FIX_FEW) {
            unsigned todo = mask;
            while (todo) {
                const int n = n0 + __ffs(todo) - 1;
                todo &= todo - 1;
                const float* wr = p.w + (size_t)dense_row(p, s, n) * C;
                MaxState<NX, TRACK> st;
                st.init(floor_word);
                for (int c0 = warp * 8; c0 < C; c0 += WARPS * 8) {
                    float v[8][NX], w[8];
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        const int c = min(c0 + e, C - 1);            // a repeated column changes nothing
                        w[e] = wr[c];
#pragma unroll
                        for (int t = 0; t < NX; t++) v[e][t] = xs[((size_t)c * NX + t) * 32 + lane];
                    }
#pragma unroll
                    for (int e = 0; e < 8; e++) {
                        const int c = min(c0 + e, C - 1);
                        st.add(v[e], w[e], TRACK ? (uint32_t)(inv ? inv[c] : c) : 0u);
                    }
                }
                constexpr int PER = (TRACK ? 2 : 1) * NX;            // partial results: [warps][NX (+ NX words)][32]
                static_assert(WARPS * PER * 32 <= 2 * STAGE, "partial results fit the stages");
                __syncthreads();
#pragma unroll
                for (int t = 0; t < NX; t++) {
                    sm[(warp * PER + t) * 32 + lane] = st.acc[t];
                    if (TRACK) sm[(warp * PER + NX + t) * 32 + lane] = __uint_as_float(st.word[TRACK ? t : 0]);
                }
                __syncthreads();
                if (warp == 0) {
                    for (int k = 1; k < WARPS; k++)
#pragma unroll
                        for (int t = 0; t < NX; t++) {
                            const float v = sm[(k * PER + t) * 32 + lane];
                            if (TRACK) {
                                const uint32_t wd = __float_as_uint(sm[(k * PER + NX + t) * 32 + lane]);
                                if (wd != SNB_NO_GRAD_ID)
                                    take_word(v, wd & ~SNB_SIGN_BIT, (wd & SNB_SIGN_BIT) != 0, st.acc[t], st.word[TRACK ? t : 0]);
                            } else {
                                st.acc[t] = fmaxf(st.acc[t], v);
                            }
                        }
                    store_output<NX, TRACK>(p, s, n, st.acc, st.word);
                }
            }
            __syncthreads();
            continue;
        }
        const bool vec = (C % 4 == 0) && ((reinterpret_cast<uintptr_t>(p.w) & 15u) == 0);
        for (int g = warp * 4; g < 32; g += WARPS * 4) {     // all warps make the same number of rounds
            MaxState<NX, TRACK> st[4];
            const float* wr[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                wr[i] = p.w + (size_t)dense_row(p, s, min(n0 + g + i, p.CO - 1)) * C;
                st[i].init(floor_word);
            }
            __syncthreads();
            fix_stage<NX, REDO_THREADS>(xs, sm, 0, C);
            cp_async_commit();
            for (int k0 = 0, cur = 0; k0 < C; k0 += FIX_K, cur ^= 1) {
                cp_async_wait<0>();
                __syncthreads();
                if (k0 + FIX_K < C) fix_stage<NX, REDO_THREADS>(xs, sm + (cur ^ 1) * STAGE, k0 + FIX_K, C);
                cp_async_commit();
                const int kn = min(FIX_K, C - k0);
                for (int k = 0; k < kn; k += 4) {
                    float w[4][4];
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        if (vec) {
                            const float4 q = __ldg(reinterpret_cast<const float4*>(wr[i] + k0 + k));
                            w[i][0] = q.x; w[i][1] = q.y; w[i][2] = q.z; w[i][3] = q.w;
                        } else {
#pragma unroll
                            for (int e = 0; e < 4; e++) w[i][e] = __ldg(wr[i] + min(k0 + k + e, C - 1));
                        }
                    }
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        if (k + e >= kn) break;
                        float v[NX];
#pragma unroll
                        for (int t = 0; t < NX; t++) v[t] = sm[cur * STAGE + ((k + e) * NX + t) * 32 + lane];
                        const uint32_t idx = TRACK ? (uint32_t)(inv ? inv[k0 + k + e] : k0 + k + e) : 0u;
#pragma unroll
                        for (int i = 0; i < 4; i++) st[i].add(v, w[i][e], idx);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++)
                if ((mask >> (g + i)) & 1u) store_output<NX, TRACK>(p, s, n0 + g + i, st[i].acc, st[i].word);
        }
        __syncthreads();
    }
}

// ---- sort neurons ------------------------------------------------------------------------------------
// A whole layer: unit = 32 rows x 32 outputs, thread 2 x 2 (rows ty + 16 i, outputs tx + 16 j) with its lists in registers.
// Bound by the insertion chains.  Values of the point first, then of the box.
template <int NT>
__device__ __forceinline__ void sort_stage(const PruneArgs& a, float* dst, int s, int t, int kt) {
    stage_dense_vec<32, NT>(dst, a.xr + (size_t)t * a.S * 32 * a.ldr, s * 32, a.S * 32, a.ldr, kt * BK, a.ldr, threadIdx.x);
}

// body(x of two rows [, u], w of two outputs) for every column; rows of xr in tensor t0 (and t0 + 1).  Past the last column the
// operands are NaN or all zero: neither enters a list.
template <bool BOX, typename F>
__device__ __forceinline__ void sort_sweep(const PruneArgs& a, float* sm, int s, int n0, int t0, F&& body) {
    constexpr int NT = 256, TILE = 2 * 32 * LDS;
    const PruneProblem& p = a.p;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, C = p.W_CI, nk = (C + BK - 1) / BK;
    const bool vec = (C & 3) == 0 && (reinterpret_cast<uintptr_t>(p.w) & 15u) == 0;
    auto stage = [&](int kt) {
        const int at = (kt & 1) * 32 * LDS;
        sort_stage<NT>(a, sm + at, s, t0, kt);
        if (BOX) sort_stage<NT>(a, sm + TILE + at, s, t0 + 1, kt);
        if (vec) stage_dense_vec<32, NT>(sm + 2 * TILE + at, p.w, n0, p.CO, C, kt * BK, C, tid);
        else stage_dense_scalar<32, NT>(sm + 2 * TILE + at, p.w, n0, p.CO, C, kt * BK, C, tid);
    };
    __syncthreads();
    stage(0);
    cp_async_commit();
    for (int kt = 0; kt < nk; kt++) {
        cp_async_wait<0>();
        __syncthreads();
        if (kt + 1 < nk) stage(kt + 1);
        cp_async_commit();
        const float* xr = sm + (kt & 1) * 32 * LDS + ty * LDS;
        const float* wr = sm + 2 * TILE + (kt & 1) * 32 * LDS + tx * LDS;
#pragma unroll 1
        for (int k = 0; k < BK; k++) {
            const float x[2] = {xr[k], xr[16 * LDS + k]}, w[2] = {wr[k], wr[16 * LDS + k]};
            const float u[2] = {BOX ? xr[TILE + k] : 0.f, BOX ? xr[TILE + 16 * LDS + k] : 0.f};
            body(x, u, w);
        }
    }
}
// The insertion of TopList::add without its second vote: the columns come in no order, so values land all over the list.
template <int KMAX>
__device__ __forceinline__ void add_any(TopList<KMAX>& top, float d) {
    if (!__any_sync(0xffffffffu, d > top.v[0])) return;
    d = fmaxf(d, 0.f);                                       // a NaN must not move the list
#pragma unroll
    for (int k = 0; k < KMAX - 1; k++) top.v[k] = fmaxf(top.v[k], fminf(top.v[k + 1], d));
    top.v[KMAX - 1] = fmaxf(top.v[KMAX - 1], d);
}

constexpr int SORT_STAGES = 3 * 2 * 32 * LDS;                // floats: two stages of x (or l), u, W

template <int NX, int KMAX>
__device__ void dense_sort(const PruneArgs& a, float* sm) {
    const PruneProblem& p = a.p;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, K = p.K;
    static_assert(NX * 32 * 33 <= SORT_STAGES, "results fit the stages");
    float(*tile)[32][33] = reinterpret_cast<float(*)[32][33]>(sm);
    const int tiles_n = (p.CO + 31) / 32;
    for (int unit = blockIdx.x; unit < a.S * tiles_n; unit += gridDim.x) {
        const int s = unit % a.S, n0 = unit / a.S * 32;
        float result[NX][4];                                 // pair i: row ty + 16 (i / 2), output tx + 16 (i % 2)
        if constexpr (NX != 2) {
            TopList<KMAX> top[4];
#pragma unroll
            for (int i = 0; i < 4; i++) top[i].init();
            sort_sweep<false>(a, sm, s, n0, 0, [&](const float(&x)[2], const float(&)[2], const float(&w)[2]) {
#pragma unroll
                for (int i = 0; i < 4; i++) add_any(top[i], fabsf(x[i >> 1] - w[i & 1]));
            });
#pragma unroll
            for (int i = 0; i < 4; i++) result[0][i] = top[i].combine(K, p.q, SNB_EPS);
        }
        if constexpr (NX >= 2) {
            TopList<KMAX> low[4], high[4];
#pragma unroll
            for (int i = 0; i < 4; i++) low[i].init(), high[i].init();
            sort_sweep<true>(a, sm, s, n0, NX - 2, [&](const float(&x)[2], const float(&u)[2], const float(&w)[2]) {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const float t1 = w[i & 1] - x[i >> 1], t2 = u[i >> 1] - w[i & 1];
                    add_any(low[i], fmaxf(-t1, -t2));
                    add_any(high[i], fmaxf(t1, t2));
                }
            });
#pragma unroll
            for (int i = 0; i < 4; i++) {
                result[NX - 2][i] = low[i].combine(K, p.q, SNB_EPS);
                result[NX - 1][i] = high[i].combine(K, p.q, SNB_EPS);
            }
        }
        __syncthreads();
#pragma unroll
        for (int t = 0; t < NX; t++)
#pragma unroll
            for (int i = 0; i < 4; i++) tile[t][ty + 16 * (i >> 1)][tx + 16 * (i & 1)] = result[t][i];
        __syncthreads();
        emit_tile<NX, NX, 0>(p, tile, s, n0);
    }
}

template <int NX, int KMAX, bool POS>
__global__ void __launch_bounds__(256, KMAX > 10 ? 1 : (NX == 1 && !POS ? 4 : 2)) prune_redo_sort(const __grid_constant__ PruneArgs a) {
    __shared__ __align__(16) float sm[SORT_STAGES];
    after_previous();
    let_next();
    if (dense_mode(a)) {
        if constexpr (!POS) dense_sort<NX, KMAX>(a, sm);    // POS: sort_positions_if
        return;
    }
    constexpr int STAGE = FIX_K * NX * 32;
    static_assert(2 * STAGE <= SORT_STAGES, "two stages");
    const PruneProblem& p = a.p;
    const int count = (int)a.counters[FAILED];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, C = p.W_CI, K = p.K;
    for (int unit = blockIdx.x; unit < count; unit += gridDim.x) {
        const int4 f = a.fail[unit];
        const int s = f.x, n0 = f.y, b = s * 32 + lane;
        const unsigned mask = (unsigned)f.z;
        const float* xs = a.xt + (size_t)s * C * NX * 32;
        for (int i = 0; i < 4; i++) {
            const int slot = warp + 8 * i;                          // the CTA's warps do eight outputs at a time
            if (((mask >> (8 * i)) & 0xffu) == 0u) continue;
            const bool mine = (mask >> slot) & 1u;
            const int n = min(n0 + slot, p.CO - 1);
            const float* wr = p.w + (size_t)n * C;
            const size_t o = (size_t)b * p.CO + n;
            auto sweep = [&](auto&& body) {
                __syncthreads();
                fix_stage<NX, 256>(xs, sm, 0, C);
                cp_async_commit();
                for (int k0 = 0, cur = 0; k0 < C; k0 += FIX_K, cur ^= 1) {
                    cp_async_wait<0>();
                    __syncthreads();
                    if (k0 + FIX_K < C) fix_stage<NX, 256>(xs, sm + (cur ^ 1) * STAGE, k0 + FIX_K, C);
                    cp_async_commit();
                    if (!mine) continue;
                    const int kn = min(FIX_K, C - k0);
                    const float wl = lane < kn ? wr[k0 + lane] : 0.f;
                    for (int k = 0; k < kn; k++) {
                        float v[NX];
#pragma unroll
                        for (int t = 0; t < NX; t++) v[t] = sm[cur * STAGE + (k * NX + t) * 32 + lane];
                        body(v, __shfl_sync(0xffffffffu, wl, k), (uint32_t)(k0 + k));
                    }
                }
            };
            SortState<NX, KMAX> st;
            st.init();
            sweep([&](const float(&v)[NX], float w, uint32_t c) { st.add(v, w, c); });
            if (mine) {
                float v[NX];
#pragma unroll
                for (int t = 0; t < NX; t++) v[t] = st.result(t, K, p.q);
                if (p.yt) emit_chain<NX>(p, s, n, v, 0u);
                if (b < p.B) {
                    if (NX != 2 && p.y) p.y[o] = shifted<NX>(p, v[0], n);
                    if (NX >= 2 && p.yl) p.yl[o] = shifted<NX>(p, v[NX - 2], n), p.yu[o] = shifted<NX>(p, v[NX - 1], n);
                }
            }
            if constexpr (POS) {
                PosList<KMAX> pl;
                pl.init(st.top[0].kth(K));
                sweep([&](const float(&v)[NX], float w, uint32_t c) { pl.add(v[0] - w, c, K); });
                if (mine && b < p.B) {
#pragma unroll
                    for (int k = 0; k < KMAX; k++)
                        if (k < K) p.pos[((size_t)k * p.B + b) * p.CO + n] = (int)pl.word[KMAX - 1 - k];
                }
            }
        }
        __syncthreads();
    }
}

}  // namespace
}  // namespace snb
