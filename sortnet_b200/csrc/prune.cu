// Pruned evaluation of the max-type distance operators: see prune.cuh for the method.
//
// What bounds it: the one read of W (prune_filter, HBM).  For 512 x 5120 x 5120 a dense max-plus
// kernel issues 13.4 G subtract / max pairs; here about 40 columns per output row survive the
// filter and about 12 of them are looked at, 1/400 of the pairs.
#include "prune.cuh"

namespace snb {

namespace {

constexpr int PAD = 8;              // lists are padded to a multiple of this
constexpr int STEP = 4;             // list entries per bound ub
constexpr int MAX_COLUMNS = 12288;  // widest row the filter takes: 512 threads x 6 x 4
constexpr int BUCKETS = 32;
constexpr size_t MOST_SCRATCH = (size_t)4 << 30;   // with millions of outputs the lists would take more than W itself
constexpr int LONG_LIST = 512;       // most entries of a list

struct PruneArgs {
    PruneProblem p;
    int S, NX, m, lcap;
    unsigned* counters;             // [FAILED], [OVERFLOWED], [GENERAL]
    const unsigned* hi;             // order codes of max(x), max(-x) per column; 0 = no value
    const unsigned* nlo;
    const float* xt;                // [S][W_CI][NX][32]
    int* inv;                       // [S][W_CI] full column -> compact position, -1 where dropped (with ci)
    int* cnt;                       // [W_CO] list length, -1: no list
    float* tau;                     // [W_CO]
    float* ub;                      // [W_CO][lcap / STEP] largest U from this step of the list on
    int2* cand;                     // [W_CO][lcap] (column, bits of w)
    int4* fail;                     // units (sub-batch, first output, mask of outputs) left to prune_redo
    // used when the layer is evaluated as a whole (dense_mode)
    int ldr;                        // W_CI up to a multiple of 4
    float* xr;                      // [tensors][S][32][ldr] the rows of xt, NaN past the last column
    char* partial;                  // [results][S][CO][32] maxima, or keys (value, chunk of columns)
    unsigned* tile_done;            // [S][blocks of 128 outputs] k-tiles merged
};

__device__ __forceinline__ bool dense_mode(const PruneArgs& a) { return prune_left(a.counters, a.p.ci != nullptr, a.p.W_CO); }

// A load that stays where it is written.
__device__ __forceinline__ unsigned load_now(const unsigned* p) {
    unsigned v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}

// ---- transpose + column ranges ----------------------------------------------------------------
// CTA = 32 rows (one sub-batch) x 64 compact columns.  Bound by the traffic of x and xt and by launch latency.
template <int NX>
__global__ void __launch_bounds__(256) prune_prep(const PrunePrep p) {
    __shared__ float tile[NX][32][65];
    const int s = blockIdx.y, c0 = blockIdx.x * 64, tid = threadIdx.x;
    const float nan = __int_as_float(0x7fc00000);
    const int col = tid & 63, r0 = tid >> 6;
    const bool cok = c0 + col < p.CI;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int r = r0 + 4 * i, b = s * 32 + r;
        const bool ok = cok && b < p.B;
        const size_t o = (size_t)b * p.CI + c0 + col;
        float x = nan;
        if (NX != 2) tile[0][r][col] = x = ok ? p.x[o] : nan;
        if (NX >= 2) {
            float l = nan, u = nan;
            if (NX == 3 && p.box) {
                l = x == x ? fmaxf(x - p.eps, p.down) : x;
                u = x == x ? fminf(x + p.eps, p.up) : x;
            } else if (ok) {
                l = p.xl[o];
                u = p.xu[o];
            }
            if (l > u) l = u = (l + u) * 0.5f;               // inverted interval -> its midpoint
            tile[NX - 2][r][col] = l;
            tile[NX - 1][r][col] = u;
        }
    }
    __syncthreads();
    const int warp = tid >> 5, lane = tid & 31;
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int lc = warp + 8 * k;
        if (c0 + lc >= p.CI) break;
        int c = c0 + lc;
        if (p.ci) {
            const int* at = p.ci + (size_t)s * p.CI + c0 + lc;
            c = *at;
            if ((unsigned)c >= (unsigned)p.W_CI) {           // the list is the caller's; nothing is written for such an entry
                if (lane == 0) atomicOr(p.general, LIST_ORDER | LIST_TWICE);
                continue;
            }
            if (lane == 0 && c0 + lc + 1 < p.CI && at[1] <= c) atomicOr(p.general, LIST_ORDER);
        }
        unsigned hi = 0u, nlo = 0u;
#pragma unroll
        for (int t = 0; t < NX; t++) {
            const float v = tile[t][lane][lc];
            p.xt[(((size_t)s * p.W_CI + c) * NX + t) * 32 + lane] = v;
            hi = max(hi, order_code(v));
            nlo = max(nlo, order_code(-v));
        }
        hi = __reduce_max_sync(0xffffffffu, hi);
        nlo = __reduce_max_sync(0xffffffffu, nlo);
        if (lane == 0) {
            atomicMax(p.hi + c, hi);
            atomicMax(p.nlo + c, nlo);
            if (p.ci && atomicExch(p.inv + (size_t)s * p.W_CI + c, c0 + lc) != -1) atomicOr(p.general, LIST_ORDER | LIST_TWICE);
        }
    }
}

// ---- candidate lists --------------------------------------------------------------------------
// Named barriers: producers that only arrive and consumers that wait.
__device__ __forceinline__ void bar_sync(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int threads) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// Persistent CTA: FT filter threads + NB R ordering warps.  A thread owns NIT x 4 columns; it keeps their centre and
// radius in registers and copies its part of the next rows of W ahead with cp.async (its own shared memory: no barrier
// for the data).  Per step of R rows:
//   sweep 1   the largest |w - mid| - rad of every thread, and the warps' best of them;
//   the ordering warps make the threshold of each row of them, the m-th largest;
//   sweep 2   every column with |w - mid| + rad at or above it goes into the row's list;
// and the ordering warps sort the list.  Sweep 1 runs a step ahead of sweep 2, so that the filter warps need not wait for the threshold,
// and there are NB list buffers with R ordering warps each, which so have the time of NB steps.  Both sweeps read W from shared memory,
// HBM is read once.
// Three rows of stages leave 50 KB of L1 to the ordering warps, which look the exact ranges of their columns up there, and they are what
// the filter waits for where lists are long: 5120 x 5120 with lists of rank 10 (180 entries) and of rank 1 (35), cold, 45.4 -> 34.8 and 29.9 -> 29.4 us
// against sweeps behind a barrier each with two rows of stages twice over and two list buffers (217 KB); two buffers here 29 instead of 25
// within an attack step, five (one CTA per SM for their registers) 38; 12288 columns 99 -> 70 and 70 -> 58.  In a training pass of six layers 42 -> 35 us per layer.
// The warps' best for m > 1: four reductions over keys that hold the lane in their low bits, so that no vote is needed to take one out; the
// m-th of all by counting larger ones, eight 16-byte reads, instead of 32 shuffles.  A lane with hits takes their places with an atomic of its own: few
// lanes have any (by a scan over the warp 27.0 instead of 25.3 us).
// The centre form is rounded, so the sweep tests against just below thr (1 - 2^-19): with rad rounded up, a column it
// leaves out has |fl(x - w)| <= thr (1 - 2^-19)(1 + 2^-21) < thr = tau for every row.
template <int R, int NIT, int FT, int STAGES, int NB, bool VEC, int FIT = FT == 512 ? 1 : NIT >= 4 ? 2 : 3>
__global__ void __launch_bounds__(FT + 32 * NB * R, FIT) prune_filter(const PruneArgs a) {
    constexpr int WARPS = FT / 32, TOP = 32 / WARPS, ALL = FT + 32 * R;   // ALL: the filter and one buffer's ordering warps
    enum { BAR_TOP = 1, BAR_THR = BAR_TOP + NB, BAR_FULL = BAR_THR + NB };
    static_assert(BAR_FULL + NB <= 16 && STAGES >= 3, "");
    extern __shared__ __align__(16) unsigned char dyn[];
    const PruneProblem& p = a.p;
    const int C = p.W_CI, lcap = a.lcap, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float4* stage = reinterpret_cast<float4*>(dyn);                                  // [STAGES][R][NIT][FT]
    int2* lists = reinterpret_cast<int2*>(stage + STAGES * R * NIT * FT);            // [NB][R][lcap] (column, w)
    float* bounds = reinterpret_cast<float*>(lists + NB * R * lcap);                 // [NB R][lcap] U, then [lcap / STEP] of steps
    __shared__ __align__(16) unsigned top[NB][R][32];
    __shared__ float thr[NB][R];
    __shared__ int n_found[NB][R];
    __shared__ int hist[NB * R][BUCKETS];
    const int steps = (p.W_CO + R - 1) / R;
    const float nan = __int_as_float(0x7fc00000);
    if (tid < NB * R) n_found[tid / R][tid % R] = 0;
    // In a whole-net call the kernel before this one has nothing to do with W, whose first rows are fetched while it ends.  Nor may any
    // kernel that still runs then: what wrote W before the call has ended, as the call's prune_prep is an ordinary launch.
    const bool ahead = p.xt && !p.ci;
    if (!ahead) after_previous();
    if (p.ci && (a.counters[GENERAL] & LIST_TWICE)) return;  // no list will be walked
    __syncthreads();

    if (tid < FT) {
        auto column = [&](int it, int e) { return it * 4 * FT + (VEC ? tid * 4 + e : e * FT + tid); };
        auto fetch = [&](int step, int st) {
#pragma unroll
            for (int r = 0; r < R; r++) {
                const int j = step * R + r;
#pragma unroll
                for (int it = 0; it < NIT; it++) {
                    float4* dst = stage + ((st * R + r) * NIT + it) * FT + tid;
                    if (VEC) {
                        const int c = column(it, 0);
                        const bool ok = j < p.W_CO && c < C;
                        cp_async16(smem_u32(dst), ok ? p.w + (size_t)j * C + c : p.w, ok ? 16 : 0);
                    } else {
#pragma unroll
                        for (int e = 0; e < 4; e++) {
                            const int c = column(it, e);
                            const bool ok = j < p.W_CO && c < C;
                            cp_async4(smem_u32(reinterpret_cast<float*>(dst) + e), ok ? p.w + (size_t)j * C + c : p.w, ok ? 4 : 0);
                        }
                    }
                }
            }
        };
#pragma unroll
        for (int k = 0; k < STAGES; k++) {
            const int step = blockIdx.x + k * gridDim.x;
            if (step < steps) fetch(step, k);
            cp_async_commit();
        }
        if (ahead) after_previous();
        let_next();
        float mid[NIT][4], rad[NIT][4];
#pragma unroll
        for (int it = 0; it < NIT; it++)
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int c = column(it, e);
                const float hi = decode(c < C ? a.hi[c] : 0u), lo = -decode(c < C ? a.nlo[c] : 0u);
                if (isinf(hi) || isinf(lo)) {
                    mid[it][e] = 0.f;
                    rad[it][e] = INFINITY;                   // always a candidate
                } else {
                    mid[it][e] = 0.5f * lo + 0.5f * hi;      // NaN without any value: never a candidate
                    rad[it][e] = fmaxf(hi - mid[it][e], mid[it][e] - lo) * (1.0f + 0x1p-22f);
                }
            }
        int st = 0, before = 0, buf = 0, last = 0;           // stage and list buffer of this step and of the one before
        for (int step = blockIdx.x;; step += gridDim.x) {
            const bool first = step == (int)blockIdx.x, more = step < steps;
            if (more) {
                if (first) cp_async_wait<STAGES - 1>();
                else cp_async_wait<STAGES - 2>();
                const float4* rows = stage + st * R * NIT * FT + tid;
#pragma unroll
                for (int r = 0; r < R; r++) {
                    float best = 0.f;
#pragma unroll
                    for (int it = 0; it < NIT; it++) {
                        const float4 w = rows[(r * NIT + it) * FT];
                        best = max3(best, fabsf(w.x - mid[it][0]) - rad[it][0], fabsf(w.y - mid[it][1]) - rad[it][1]);
                        best = max3(best, fabsf(w.z - mid[it][2]) - rad[it][2], fabsf(w.w - mid[it][3]) - rad[it][3]);
                    }
                    unsigned mine = __float_as_uint(best);   // non-negative: integer order = float order
                    if (a.m == 1) {
                        mine = __reduce_max_sync(0xffffffffu, mine);
                        if (lane < TOP) top[buf][r][warp * TOP + lane] = lane == 0 ? mine : 0u;
                    } else {
                        mine = (mine & ~31u) | lane;         // no two alike: each round takes one out, and the bound moves by 2^-18 at most
                        unsigned kept = 0u;
#pragma unroll
                        for (int k = 0; k < TOP; k++) {
                            const unsigned mx = __reduce_max_sync(0xffffffffu, mine);
                            if (lane == k) kept = mx;
                            if (mine == mx) mine = 0u;
                        }
                        if (lane < TOP) top[buf][r][warp * TOP + lane] = kept & ~31u;
                    }
                }
                __syncwarp();                                // the barriers are for whole warps: here and below lanes come out of branches of their own
                bar_arrive(BAR_TOP + buf, ALL);
            }
            if (!first) {
                bar_sync(BAR_THR + last, ALL);               // the thresholds of the step before, whose list buffer is free again
                const float4* rows = stage + before * R * NIT * FT + tid;
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const float t = thr[last][r];
                    unsigned hit = 0u;                       // a bit per column, the last one lowest: the sign of t - U (none for NaN)
#pragma unroll
                    for (int it = 0; it < NIT; it++) {
                        const float4 w = rows[(r * NIT + it) * FT];
                        hit = __funnelshift_l(__float_as_uint(t - (fabsf(w.x - mid[it][0]) + rad[it][0])), hit, 1);
                        hit = __funnelshift_l(__float_as_uint(t - (fabsf(w.y - mid[it][1]) + rad[it][1])), hit, 1);
                        hit = __funnelshift_l(__float_as_uint(t - (fabsf(w.z - mid[it][2]) + rad[it][2])), hit, 1);
                        hit = __funnelshift_l(__float_as_uint(t - (fabsf(w.w - mid[it][3]) + rad[it][3])), hit, 1);
                    }
                    if (!hit) continue;
                    int at = atomicAdd(&n_found[last][r], __popc(hit));
                    while (hit) {
                        const int k = 4 * NIT - __ffs(hit);
                        hit &= hit - 1;
                        if (at < lcap)
                            lists[(last * R + r) * lcap + at] =
                                make_int2(column(k >> 2, k & 3), reinterpret_cast<const int*>(rows + (r * NIT + (k >> 2)) * FT)[k & 3]);
                        at++;
                    }
                }
                __syncwarp();
                bar_arrive(BAR_FULL + last, ALL);
                const int next = step + (STAGES - 1) * (int)gridDim.x;
                if (next < steps) fetch(next, before);
                cp_async_commit();
            }
            if (!more) break;
            before = st, last = buf;
            st = st + 1 == STAGES ? 0 : st + 1;
            buf = buf + 1 == NB ? 0 : buf + 1;
        }
        cp_async_wait<0>();
        return;
    }

    // ordering warps: list r of every NB-th step, by U, largest first, in BUCKETS steps of U
    if (ahead) after_previous();
    let_next();
    const int o = warp - WARPS, r = o % R, buf = o / R;
    float* u_in = bounds + o * (lcap + lcap / STEP);
    unsigned* u_step = reinterpret_cast<unsigned*>(u_in + lcap);                     // largest U of each step of four
    const int2* c_in = lists + (buf * R + r) * lcap;
    for (int step = blockIdx.x + buf * (int)gridDim.x; step < steps; step += NB * (int)gridDim.x) {
        const int j = step * R + r;
        bar_sync(BAR_TOP + buf, ALL);
        unsigned kth = top[buf][r][lane];
        if (a.m == 1) {
            kth = __reduce_max_sync(0xffffffffu, kth);
        } else {
            const uint4* all = reinterpret_cast<const uint4*>(top[buf][r]);
            int above = 0;                                   // the m-th largest: the smallest that fewer than m are larger than
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const uint4 v = all[k];
                above += (v.x > kth) + (v.y > kth) + (v.z > kth) + (v.w > kth);
            }
            kth = __reduce_min_sync(0xffffffffu, above < a.m ? kth : 0xffffffffu);
        }
        const float t = __uint_as_float(kth) * (1.0f - 0x1p-21f);
        const int below = __float_as_int(t * (1.0f - 0x1p-19f));
        if (lane == 0) thr[buf][r] = __int_as_float(max(below - 1, 0));
        __syncwarp();
        bar_arrive(BAR_THR + buf, ALL);
        bar_sync(BAR_FULL + buf, ALL);
        const int n = n_found[buf][r];
        if (j < p.W_CO && n <= lcap) {
            float umax = 0.f;
            for (int k0 = 0; k0 < n; k0 += 128) {            // four entries per lane: their loads overlap
                int2 e[4];
                unsigned h[4], l[4];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int k = k0 + 32 * q + lane;
                    e[q] = k < n ? c_in[k] : make_int2(0, __float_as_int(nan));
                }
#pragma unroll
                for (int q = 0; q < 4; q++) h[q] = a.hi[e[q].x], l[q] = a.nlo[e[q].x];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    const int k = k0 + 32 * q + lane;
                    const float w = __int_as_float(e[q].y);
                    const float u = fmaxf(decode(h[q]) - w, w + decode(l[q]));     // exact: rounding is monotone
                    if (k < n) {
                        u_in[k] = u;
                        umax = fmaxf(umax, u);
                    }
                }
            }
            umax = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(umax)));
            const float scale = umax > t ? (BUCKETS - 0.01f) / (umax - t) : 0.f;
            auto bucket = [&](float u) { return min(BUCKETS - 1, max(0, (int)((umax - u) * scale))); };
            const int padded = (n + PAD - 1) / PAD * PAD;
            hist[o][lane] = 0;
            for (int k = lane; k < padded / STEP; k += 32) u_step[k] = 0u;
            __syncwarp();
            for (int k = lane; k < n; k += 32) atomicAdd(&hist[o][bucket(u_in[k])], 1);
            __syncwarp();
            {
                const int h = hist[o][lane];
                int incl = h;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int below = __shfl_up_sync(0xffffffffu, incl, d);
                    if (lane >= d) incl += below;
                }
                hist[o][lane] = incl - h;
            }
            __syncwarp();
            int2* c_out = a.cand + (size_t)j * lcap;
            for (int k = lane; k < n; k += 32) {
                const float u = u_in[k];
                const int at = atomicAdd(&hist[o][bucket(u)], 1);
                atomicMax(&u_step[at / STEP], __float_as_uint(u));
                c_out[at] = c_in[k];
            }
            if (n + lane < padded) c_out[n + lane] = make_int2(c_in[0].x, __float_as_int(nan));   // w = NaN: changes nothing
            __syncwarp();
            // ub[b]: no entry of step b or later has a larger U
            const int nb = padded / STEP;
            float tail = 0.f;
            for (int base = (nb - 1) / 32 * 32; base >= 0; base -= 32) {
                const int b = base + lane;
                float v = b < nb ? __uint_as_float(u_step[b]) : 0.f;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const float after = __shfl_down_sync(0xffffffffu, v, d);
                    if (lane + d < 32) v = fmaxf(v, after);
                }
                v = fmaxf(v, tail);
                if (b < nb) a.ub[(size_t)j * (lcap / STEP) + b] = v;
                tail = __shfl_sync(0xffffffffu, v, 0);
            }
        }
        __syncwarp();
        if (lane == 0) {
            if (j < p.W_CO) {
                a.cnt[j] = n <= lcap ? n : -1;
                a.tau[j] = t;
                if (n > lcap) atomicAdd(a.counters + OVERFLOWED, 1u);
            }
            n_found[buf][r] = 0;
        }
        __syncwarp();
    }
}

// ---- one column against the 32 rows of a warp ----------------------------------------------------
// Argmax word of the reference: position | sign bit of (x - w); the lowest position wins a tie, whatever
// the order in which the columns come.
__device__ __forceinline__ void take_word(float v, uint32_t idx, bool negative, float& acc, uint32_t& word) {
    if (v > acc || (v == acc && word != SNB_NO_GRAD_ID && idx < (word & ~SNB_SIGN_BIT))) {
        acc = v;
        word = idx | (negative ? SNB_SIGN_BIT : 0u);
    }
}

// Running result of one output (K = 1): plain maxima, or maxima with their words.
template <int NX, bool TRACK>
struct MaxState {
    float acc[NX];
    uint32_t word[TRACK ? NX : 1];
    __device__ __forceinline__ void init(uint32_t floor_word) {
#pragma unroll
        for (int t = 0; t < NX; t++) acc[t] = SNB_EPS;
        if (TRACK) {
            word[0] = NX == 2 ? SNB_NO_GRAD_ID : floor_word; // lower bound: no gradient until it leaves its floor
            if (NX == 2) word[NX - 1] = 0u;
        }
    }
    // v: the row's values of this column (x | l, u | x, l, u)
    __device__ __forceinline__ void add(const float (&v)[NX], float w, uint32_t idx) {
        if (NX != 2) {
            const float t = v[0] - w;
            if (TRACK) take_word(fabsf(t), idx, t < 0.f, acc[0], word[0]);
            else acc[0] = fmaxf(acc[0], fabsf(t));
        }
        if (NX >= 2) {
            const float t1 = w - v[NX - 2], t2 = v[NX - 1] - w;
            if (TRACK) {
                const bool second = !(t1 <= t2);
                take_word(fmaxf(-t1, -t2), idx, second, acc[NX - 2], word[0]);
                take_word(fmaxf(t1, t2), idx, second, acc[NX - 1], word[TRACK ? NX - 1 : 0]);
            } else {
                acc[NX - 2] = max3(acc[NX - 2], -t1, -t2);
                acc[NX - 1] = max3(acc[NX - 1], t1, t2);
            }
        }
    }
    __device__ __forceinline__ float worst() const {
        float m = acc[0];
#pragma unroll
        for (int t = 1; t < NX; t++) m = fminf(m, acc[t]);
        return m;
    }
};

// The KMAX largest values of one output, ascending; slots above the number of values seen stay 0.
template <int KMAX>
struct TopList {
    float v[KMAX];
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int s = 0; s < KMAX; s++) v[s] = 0.f;
    }
    // Warp-uniform branches: a value that beats no row's weakest slot changes nothing, and one that beats no row's
    // slot HALF only moves the slots below it (the lists are walked largest first, so that is the later entries' lot).
    __device__ __forceinline__ void add(float d) {
        constexpr int HALF = KMAX / 2;
        if (__any_sync(0xffffffffu, d > v[0])) {
            const float e = d == d ? d : 0.f;                // a NaN must not move the list
            if (__any_sync(0xffffffffu, d > v[HALF])) {
#pragma unroll
                for (int s = 0; s < KMAX - 1; s++) v[s] = fmaxf(v[s], fminf(v[s + 1], e));
                v[KMAX - 1] = fmaxf(v[KMAX - 1], e);
            } else {
#pragma unroll
                for (int s = 0; s < HALF - 1; s++) v[s] = fmaxf(v[s], fminf(v[s + 1], e));
                v[HALF - 1] = fmaxf(v[HALF - 1], e);
            }
        }
    }
    // Four values at once, none of them NaN or negative: sorted, paired with the four weakest slots (ascending against descending: the
    // larger of each pair stays, and the slots are a bitonic sequence) and merged.  46 minima and maxima of ten slots against 80
    // one by one, 26 against 40 where no row's slot HALF is beaten; the votes are per four as well.  Point and box of a
    // 512 x 5120 x 5120 layer: 300 -> 212 us.
    template <int N>
    __device__ __forceinline__ void merge() {                // slots 0 .. N - 1 bitonic -> ascending
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
#pragma unroll
            for (int s = 0; s < N; s++)
                if ((s & d) == 0 && s + d < N) {
                    const float lo = fminf(v[s], v[s + d]), hi = fmaxf(v[s], v[s + d]);
                    v[s] = lo, v[s + d] = hi;
                }
    }
    __device__ __forceinline__ void add4(float a, float b, float c, float d) {
        constexpr int HALF = KMAX / 2;
        const float most = fmaxf(max3(a, b, c), d);
        if (!__any_sync(0xffffffffu, most > v[0])) return;
        auto order = [](float& x, float& y) {                // x >= y
            const float lo = fminf(x, y);
            x = fmaxf(x, y), y = lo;
        };
        order(a, b), order(c, d), order(a, c), order(b, d), order(b, c);
        const bool high = __any_sync(0xffffffffu, a > v[HALF]);
        v[0] = fmaxf(v[0], a), v[1] = fmaxf(v[1], b), v[2] = fmaxf(v[2], c), v[3] = fmaxf(v[3], d);
        if (high) merge<KMAX>();
        else merge<HALF>();
    }
    // The first eight values, none of them NaN or negative: 19 compare-and-swaps (Batcher's odd-even merge sort).
    __device__ __forceinline__ void start8(float (&e)[8]) {
        auto order = [&](int i, int j) {                     // ascending
            const float lo = fminf(e[i], e[j]);
            e[j] = fmaxf(e[i], e[j]), e[i] = lo;
        };
        order(0, 1), order(2, 3), order(4, 5), order(6, 7);
        order(0, 2), order(1, 3), order(4, 6), order(5, 7);
        order(1, 2), order(5, 6);
        order(0, 4), order(1, 5), order(2, 6), order(3, 7);
        order(2, 4), order(3, 5);
        order(1, 2), order(3, 4), order(5, 6);
#pragma unroll
        for (int s = 0; s < KMAX; s++) v[s] = s < KMAX - 8 ? 0.f : e[s < KMAX - 8 ? 0 : s - (KMAX - 8)];
    }
    // v[KMAX - K], as a minimum over an ascending tail: an index that is not a constant would move the list to local memory
    __device__ __forceinline__ float kth(int K) const {
        if (K == KMAX) return v[0];
        float r = v[KMAX - 1];
#pragma unroll
        for (int s = 0; s < KMAX - 1; s++)
            if (s >= KMAX - K) r = fminf(r, v[s]);
        return r;
    }
    // (eps0 + sum_r q (1-q)^r v_r) / (1 - (1-q)^K), largest first, in the reference's order of operations
    __device__ __forceinline__ float combine(int K, float q, float eps0) const {
        float ans = eps0, c = 1.0f;
#pragma unroll
        for (int r = 0; r < KMAX; r++)
            if (r < K) {
                ans += v[KMAX - 1 - r] * c * q;
                c *= 1 - q;
            }
        return ans / (1 - c);
    }
};

template <int NX, int KMAX>
struct SortState {
    TopList<KMAX> top[NX];
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int t = 0; t < NX; t++) top[t].init();
    }
    __device__ __forceinline__ void add(const float (&v)[NX], float w, uint32_t) {
        if (NX != 2) top[0].add(fabsf(v[0] - w));
        if (NX >= 2) {
            const float t1 = w - v[NX - 2], t2 = v[NX - 1] - w;
            top[NX - 2].add(fmaxf(-t1, -t2));
            top[NX - 1].add(fmaxf(t1, t2));
        }
    }
    // the lower bound's list holds the mirrored values: -combine(-1e-10, -v) = combine(1e-10, v)
    __device__ __forceinline__ float result(int t, int K, float q) const { return top[t].combine(K, q, SNB_EPS); }
};

// Positions of the K largest values, given a lower bound `floor_` of the K-th: columns must come in
// ascending order.  A value enters when it beats the weakest entry and passes every entry that it is >=
// to (the later of two equal columns ranks higher), the reference's bubble rule.
template <int KMAX>
struct PosList {
    float v[KMAX];
    uint32_t word[KMAX];
    float seed;
    __device__ __forceinline__ void init(float floor_) {
#pragma unroll
        for (int s = 0; s < KMAX; s++) v[s] = 0.f, word[s] = 0u;
        seed = floor_ > 0.f ? __int_as_float(__float_as_int(floor_) - 1) : 0.f;
    }
    // entries KMAX - K .. KMAX - 1 are in use
    __device__ __forceinline__ void add(float t, uint32_t c, int K) {
        const float d = fabsf(t);
        if (!__any_sync(0xffffffffu, d > seed)) return;
        float weakest = v[KMAX - 1];
#pragma unroll
        for (int s = 0; s < KMAX - 1; s++)
            if (s >= KMAX - K) weakest = fminf(weakest, v[s]);
        const bool enter = d > seed && d > weakest;
        const uint32_t wd = c | (t >= 0.f ? 0u : SNB_SIGN_BIT);
#pragma unroll
        for (int s = 0; s < KMAX; s++) {
            if (s < KMAX - K) continue;
            const bool here = enter && (s == KMAX - K || d >= v[s]);
            const bool above = s + 1 < KMAX && enter && d >= v[s + 1 < KMAX ? s + 1 : s];
            v[s] = above ? v[s + 1 < KMAX ? s + 1 : s] : (here ? d : v[s]);
            word[s] = above ? word[s + 1 < KMAX ? s + 1 : s] : (here ? wd : word[s]);
        }
    }
};

// Position of an output at its floor: the first kept column (never one outside W, whatever the list holds).
__device__ __forceinline__ uint32_t first_kept(const PruneProblem& p, int s) {
    return p.kept_list ? min((uint32_t)p.kept_list[(size_t)s * p.kept], (uint32_t)p.W_CI - 1u) : 0u;
}

// ---- results of 32 outputs / of one output ---------------------------------------------------------
template <int NV>
__device__ __forceinline__ float shifted(const PruneProblem& p, float v, int j) {
    if (p.mean) v = v - p.mean[j];
    if (p.bias) v = v + p.bias[j];
    return v;
}

// One output of a sub-batch in the chain form, lane = row.
template <int NV>
__device__ __forceinline__ void emit_chain(const PruneProblem& p, int s, int j, const float (&v)[NV], uint32_t word, bool final = true) {
    const int lane = threadIdx.x & 31;
    const bool live = s * 32 + lane < p.B, kept = !p.keep || p.keep[(size_t)s * p.CO + j];
    if (p.yt) {
        unsigned hi = 0u, nlo = 0u;
#pragma unroll
        for (int t = 0; t < NV; t++) {
            const float o = live && kept ? shifted<NV>(p, v[t], j) : __int_as_float(0x7fc00000);
            p.yt[(((size_t)s * p.CO + j) * NV + t) * 32 + lane] = o;
            hi = max(hi, order_code(o));
            nlo = max(nlo, order_code(-o));
        }
        if (p.yhi && final) {                                // values that will be done again would widen the ranges
            hi = __reduce_max_sync(0xffffffffu, hi);
            nlo = __reduce_max_sync(0xffffffffu, nlo);
            if (lane == 0) {
                atomicMax(p.yhi + j, hi);
                atomicMax(p.ynlo + j, nlo);
            }
        }
    }
    if (p.post) p.post[((size_t)s * p.CO + j) * 32 + lane] = live && kept ? (int)word : (int)SNB_NO_GRAD_ID;
}

// SLOTS outputs from the tile [NV values (+ NW words)][row][output]: row-major arrays and the chain form.
template <int NX, int NV, int NW, int SLOTS = 32>
__device__ __forceinline__ void emit_tile(const PruneProblem& p, float (*tile)[32][SLOTS + 1], int s, int n0, unsigned again = 0u) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float* outs[NV];
    if (NX != 2) outs[0] = p.y;
    if (NX >= 2) outs[NV - 2] = p.yl, outs[NV - 1] = p.yu;
    const int col = tid % SLOTS, no = n0 + col;
    const bool here = no < p.CO, kept = here && (!p.keep || p.keep[(size_t)s * p.CO + no]);
#pragma unroll
    for (int k = 0; k < SLOTS / 8; k++) {
        const int r = tid / SLOTS + 256 / SLOTS * k, b = s * 32 + r;
        if (b >= p.B || !here) continue;
        const size_t o = (size_t)b * p.CO + no;
#pragma unroll
        for (int t = 0; t < NV; t++)
            if (outs[t]) outs[t][o] = shifted<NV>(p, tile[t][r][col], no);
        if (NW == 1 && NX == 1 && p.pos) p.pos[o] = kept ? __float_as_int(tile[NV][r][col]) : (int)SNB_NO_GRAD_ID;
        if (NW == 2) {
            p.posl[o] = __float_as_int(tile[NV][r][col]);
            p.posu[o] = __float_as_int(tile[NV + NW - 1][r][col]);
        }
    }
    if (p.yt || p.post) {
#pragma unroll
        for (int i = 0; i < SLOTS / 8; i++) {
            const int slot = warp * (SLOTS / 8) + i;
            if (n0 + slot >= p.CO) break;
            float v[NV];
#pragma unroll
            for (int t = 0; t < NV; t++) v[t] = tile[t][lane][slot];
            emit_chain<NV>(p, s, n0 + slot, v, NW > 0 ? __float_as_uint(tile[NW > 0 ? NV : 0][lane][slot]) : 0u, !((again >> slot) & 1u));
        }
    }
    if (p.part && tid < SLOTS && here) {
        float sum = 0.f;
        const int rows = min(32, p.B - s * 32);
        for (int r = 0; r < rows; r++) sum += tile[0][r][col];
        p.part[(size_t)s * p.CO + no] = kept ? sum : 0.f;
    }
}

// Whether this warp is the last of its CTA's to come here (`arrived` zeroed before); what the others wrote before is visible then. Nobody waits.
__device__ __forceinline__ bool last_warp(unsigned* arrived) {
    __threadfence_block();
    __syncwarp();
    unsigned n = 0;
    if ((threadIdx.x & 31) == 0) n = atomicAdd(arrived, 1u);
    const bool last = __shfl_sync(0xffffffffu, n, 0) + 1 == blockDim.x / 32;
    if (last) __threadfence_block();
    return last;
}

// ---- a layer that will be evaluated as a whole ------------------------------------------------------
// What prune_redo needs, shared out over the CTAs (s, n0) of the walk it replaces: the rows of x side by side again, empty
// partial results (`bytes` per value; 0: none are kept), and the outputs that `keep` drops.  256 threads.
template <int NX>
__device__ __noinline__ void dense_prepare(const PruneArgs& a, int s, int n0, int bytes, int slots = 32) {
    const PruneProblem& p = a.p;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, C = p.W_CI;
    const float nan = __int_as_float(0x7fc00000);
    if (!p.ci || a.counters[GENERAL] == 0u) {
        const int pieces = (C + 7) / 8;
        for (int k = (int)((long long)pieces * blockIdx.x / gridDim.x) + warp; k < (long long)pieces * (blockIdx.x + 1) / gridDim.x; k += 8)
#pragma unroll
            for (int t = 0; t < NX; t++) {
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; e++) {
                    const int c = 8 * k + e;
                    v[e] = c < C ? a.xt[(((size_t)s * C + c) * NX + t) * 32 + lane] : nan;
                }
                float4* dst = reinterpret_cast<float4*>(a.xr + ((size_t)(t * a.S + s) * 32 + lane) * a.ldr + 8 * k);
                dst[0] = make_float4(v[0], v[1], v[2], v[3]);
                if (8 * k + 4 < a.ldr) dst[1] = make_float4(v[4], v[5], v[6], v[7]);
            }
    }
    if (bytes) {
        const int quads = min(32, p.CO - n0) * 32 * bytes / 16;
#pragma unroll
        for (int t = 0; t < NX; t++) {
            int4* part = reinterpret_cast<int4*>(a.partial + ((size_t)(t * a.S + s) * p.CO + n0) * 32 * bytes);
            for (int k = tid; k < quads; k += 256) part[k] = make_int4(0, 0, 0, 0);
        }
        if (tid == 0 && n0 % 128 == 0) a.tile_done[(size_t)s * ((p.CO + 127) / 128) + n0 / 128] = 0u;
    }
    if (!p.keep) return;
    for (int i = 0; i < slots / 8; i++) {
        const int n = n0 + warp * (slots / 8) + i, b = s * 32 + lane;
        if (n >= p.CO || p.keep[(size_t)s * p.CO + n]) continue;
        const float v[NX] = {};
        emit_chain<NX>(p, s, n, v, 0u);
        if (b < p.B && p.pos) p.pos[(size_t)b * p.CO + n] = (int)SNB_NO_GRAD_ID;
        if (p.part && lane == 0) p.part[(size_t)s * p.CO + n] = 0.f;
    }
}

// ---- list walks -----------------------------------------------------------------------------------
// CTA = 32 outputs of one sub-batch, eight lanes per output, four rows per lane (one 16-byte load of xt per tensor and
// column): a warp walks four lists side by side.  A step is STEP columns; the entries of the next step are fetched
// while this one's columns are on their way; a walk ends when the largest U left is below the results of all 32 rows.
// Bound by the latency of the two dependent loads (list, column) and by the columns' traffic from L2.
// TRACK keeps, per row, the step that set the maximum; the word is made at the end from the step's columns.  A
// later step that only equals the maximum (rare) sends the lane over the list once more for the lowest position.
template <int NX, bool TRACK>
constexpr int WALK_CTAS = NX == 1 && !TRACK ? 6 : NX == 2 && TRACK ? 3 : 4;
template <int NX, bool TRACK>
__global__ void __launch_bounds__(256, WALK_CTAS<NX, TRACK>) prune_max(const __grid_constant__ PruneArgs a) {
    constexpr int NV = NX == 3 ? 3 : NX;                     // values per row: |x - w|, lower, upper
    constexpr int WORDS = TRACK ? NX : 0;
    __shared__ float tile[NV + WORDS][32][33];
    __shared__ unsigned failed, arrived;
    const PruneProblem& p = a.p;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 3, l = lane & 7;
    const int s = blockIdx.y, n0 = blockIdx.x * 32, C = p.W_CI, slot = warp * 4 + g, n = n0 + slot;
    const float4* xt = reinterpret_cast<const float4*>(a.xt + (size_t)s * C * NX * 32) + l;
    after_previous();
    let_next();
    const unsigned overflowed = load_now(a.counters + OVERFLOWED), general = p.ci ? load_now(a.counters + GENERAL) : 0u;
    const int j = n < p.CO ? (p.co ? p.co[(size_t)s * p.CO + n] : n) : 0;
    // What the walk starts from comes together, not one after the other: the head of a list that is not there (or not wanted) is memory all the
    // same, and not looked at.  Seven layers of points and boxes 460 -> 443 us.
    const int4* list = reinterpret_cast<const int4*>(a.cand + (size_t)j * a.lcap);
    const int listed = a.cnt[j];
    int4 e01 = list[0], e23 = list[1];
    const float tau = a.tau[j];
    const bool wanted = n < p.CO && (!p.keep || p.keep[(size_t)s * p.CO + j]);
    const int cnt = wanted ? listed : 0;
    const float* ub = a.ub + (size_t)j * (a.lcap / STEP);
    const int live = min(4, p.B - s * 32 - 4 * l);           // rows of this lane that exist (may be <= 0)

    float acc[NV][4];
    int at[TRACK ? NV : 1][TRACK ? 4 : 1];                   // step of the maximum, -1: at its floor
    unsigned tied = 0u;                                      // bit t * 4 + q: another step reaches the same value
#pragma unroll
    for (int t = 0; t < NV; t++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
            acc[t][q] = q < live ? SNB_EPS : INFINITY;       // rows past the batch never hold a walk up
            if (TRACK) at[TRACK ? t : 0][TRACK ? q : 0] = -1;
        }
    auto worst = [&]() {
        float m = acc[0][0];
#pragma unroll
        for (int t = 0; t < NV; t++)
#pragma unroll
            for (int q = 0; q < 4; q++) m = fminf(m, acc[t][q]);
        return m;
    };
    // the row's values for column value(s) x and weight w
    auto values = [&](const float (&x)[NX], float w, float (&v)[NV]) {
        if (NX != 2) v[0] = fabsf(x[0] - w);
        if (NX >= 2) {
            const float t1 = w - x[NX - 2], t2 = x[NX - 1] - w;
            v[NV - 2] = fmaxf(-t1, -t2);
            v[NV - 1] = fmaxf(t1, t2);
        }
    };
    bool active = cnt > 0;
    float left = 0.f;
    int walked = 0;
    // looked at only here, so that it is on its way together with the head of the list
    if ((general & LIST_TWICE) || prune_gives_up(overflowed, p.W_CO)) {
        if (!p.leave) dense_prepare<NX>(a, s, n0, TRACK ? 8 : 4);
        return;
    }
    if (tid == 0) failed = arrived = 0u;
    __syncthreads();
    for (int b = 0;; b++) {
        if (b > 0) {
            const unsigned over = __ballot_sync(0xffffffffu, worst() > left);
            active = active && b * STEP < cnt && ((over >> (8 * g)) & 0xffu) != 0xffu;
        }
        if (!__any_sync(0xffffffffu, active)) break;
        if (active) {
            const int c[STEP] = {e01.x, e01.z, e23.x, e23.z};
            const float w[STEP] = {__int_as_float(e01.y), __int_as_float(e01.w), __int_as_float(e23.y), __int_as_float(e23.w)};
            float4 x[STEP][NX];
#pragma unroll
            for (int e = 0; e < STEP; e++)
#pragma unroll
                for (int t = 0; t < NX; t++) x[e][t] = xt[((size_t)c[e] * NX + t) * 8];
            if ((b + 1) * STEP < cnt) {
                e01 = list[2 * b + 2];
                e23 = list[2 * b + 3];
                left = ub[b + 1];
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float v[STEP][NV];
#pragma unroll
                for (int e = 0; e < STEP; e++) {
                    float xq[NX];
#pragma unroll
                    for (int t = 0; t < NX; t++) xq[t] = q == 0 ? x[e][t].x : q == 1 ? x[e][t].y : q == 2 ? x[e][t].z : x[e][t].w;
                    values(xq, w[e], v[e]);
                }
#pragma unroll
                for (int t = 0; t < NV; t++) {
                    if (TRACK) {
                        const float m = fmaxf(max3(v[0][t], v[1][t], v[2][t]), v[3][t]);
                        if (m == acc[t][q]) tied |= 1u << (t * 4 + q);
                        if (m > acc[t][q]) {
                            at[TRACK ? t : 0][TRACK ? q : 0] = b;
                            tied &= ~(1u << (t * 4 + q));
                        }
                        acc[t][q] = fmaxf(acc[t][q], m);
                    } else {
                        acc[t][q] = max3(max3(acc[t][q], v[0][t], v[1][t]), v[2][t], v[3][t]);
                    }
                }
            }
            walked = b + 1;
        }
    }
    const unsigned good = __ballot_sync(0xffffffffu, worst() >= tau);
    const bool again = wanted && (cnt < 0 || ((good >> (8 * g)) & 0xffu) != 0xffu);
    if (l == 0 && again) atomicOr(&failed, 1u << slot);
    // Row-major results go through a tile; the chain form is written from here, and no warp waits for the others.
    const bool chain = NX == 3 - 2 * TRACK && !p.y && !p.yl && !p.yu;
    if (!chain || p.part) {
#pragma unroll
        for (int t = 0; t < NV; t++)
#pragma unroll
            for (int q = 0; q < 4; q++) tile[t][4 * l + q][slot] = acc[t][q];
    }
    uint32_t word[TRACK ? NV : 1][4];
    if (TRACK) {
        const int* inv = p.ci ? a.inv + (size_t)s * C : nullptr;
        const float* xs = reinterpret_cast<const float*>(xt);
        // lowest position among the entries of step k whose value for row q is `want`
        auto step_word = [&](int t, int q, int k, float want, uint32_t word) {
            const int4 a01 = list[2 * k], a23 = list[2 * k + 1];
            const int c[STEP] = {a01.x, a01.z, a23.x, a23.z};
            const float w[STEP] = {__int_as_float(a01.y), __int_as_float(a01.w), __int_as_float(a23.y), __int_as_float(a23.w)};
            float xq[STEP][NX];
            int idx[STEP];
#pragma unroll
            for (int e = 0; e < STEP; e++) {
                idx[e] = inv ? inv[c[e]] : c[e];
#pragma unroll
                for (int u = 0; u < NX; u++) xq[e][u] = xs[((size_t)c[e] * NX + u) * 32 + q];
            }
#pragma unroll
            for (int e = 0; e < STEP; e++) {
                float v[NV];
                values(xq[e], w[e], v);
                bool negative = xq[e][0] - w[e] < 0.f;
                if (NX == 2) negative = !(w[e] - xq[e][0] <= xq[e][NX - 1] - w[e]);
                if (v[t] == want && (uint32_t)idx[e] < (word & ~SNB_SIGN_BIT)) word = (uint32_t)idx[e] | (negative ? SNB_SIGN_BIT : 0u);
            }
            return word;
        };
        const uint32_t floor_word = first_kept(p, s);
#pragma unroll
        for (int t = 0; t < NV; t++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int k = at[TRACK ? t : 0][TRACK ? q : 0];
                uint32_t wd = (NX == 2 && t == 0) ? SNB_NO_GRAD_ID : floor_word;
                if (k >= 0) {
                    wd = step_word(t, q, k, acc[t][q], 0x7fffffffu);
                    if ((tied >> (t * 4 + q)) & 1u)
                        for (int k2 = 0; k2 < walked; k2++) wd = step_word(t, q, k2, acc[t][q], wd);
                }
                word[TRACK ? t : 0][q] = wd;
            }
    }
    if (!chain) {
        if (TRACK) {
#pragma unroll
            for (int t = 0; t < NV; t++)
#pragma unroll
                for (int q = 0; q < 4; q++) tile[NV + (TRACK ? t : 0)][4 * l + q][slot] = __uint_as_float(word[TRACK ? t : 0][q]);
        }
        __syncthreads();
        emit_tile<NX, NV, WORDS>(p, tile, s, n0, failed);
        if (tid == 0 && failed) a.fail[atomicAdd(a.counters + FAILED, 1u)] = make_int4(s, n0, (int)failed, 0);
        return;
    }
    if (p.yt) {
        unsigned hi = 0u, nlo = 0u;
#pragma unroll
        for (int t = 0; t < NV; t++) {
            float o[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                o[q] = q < live && wanted ? shifted<NV>(p, acc[t][q], n) : __int_as_float(0x7fc00000);
                hi = max(hi, order_code(o[q]));
                nlo = max(nlo, order_code(-o[q]));
            }
            if (n < p.CO) reinterpret_cast<float4*>(p.yt)[(((size_t)s * p.CO + n) * NV + t) * 8 + l] = make_float4(o[0], o[1], o[2], o[3]);
        }
        if (p.yhi) {
#pragma unroll
            for (int d = 4; d > 0; d >>= 1) {
                hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, d));
                nlo = max(nlo, __shfl_xor_sync(0xffffffffu, nlo, d));
            }
            if (l == 0 && wanted && !again) {                // values that will be done again would widen the ranges
                atomicMax(p.yhi + n, hi);
                atomicMax(p.ynlo + n, nlo);
            }
        }
    }
    if (TRACK && p.post && n < p.CO) {
        int o[4];
#pragma unroll
        for (int q = 0; q < 4; q++) o[q] = q < live && wanted ? (int)word[0][q] : (int)SNB_NO_GRAD_ID;
        reinterpret_cast<int4*>(p.post)[((size_t)s * p.CO + n) * 8 + l] = make_int4(o[0], o[1], o[2], o[3]);
    }
    if (!last_warp(&arrived)) return;
    if (p.part && n0 + lane < p.CO) {
        const bool kept = !p.keep || p.keep[(size_t)s * p.CO + n0 + lane];
        const int rows = min(32, p.B - s * 32);
        float sum = 0.f;
        for (int r = 0; r < rows; r++) sum += tile[0][r][lane];
        p.part[(size_t)s * p.CO + n0 + lane] = kept ? sum : 0.f;
    }
    if (lane == 0) {
        const unsigned mask = *(volatile unsigned*)&failed;
        if (mask) a.fail[atomicAdd(a.counters + FAILED, 1u)] = make_int4(s, n0, (int)mask, 0);
    }
}

// Positions of one output whose K-th largest value is shared by several columns in some row: the entries of
// the list in ascending column order through PosList (rare; 32 lanes pick the next column together).
template <int KMAX, int LD>
__device__ __noinline__ void ordered_positions(const int2* entries, int cnt, const float* xt, float least, int K,
                                               float (*words)[32][LD], int slot) {
    const int lane = threadIdx.x & 31;
    PosList<KMAX> pl;
    pl.init(least);
    int last = -1;
    for (;;) {
        uint32_t next = 0xffffffffu;                         // (column << 9 | entry) of the lowest column above `last`
        for (int k = lane; k < cnt; k += 32) {
            const int c = entries[k].x;
            if (c > last) next = min(next, (uint32_t)c << 9 | (uint32_t)k);
        }
        next = __reduce_min_sync(0xffffffffu, next);
        if (next == 0xffffffffu) break;
        const int2 e = entries[next & 511u];
        last = e.x;
        pl.add(xt[(size_t)e.x * 32] - __int_as_float(e.y), (uint32_t)e.x, K);
    }
#pragma unroll
    for (int k = 0; k < KMAX; k++)
        if (k < K) words[k][lane][slot] = __uint_as_float(pl.word[KMAX - 1 - k]);
}

// What may enter a row's list waits in shared memory until a row has four of them, and only then are the lists touched: after the first eight entries a row takes
// one in five, but some row of the warp takes one of nearly every step.  512 x 5120 x 3000, K = 17: values 370 -> 291 us, boxes
// 800 -> 525; K = 10: values 147 -> 131.  Boxes, and points with boxes, of up to ten values are inserted as they come: three tests and a store per column
// cost what they save (box 512 x 2048 x 2000 109 us as they come, 121 queued).  With positions of up to ten values the queue is a log of (value,
// column) that the ranking reads; of more, it lies where the ranking's values come later.
template <int NX, int KMAX, bool POS>
struct SortQueue {
    static constexpr bool LOG = POS && KMAX <= 10;
    static constexpr bool USED = POS || NX == 1 || KMAX > 10;
    static constexpr int DEPTH = LOG ? 16 : USED ? 8 : 0;
    static constexpr int WIDTH = NX == 3 ? 4 : NX;           // floats of an entry: the values of all tensors side by side
};
constexpr int SORT_SLOTS = 8;           // outputs of a CTA of prune_sort
template <int KMAX>
constexpr int SORT_CTAS = KMAX <= 10 ? 4 : 2;
template <int NX, int KMAX, bool POS>
constexpr int sort_walk_smem(int K) {
    using Q = SortQueue<NX, KMAX, POS>;
    const int tile = (NX + (POS ? K : 0)) * 32 * (SORT_SLOTS + 1), found = POS ? 8 * K * 32 : 0;
    const int queue = POS && !Q::LOG ? 0 : 8 * Q::DEPTH * Q::WIDTH * 32;
    return (tile + found + queue) * (int)sizeof(float) + (Q::LOG ? 8 * Q::DEPTH * 32 * (int)sizeof(unsigned short) : 0);
}
// Without a branch: a row's values of a column go to the end of its queue if one of them beats the least of its list.
__device__ __forceinline__ void push_above(unsigned& end, const float (&v)[1], const float (&least)[1]) {
    asm volatile("{\n .reg .pred p;\n setp.gt.f32 p, %1, %2;\n @p st.shared.f32 [%0], %1;\n @p add.u32 %0, %0, 128;\n}"
                 : "+r"(end) : "f"(v[0]), "f"(least[0]) : "memory");
}
__device__ __forceinline__ void push_above(unsigned& end, const float (&v)[2], const float (&least)[2]) {
    asm volatile(
        "{\n .reg .pred p;\n setp.gt.f32 p, %1, %3;\n setp.gt.or.f32 p, %2, %4, p;\n @p st.shared.v2.f32 [%0], {%1, %2};\n"
        " @p add.u32 %0, %0, 256;\n}"
        : "+r"(end) : "f"(v[0]), "f"(v[1]), "f"(least[0]), "f"(least[1]) : "memory");
}
__device__ __forceinline__ void push_above(unsigned& end, const float (&v)[3], const float (&least)[3]) {
    asm volatile(
        "{\n .reg .pred p;\n setp.gt.f32 p, %1, %4;\n setp.gt.or.f32 p, %2, %5, p;\n setp.gt.or.f32 p, %3, %6, p;\n"
        " @p st.shared.v4.f32 [%0], {%1, %2, %3, %3};\n @p add.u32 %0, %0, 512;\n}"
        : "+r"(end) : "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(least[0]), "f"(least[1]), "f"(least[2]) : "memory");
}
// An entry of the queue, which is empty (zero) then.
__device__ __forceinline__ void take_entry(unsigned at, float (&v)[1]) {
    asm volatile("ld.shared.f32 %0, [%1];\n st.shared.f32 [%1], %2;" : "=&f"(v[0]) : "r"(at), "f"(0.f) : "memory");
}
__device__ __forceinline__ void take_entry(unsigned at, float (&v)[2]) {
    asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];\n st.shared.v2.f32 [%2], {%3, %3};" : "=&f"(v[0]), "=&f"(v[1]) : "r"(at), "f"(0.f) : "memory");
}
__device__ __forceinline__ void take_entry(unsigned at, float (&v)[3]) {
    float none;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n st.shared.v4.f32 [%4], {%5, %5, %5, %5};"
                 : "=&f"(v[0]), "=&f"(v[1]), "=&f"(v[2]), "=&f"(none) : "r"(at), "f"(0.f) : "memory");
}
// The same for a value and its column, if the value's size is at least `least`.
__device__ __forceinline__ void push_pair(unsigned& end, unsigned& column_end, float v, int column, float least) {
    asm volatile(
        "{\n .reg .pred p;\n .reg .f32 d;\n abs.f32 d, %2;\n setp.ge.f32 p, d, %4;\n @p st.shared.f32 [%0], %2;\n @p st.shared.u16 [%1], %3;\n"
        " @p add.u32 %0, %0, 128;\n @p add.u32 %1, %1, 64;\n}"
        : "+r"(end), "+r"(column_end) : "f"(v), "h"((unsigned short)column), "f"(least) : "memory");
}
// A column that reaches a row's K-th value: its size and its word, as long as there is room.
__device__ __forceinline__ void push_hit(int& hits, unsigned& at, unsigned& word_at, float v, int column, float least, int K, unsigned word_stride) {
    asm volatile(
        "{\n .reg .pred p, r;\n .reg .f32 d;\n .reg .b32 w;\n abs.f32 d, %3;\n setp.ge.f32 p, d, %5;\n setp.gt.and.f32 p, d, 0f00000000, p;\n"
        " setp.lt.and.s32 r, %0, %6, p;\n mov.b32 w, %3;\n and.b32 w, w, 0x80000000;\n or.b32 w, w, %4;\n"
        " @r st.shared.f32 [%1], d;\n @r st.shared.b32 [%2], w;\n @r add.u32 %1, %1, 128;\n @r add.u32 %2, %2, %7;\n @p add.s32 %0, %0, 1;\n}"
        : "+r"(hits), "+r"(at), "+r"(word_at) : "f"(v), "r"(column), "f"(least), "r"(K), "r"(word_stride) : "memory");
}
__device__ __forceinline__ float shared_f32(unsigned at) {
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ int shared_u16(unsigned at) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(at) : "memory");
    return v;
}

// The sort neuron over the same lists, one warp per output, lane = row; POS: the K positions too.  Bound by the issue of minima and maxima
// (half-rate pipe, 73 % busy).  The first eight entries of the list (largest upper bounds) start a row's list, by sorting; the others are inserted four
// at a time.  In the chain form a warp writes its output and leaves, without a tile.  Point and box of 512 x 5120 x 5120: 287 -> 243 us.
// POS: with the values known, the columns that reach a row's K-th value are collected, from the first entries and the log of what was
// queued (from a second walk where the log ran over, and for more than ten values); there are K of them, and the rank of one is the
// number of larger values in the row's list, of equal values the later column first.  Only where more columns share the K-th value than there is room for does the
// order of insertion decide (ordered_positions).  128 x 5120 x 5120, K = 10: 107 -> 86 us; always with a second walk, and
// each word stored for eight of 32 lanes: 107.
template <int NX, int KMAX, bool POS>
__global__ void __launch_bounds__(256, SORT_CTAS<KMAX>) prune_sort(const __grid_constant__ PruneArgs a) {
    constexpr uint32_t EMPTY = 0xffffffffu;
    constexpr int LD = SORT_SLOTS + 1;
    constexpr bool LOG = SortQueue<NX, KMAX, POS>::LOG, QUEUED = SortQueue<NX, KMAX, POS>::USED;
    constexpr int DEPTH = SortQueue<NX, KMAX, POS>::DEPTH, FLUSH = 3;
    constexpr int WIDTH = SortQueue<NX, KMAX, POS>::WIDTH;
    constexpr unsigned ROW = WIDTH * 32 * sizeof(float);     // bytes from one queued entry to the next
    extern __shared__ __align__(16) unsigned char dyn[];
    float(*tile)[32][LD] = reinterpret_cast<float(*)[32][LD]>(dyn);   // [NX] values, then [K] words
    float* const found = reinterpret_cast<float*>(dyn) + (NX + (POS ? a.p.K : 0)) * 32 * LD;  // POS: [8 warps][K][32]
    __shared__ unsigned failed, arrived;
    const PruneProblem& p = a.p;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int s = blockIdx.y, n0 = blockIdx.x * SORT_SLOTS, C = p.W_CI, K = p.K;
    const bool live = s * 32 + lane < p.B;
    const float* xt = a.xt + (size_t)s * C * NX * 32 + lane;
    // queue [8 warps][DEPTH][32 rows][WIDTH], columns [8 warps][DEPTH][32]
    const unsigned found_at = smem_u32(found), queues = POS && !LOG ? found_at : found_at + (POS ? 8 * K * 128 : 0);
    const unsigned queue = queues + (POS && !LOG ? warp * K * 128 : warp * DEPTH * ROW) + lane * WIDTH * 4;
    const unsigned columns = queues + 8 * DEPTH * ROW + warp * DEPTH * 64 + lane * 2;
    const int fill = max(8, (K + 3) / 4 * 4);                // LOG: entries that are not logged
    after_previous();
    if (dense_mode(a)) {                                     // no CTA of the next kernel before the last of these: its few hundred long ones spread evenly then
        if (!POS) dense_prepare<NX>(a, s, n0, 0, SORT_SLOTS);     // positions: sort_positions_if reads the rows as they came
        return;
    }
    let_next();
    const bool chain = !POS && !p.y && !p.yl && !p.yu && !p.part;   // written from here: no warp waits for the others
    if (tid == 0) failed = arrived = 0u;
    __syncthreads();
    const int slot = warp, j = n0 + slot;
    if (j < p.CO) {
        if (QUEUED && !LOG) {
            float none[NX];
#pragma unroll
            for (int q = 0; q < DEPTH; q++) take_entry(queue + q * ROW, none);
        }
        const int cnt = a.cnt[j];
        const float tau = a.tau[j];
        const int4* list = reinterpret_cast<const int4*>(a.cand + (size_t)j * a.lcap);
        const float* ub = a.ub + (size_t)j * (a.lcap / STEP);
        TopList<KMAX> top[NX];
        float reach[NX];                                     // the K-th value when the list was last touched
        unsigned end = queue;                                // of what is queued
        unsigned merged = queue;                             // LOG: of what of it is in the list
        unsigned column_end = columns;
        bool lost = false;                                   // LOG: it ran over
#pragma unroll
        for (int t = 0; t < NX; t++) top[t].init(), reach[t] = 0.f;
        // Row values of one column: x - w or |x - w|, lower, upper.
        auto values = [&](const float (&x)[NX], float w, float (&e)[NX]) {
            if (NX != 2) e[0] = LOG ? x[0] - w : fabsf(x[0] - w);
            if (NX >= 2) {
                const float t1 = w - x[NX - 2], t2 = x[NX - 1] - w;
                e[NX - 2] = fmaxf(-t1, -t2);
                e[NX - 1] = fmaxf(t1, t2);
            }
        };
        float w[STEP], v[STEP][NX];
        int c[STEP];
        int4 two[STEP / 2];
        auto entries = [&](int at) {
#pragma unroll
            for (int e = 0; e < STEP / 2; e++) two[e] = list[at / 2 + e];
        };
        auto fetch = [&]() {
#pragma unroll
            for (int e = 0; e < STEP; e++) {
                c[e] = e % 2 ? two[e / 2].z : two[e / 2].x;
                w[e] = __int_as_float(e % 2 ? two[e / 2].w : two[e / 2].y);
#pragma unroll
                for (int t = 0; t < NX; t++) v[e][t] = xt[((size_t)c[e] * NX + t) * 32];
            }
        };
        int k = 0;                                           // entries seen
        if (cnt > 0) {
            float left = 0.f;
            {
                float first[NX][8];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    entries(4 * h);
                    fetch();
#pragma unroll
                    for (int q = 0; q < STEP; q++) {
                        float e[NX];
                        values(v[q], w[q], e);
#pragma unroll
                        for (int t = 0; t < NX; t++) first[t][4 * h + q] = fmaxf(t == 0 && LOG ? fabsf(e[t]) : e[t], 0.f);   // NaN -> 0
                    }
                }
#pragma unroll
                for (int t = 0; t < NX; t++) top[t].start8(first[t]), reach[t] = top[t].kth(K);
            }
            k = 8;
            if (!QUEUED) {
                for (; k < cnt; k += STEP) {
                    left = ub[k / STEP];
                    float least = top[0].kth(K);
#pragma unroll
                    for (int t = 1; t < NX; t++) least = fminf(least, top[t].kth(K));
                    if (__all_sync(0xffffffffu, !live || least > left)) break;
                    entries(k);
                    fetch();
                    float e[STEP][NX];
#pragma unroll
                    for (int q = 0; q < STEP; q++) {
                        values(v[q], w[q], e[q]);
#pragma unroll
                        for (int t = 0; t < NX; t++) e[q][t] = fmaxf(e[q][t], 0.f);     // NaN -> 0
                    }
#pragma unroll
                    for (int t = 0; t < NX; t++) top[t].add4(e[0][t], e[1][t], e[2][t], e[3][t]);
                }
#pragma unroll
                for (int t = 0; t < NX; t++) reach[t] = top[t].kth(K);
            }
            if (QUEUED && k < cnt) left = ub[k / STEP];
            if (QUEUED && NX < 3 && k < cnt) entries(k);
            while (QUEUED) {
                float least = reach[0];
#pragma unroll
                for (int t = 1; t < NX; t++) least = fminf(least, reach[t]);
                const bool over = k >= cnt || __all_sync(0xffffffffu, !live || least > left);
                if (!over) {
                    if (NX == 3) entries(k);                 // registers
                    fetch();
                    k += STEP;
                    if (NX < 3 && k < cnt) entries(k);
                    if (k < cnt) left = ub[k / STEP];
#pragma unroll
                    for (int q = 0; q < STEP; q++) {
                        float e[NX];
                        values(v[q], w[q], e);
                        if (LOG) push_pair(end, column_end, e[0], c[q], reach[0]);
                        else push_above(end, e, reach);
                    }
                }
                const bool full = LOG && __any_sync(0xffffffffu, end > queue + (DEPTH - 4) * ROW);
                if (over || full || (LOG && k <= fill) || __any_sync(0xffffffffu, end > merged + FLUSH * ROW)) {
                    for (unsigned r = merged; __any_sync(0xffffffffu, r < end); r += 4 * ROW) {
                        float e[4][NX];
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            if (LOG) {
                                const float queued = shared_f32(r + q * ROW);   // past the end: whatever follows in shared memory
                                e[q][0] = r + q * ROW < end ? fabsf(queued) : 0.f;
                            } else {
                                take_entry(r + q * ROW, e[q]);
#pragma unroll
                                for (int t = 0; t < NX; t++) e[q][t] = fmaxf(e[q][t], 0.f);     // NaN -> 0
                            }
                        }
#pragma unroll
                        for (int t = 0; t < NX; t++) top[t].add4(e[0][t], e[1][t], e[2][t], e[3][t]);
                    }
#pragma unroll
                    for (int t = 0; t < NX; t++) reach[t] = top[t].kth(K);
                    if (LOG) {
                        merged = end;
                        if (k <= fill || (full && !over)) {  // a new log
                            lost = lost || k > fill;
                            end = merged = queue;
                            column_end = columns;
                        }
                    } else {
                        end = queue;
                    }
                }
                if (over) break;
            }
        }
        float worst = reach[0];
#pragma unroll
        for (int t = 1; t < NX; t++) worst = fminf(worst, reach[t]);
        const bool good = cnt >= 0 && __all_sync(0xffffffffu, !live || worst >= tau);
        if (!good && lane == 0) atomicOr(&failed, 1u << slot);
        float result[NX];
#pragma unroll
        for (int t = 0; t < NX; t++) result[t] = top[t].combine(K, p.q, SNB_EPS);
        if (chain) emit_chain<NX>(p, s, j, result, 0u, good);
        else
#pragma unroll
            for (int t = 0; t < NX; t++) tile[t][lane][slot] = result[t];
        if (POS && good) {
            const float least = reach[0];
            float* mine = found + warp * K * 32 + lane;      // this row's values in the order of the walk; their words in the tile
            int hits = 0;
            bool twice = false;
#pragma unroll
            for (int r = 1; r < KMAX; r++) twice = twice || (r > KMAX - K && top[0].v[r] > 0.f && top[0].v[r] == top[0].v[r - 1]);
            unsigned at = smem_u32(mine), word_at = smem_u32(&tile[NX][lane][slot]);
            // Entries past k have smaller upper bounds than every row's K-th value: none of them is a hit.
            const int again = LOG && !lost ? min(fill, k) : k;
            for (int k2 = 0; k2 < again; k2 += STEP) {
                entries(k2);
                fetch();
#pragma unroll
                for (int q = 0; q < STEP; q++) push_hit(hits, at, word_at, v[q][0] - w[q], c[q], least, K, 32 * LD * 4);
            }
            if (LOG && !lost) {
                unsigned cr = columns;
                for (unsigned r = queue; __any_sync(0xffffffffu, r < end); r += 4 * ROW, cr += 4 * 64)
#pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const float queued = shared_f32(r + q * ROW);
                        push_hit(hits, at, word_at, r + q * ROW < end ? queued : 0.f, shared_u16(cr + q * 64), least, K, 32 * LD * 4);
                    }
            }
            const bool crowded = hits > K;
            uint32_t word[KMAX];
#pragma unroll
            for (int r = 0; r < KMAX; r++) word[r] = r < K && r < hits ? __float_as_uint(tile[NX + r][lane][slot]) : EMPTY;
            twice = __any_sync(0xffffffffu, twice);
#pragma unroll
            for (int i = 0; i < KMAX; i++) {
                if (i >= K) break;
                const float d = i < hits ? mine[i * 32] : -1.f;
                int rank = 0;
#pragma unroll
                for (int r = 0; r < KMAX; r++) rank += top[0].v[r] > d;
                if (twice)                                   // of equal values, the later column comes first
#pragma unroll
                    for (int r = 0; r < KMAX; r++)
                        if (r < K && r < hits && i < hits && mine[r * 32] == d && (word[r] & ~SNB_SIGN_BIT) > (word[i] & ~SNB_SIGN_BIT)) rank++;
                tile[NX + (i < hits ? min(rank, K - 1) : i)][lane][slot] = __uint_as_float(word[i]);
            }
            if (__any_sync(0xffffffffu, live && crowded))
                ordered_positions<KMAX, LD>(a.cand + (size_t)j * a.lcap, cnt, xt, live ? least : 0.f, K, tile + NX, slot);
        }
    }
    if (chain) {
        if (last_warp(&arrived) && lane == 0) {
            const unsigned mask = *(volatile unsigned*)&failed;
            if (mask) a.fail[atomicAdd(a.counters + FAILED, 1u)] = make_int4(s, n0, (int)mask, 0);
        }
        return;
    }
    __syncthreads();
    emit_tile<NX, NX, 0, SORT_SLOTS>(p, tile, s, n0, failed);
    const int col = tid % SORT_SLOTS, r = tid / SORT_SLOTS, b = s * 32 + r, n = n0 + col;
    if (POS && b < p.B && n < p.CO)
        for (int t = 0; t < K; t++) {
            const uint32_t word = __float_as_uint(tile[NX + t][r][col]);
            p.pos[((size_t)t * p.B + b) * p.CO + n] = word == EMPTY ? 0 : (int)word;       // fewer than K values above 0
        }
    if (tid == 0 && failed) a.fail[atomicAdd(a.counters + FAILED, 1u)] = make_int4(s, n0, (int)failed, 0);
}

}  // namespace
}  // namespace snb

#include "prune_redo.cuh"

namespace snb {

namespace {

// ---- host side ----------------------------------------------------------------------------------

int tensors(const PruneProblem& p) { return (p.x ? 1 : 0) + (p.xl ? 2 : 0); }
bool with_words(const PruneProblem& p) { return p.pos || p.posl || p.post; }

// How many columns must reach the threshold.  Without masks K: the K-th largest value of every row then
// reaches it by construction.  With column lists the m columns may all be missing from a sub-batch's list; m is chosen so
// that this happens to about one output in 10^7 for random lists, and such outputs go to prune_redo.
int threshold_rank(const PruneProblem& p) {
    int m = p.K;
    if (p.ci || p.kept) {
        const double gone = 1.0 - (double)(p.kept ? p.kept : p.CI) / p.W_CI;
        m = 1;
        for (double all = gone; all > 1e-7 && m < 16; all *= gone) m++;
        if (m < p.K) m = p.K;
    }
    return m;
}
// List capacity: N(0,1)-like weights leave 35 columns on average for the maximum, 180 for ten values, 230 for rank 14.
int list_capacity(const PruneProblem& p) {
    const int m = threshold_rank(p);
    const int want = m <= 2 ? 192 : LONG_LIST;
    const int c = (p.W_CI + PAD - 1) / PAD * PAD;
    return c < want ? c : want;
}

size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }

size_t layout(const PruneProblem& p, char* base, PruneArgs* a) {
    const size_t S = (p.B + 31) / 32, NX = tensors(p), lcap = list_capacity(p), C = p.W_CI, J = p.W_CO;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        char* at = base + off;
        off += up256(bytes);
        return at;
    };
    const bool given = p.xt != nullptr;
    char* zeroed = take(64 + (given ? 0 : 2 * up256(sizeof(unsigned) * C)));    // counters and ranges: one memset
    char* xt = take(given ? 0 : sizeof(float) * S * C * NX * 32);
    char* inv = take(p.ci ? sizeof(int) * S * C : 0);
    char* cnt = take(sizeof(int) * J);
    char* tau = take(sizeof(float) * J);
    char* ub = take(sizeof(float) * J * (lcap / STEP));
    char* cand = take(sizeof(int2) * J * lcap);
    char* fail = take(sizeof(int4) * S * ((p.CO + 31) / 32) * (p.K > 1 ? 4 : 1));      // prune_sort: down to eight outputs per CTA
    const size_t ldr = (C + 3) / 4 * 4;
    const bool whole = !p.leave;                             // evaluated as a whole here, should it come to that
    char* xr = take(whole ? sizeof(float) * NX * S * 32 * ldr : 0);
    char* partial = take(p.K > 1 || !whole ? 0 : (with_words(p) ? 8 : 4) * NX * S * p.CO * 32);
    char* tile_done = take(p.K > 1 || !whole ? 0 : sizeof(unsigned) * S * ((p.CO + 127) / 128));
    if (a) {
        a->ldr = (int)ldr;
        a->xr = reinterpret_cast<float*>(xr);
        a->partial = partial;
        a->tile_done = reinterpret_cast<unsigned*>(tile_done);
        a->p = p;
        a->S = (int)S;
        a->NX = (int)NX;
        a->m = threshold_rank(p);
        a->lcap = (int)lcap;
        a->counters = p.counters ? p.counters : reinterpret_cast<unsigned*>(zeroed);
        a->hi = given ? p.hi : reinterpret_cast<unsigned*>(zeroed + 64);
        a->nlo = given ? p.nlo : reinterpret_cast<unsigned*>(zeroed + 64 + up256(sizeof(unsigned) * C));
        a->xt = given ? p.xt : reinterpret_cast<float*>(xt);
        a->inv = p.ci ? reinterpret_cast<int*>(inv) : nullptr;
        a->cnt = reinterpret_cast<int*>(cnt);
        a->tau = reinterpret_cast<float*>(tau);
        a->ub = reinterpret_cast<float*>(ub);
        a->cand = reinterpret_cast<int2*>(cand);
        a->fail = reinterpret_cast<int4*>(fail);
    }
    return off;
}

// Persistent grid: as many CTAs as fit.  FIT, for which the registers are allotted: one CTA of 512 filter threads, two where the stages of wide rows leave no room for
// more, three otherwise.
template <int R, int NIT, int FT, int STAGES, int NB, bool VEC, int FIT = FT == 512 ? 1 : NIT >= 4 ? 2 : 3>
cudaError_t launch_filter(const PruneArgs& a, cudaStream_t st) {
    constexpr auto bytes = [](int lcap) {
        return STAGES * R * NIT * FT * 16 + NB * R * (lcap * ((int)sizeof(int2) + (int)sizeof(float)) + lcap / STEP * (int)sizeof(float));
    };
    constexpr auto KERN = prune_filter<R, NIT, FT, STAGES, NB, VEC, FIT>;
    const int smem = bytes(a.lcap), threads = FT + 32 * NB * R;
    cudaError_t e = allow_smem<KERN, bytes(LONG_LIST)>();
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KERN, threads, smem);
    if (e != cudaSuccess) return e;
    const int steps = (a.p.W_CO + R - 1) / R, slots = sm_count() * (per_sm > 0 ? per_sm : 1);
    const int grid = steps < slots ? steps : slots;
    // Long lists: all for shared memory (32 x 1024 x 1024, ten and seventeen values 20.0 and 25.7 us, left alone 21.5 and 34.0).  Short ones leave the division as it is, and the
    // walk behind them has what they do not use (boxes with positions of 67 x 300 x 700 19.1 us, else 21.9; of 67 x 1024 x 1024 20.6, else 21.9).
    const int share = a.m > 2 ? l1_share(FIT, bytes(LONG_LIST), grid, 1) : -1;
    return launch_next_with(share, KERN, grid, threads, smem, st, a);
}

template <bool VEC>
cudaError_t filter(const PruneArgs& a, cudaStream_t st) {
    const int C = a.p.W_CI;
    // Narrow rows take two per step, for which three list buffers are too few where lists are long (us at 5120 rows, cold, rank 1 / 10; before: sweeps behind a barrier each,
    // four rows per step): 512 columns 12.5 / 22.7 with three, 12.3 / 18.1 with four, before 13.4 / 20.2; 1024 columns 14.0 / 23.7, 14.0 / 19.5, before 15.2 / 21.4; one
    // row per step 13.7 / 16.6 and 14.9 / 19.1.  Wider ones, one row per step, before -> now: 1500 18.1 -> 17.0 / 25.6 -> 21.4, 2048 19.1 -> 17.5 / 26.5 -> 22.1, 3000 22.0 ->
    // 20.5 / 30.1 -> 25.8, 4000 26.3 -> 26.4 / 34.3 -> 30.3.
    if (C <= 1024) return launch_filter<2, 1, 256, 3, 4, VEC>(a, st);
    if (C <= 2048) return launch_filter<1, 2, 256, 3, 4, VEC>(a, st);
    if (C <= 3072) return launch_filter<1, 3, 256, 3, 4, VEC>(a, st);
    if (C <= 4096) return launch_filter<1, 4, 256, 3, 4, VEC>(a, st);
    if (C <= 5120) return launch_filter<1, 5, 256, 3, 4, VEC>(a, st);
    // Copied by single floats three list buffers are better than four, and than 16 warps of fewer columns each (which let the walk start late, too): 3000 x 6001,
    // cold, rank 1 / 10, 30.3 / 35.6 us against 34.1 / 41.4 and 30.3 / 36.3; values with positions of 67 rows, W in L2, 40.6 against 40.8 and 43.5 in all.  By fours 3000 x 6000
    // 23.4 with four buffers, 27.3 with 16 warps.
    if (C <= 6144) return VEC ? launch_filter<1, 6, 256, 3, 4, true>(a, st) : launch_filter<1, 6, 256, 3, 3, false>(a, st);
    if (C <= 8192) return launch_filter<1, 4, 512, 3, 4, VEC>(a, st);
    return launch_filter<1, 6, 512, 3, 4, VEC>(a, st);
}

// As many CTAs of the redo kernel as fit: with nothing to redo they read a few counters and end.
template <auto KERN>
cudaError_t redo_grid(int threads, int smem, int* grid) {
    int per_sm = 0;
    const cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, KERN, threads, smem);
    *grid = sm_count() * (per_sm > 0 ? per_sm : 1);
    return e;
}

template <int NX, bool TRACK, bool LEAVE = false>
cudaError_t run_max(const PruneArgs& a, dim3 grid, cudaStream_t st) {
    constexpr int smem = redo_max_smem<NX, TRACK>();
    constexpr auto REDO = prune_redo_max<NX, TRACK, LEAVE>;
    cudaError_t e = allow_smem<REDO, smem>();
    if (e != cudaSuccess) return e;
    int redo = 0;
    if ((e = redo_grid<REDO>(REDO_THREADS, smem, &redo)) != cudaSuccess) return e;
    constexpr int tile = (TRACK ? 2 : 1) * NX * 32 * 33 * (int)sizeof(float);
    // By CTAs, divided / left alone.  Points with positions: 441 (200 x 2048 x 2000) 23.2 / 21.8 us, 480 (67 x 5120 x 5120) 42.4 / 42.2, 512 (512 x 1024 x 1024) 19.7 / 20.7,
    // 2560 72.2 / 72.9, masked 84.4 / 86.8; boxes with positions: 189 (67 x 2048 x 2000) 27.8 / 25.9, 224 24.8 / 24.8, 352 (512 x 300 x 700) 24.8 / 25.9, 480 49.9 / 52.2, 2560
    // 115 / 119; values: 512 19.6 / 18.9, 1008 (512 x 2048 x 2000) 27.9 / 26.9, 1120 47.7 / 47.8, 2560 (512 x 5120 x 5120) 58.8 / 60.1.  Boxes and points with boxes without
    // positions gain nothing (seven layers of 2560 441 / 439).
    constexpr float from = TRACK ? (NX == 1 ? 3.4f : 2) : 12;
    const int share = TRACK || NX == 1 ? l1_share(WALK_CTAS<NX, TRACK>, tile, (long long)grid.x * grid.y, from) : -1;
    if ((e = launch_next_with(share, prune_max<NX, TRACK>, grid, 256, 0, st, a)) != cudaSuccess) return e;
    return launch_next(REDO, redo, REDO_THREADS, smem, st, a);
}

// Eight outputs per CTA, a warp each.  With 32, four one after the other per warp, a few long CTAs end last: 8 / 32 outputs, values of K = 10
// 512 x 2048 x 2000 79.6 / 89.5 us, 512 x 5120 x 5120 215 / 225, K = 17 485 / 562; boxes of K = 10 119 / 127 and 333 / 332, K = 17 321 / 339 and
// 872 / 908, chained points and boxes of K = 10 243 / 249; positions of K = 11 64 x 1024 x 2048 53 / 88, 512 x 5120 x 5120 842 / 852.
template <int NX, int KMAX, bool POS>
cudaError_t run_sort(const PruneArgs& a, cudaStream_t st) {
    int redo = 0;
    cudaError_t e = redo_grid<prune_redo_sort<NX, KMAX, POS>>(256, 0, &redo);
    if (e == cudaSuccess) e = allow_smem<prune_sort<NX, KMAX, POS>, sort_walk_smem<NX, KMAX, POS>(KMAX)>();
    if (e != cudaSuccess) return e;
    const dim3 grid((a.p.CO + SORT_SLOTS - 1) / SORT_SLOTS, a.S);
    // By CTAs, divided / left alone: values of K = 10 250 (32 x 2048 x 2000) 27.9 / 25.8 us, 384 23.7 / 22.2, 750 32.0 / 31.9, 10240 202.5 / 202.9; boxes 384 30.9 / 29.0, 616 31.7 /
    // 32.9, 10240 315.5 / 319.5; points and boxes of five layers 1125 / 1138.  Positions of more than ten values, whose walks are long: 188 (32 x 9000 x 1500) 216 / 224, 264 49.7 / 50.6,
    // 10240 1109 / 1142.
    const int smem = sort_walk_smem<NX, KMAX, POS>(a.p.K);
    const int share = l1_share(SORT_CTAS<KMAX>, smem, (long long)grid.x * grid.y, POS && KMAX > 10 ? 1 : 3.4f);
    e = launch_next_with(share, prune_sort<NX, KMAX, POS>, grid, 256, smem, st, a);
    if (e != cudaSuccess) return e;
    if ((e = launch_next(prune_redo_sort<NX, KMAX, POS>, redo, 256, 0, st, a)) != cudaSuccess || !POS) return e;
    return sort_positions_if(a.p, a.counters + OVERFLOWED, st);
}

}  // namespace

bool prune_applies(const PruneProblem& p) {
    if (p.W_CI > MAX_COLUMNS) return false;
    if (p.ci && 5ll * p.CI < 2ll * p.W_CI) return false;
    if ((p.B + 31) / 32 > 65535) return false;
    // below these sizes it cannot pay; where it does is up to the caller (snb_prune_pays)
    const long long least = p.K > 1 ? 1ll << 20 : p.xl ? 4ll << 20 : 12ll << 20;
    if ((long long)p.B * p.CO * p.W_CI < least || p.W_CI < 128) return false;
    return layout(p, nullptr, nullptr) <= MOST_SCRATCH;
}

size_t prune_workspace_bytes(const PruneProblem& p) { return layout(p, nullptr, nullptr); }

cudaError_t prune_prepare(const PrunePrep& q, cudaStream_t st) {
    const dim3 grid((q.CI + 63) / 64, (q.B + 31) / 32);
    if (!q.x) prune_prep<2><<<grid, 256, 0, st>>>(q);
    else if (q.box || q.xl) prune_prep<3><<<grid, 256, 0, st>>>(q);
    else prune_prep<1><<<grid, 256, 0, st>>>(q);
    return launched();
}

cudaError_t prune_forward(const PruneProblem& p, void* ws, cudaStream_t st) {
    PruneArgs a{};
    layout(p, static_cast<char*>(ws), &a);
    const size_t C = p.W_CI;
    cudaError_t e = cudaSuccess;
    if (!p.counters) e = cudaMemsetAsync(a.counters, 0, 64 + (p.xt ? 0 : 2 * up256(sizeof(unsigned) * C)), st);
    if (e != cudaSuccess) return e;
    if (!p.xt) {
        // all bits set is a NaN (the dropped columns) and a -1 (inv, which lies behind xt)
        float* xt = const_cast<float*>(a.xt);
        if (p.ci && (e = cudaMemsetAsync(xt, 0xff, (char*)(a.inv + a.S * C) - (char*)xt, st)) != cudaSuccess) return e;
        PrunePrep q;
        q.x = p.x, q.xl = p.xl, q.xu = p.xu, q.ci = p.ci, q.inv = a.inv, q.B = p.B, q.CI = p.CI, q.W_CI = p.W_CI;
        q.xt = xt, q.hi = const_cast<unsigned*>(a.hi), q.nlo = const_cast<unsigned*>(a.nlo), q.general = a.counters + GENERAL;
        if ((e = prune_prepare(q, st)) != cudaSuccess) return e;
    }
    e = (C % 4 == 0) && aligned16(p.w) ? filter<true>(a, st) : filter<false>(a, st);
    if (e != cudaSuccess) return e;
    const dim3 grid((p.CO + 31) / 32, a.S);
    if (p.K == 1) {
        const bool track = with_words(p);
        if (p.leave) return run_max<1, false, true>(a, grid, st);
        if (a.NX == 1) return track ? run_max<1, true>(a, grid, st) : run_max<1, false>(a, grid, st);
        if (a.NX == 2) return track ? run_max<2, true>(a, grid, st) : run_max<2, false>(a, grid, st);
        return run_max<3, false>(a, grid, st);
    }
    if (p.K <= 10) {
        if (a.NX == 1) return p.pos ? run_sort<1, 10, true>(a, st) : run_sort<1, 10, false>(a, st);
        return a.NX == 2 ? run_sort<2, 10, false>(a, st) : run_sort<3, 10, false>(a, st);
    }
    if (a.NX == 1) return p.pos ? run_sort<1, 25, true>(a, st) : run_sort<1, 25, false>(a, st);
    return a.NX == 2 ? run_sort<2, 25, false>(a, st) : run_sort<3, 25, false>(a, st);
}

}  // namespace snb

// Whether the pruned form is the faster one for data that can be pruned (inputs in [0, 1], N(0, 1) weights).  B200, one call
// inside a graph, dense / pruned: values 9.0 / 17.1 us at 32 M terms, 12.2 / 17.9 at 64 M, 16.1 / 17.8 at 128 M, 42 / 20 at 512 M; with
// positions 12.7 / 16.8 at 32 M, 16.1 / 16.7 at 64 M, 22.3 / 17.4 at 128 M, the same with ascending lists 15.7 / 24.9 at 29 M, 19.2 / 25.7 at
// 58 M, 26.3 / 26.0 at 115 M, 39.6 / 27.0 at 230 M; bounds 18.0 / 18.1 at 2 M, 17.7 / 16.4 at 4 M,
// 24.0 / 18.4 at 32 M; ten largest 97 / 44 at 1 M.  It takes five launches however small the problem.
extern "C" int snb_prune_pays(int tensors, int K, int words, int B, int CO, int W_CI) {
    const long long terms = (long long)B * CO * W_CI;
    if (K > 1) return terms >= 1ll << 20;
    if (tensors != 1) return terms >= 4ll << 20;
    return terms >= (words ? 96ll << 20 : 160ll << 20);
}

// Scratch with which the `_ws` entry points evaluate a problem in the pruned form: tensors = 1 (point value),
// 2 (box) or 3 (both), K = 1 or the sort neuron's size, words = positions wanted, column_lists = kept-column
// lists given.  0: the problem is too small or too wide for it, the entry points then need no (other) scratch.
extern "C" size_t snb_prune_scratch_bytes(int tensors, int K, int words, int B, int CO, int CI, int W_CO, int W_CI,
                                          int column_lists) {
    if (B <= 0 || CO <= 0 || CI <= 0 || W_CO <= 0 || W_CI <= 0 || tensors < 1 || tensors > 3) return 0;
    static const float some = 0.f;
    static const int none = 0;
    snb::PruneProblem p;
    p.x = tensors != 2 ? &some : nullptr;
    p.xl = tensors != 1 ? &some : nullptr;
    p.ci = column_lists ? &none : nullptr;
    static int word = 0;
    p.pos = words ? &word : nullptr;
    p.B = B, p.CO = CO, p.CI = CI, p.W_CO = W_CO, p.W_CI = W_CI, p.K = K;
    return snb::prune_applies(p) ? snb::prune_workspace_bytes(p) : 0;
}
