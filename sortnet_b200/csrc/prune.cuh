// Exact pruned evaluation of the max-type distance operators (l-infinity values, positions, interval
// bounds, sort neurons): only the columns of W that can matter are looked at per row of the batch.
//
// max_c |x[b,c] - w[j,c]| over thousands of columns is decided by a handful of them.  With lo[c] and
// hi[c] the smallest and largest value of column c of the input over the batch,
//     L[j,c] = max(lo - w, w - hi, 0)  <=  |x[b,c] - w[j,c]|  <=  U[j,c] = max(hi - w, w - lo)
// holds for every row b, in rounded fp32 arithmetic too (rounding is monotone).  A column whose U lies
// below a threshold tau that the result reaches cannot be the maximum, nor tie with it.  Steps:
//   prune_prep     transposes the input to xt[sub-batch][column][tensor][32 rows] (NaN where a column
//                  was dropped or a row does not exist: NaN never enters a maximum) and collects lo / hi;
//   prune_filter   reads W once: per row j the threshold tau (the m-th largest L among disjoint
//                  groups of columns) and the list of columns with U >= tau, largest U first;
//   prune_max / prune_sort   one warp per (sub-batch, output), lane = row: walks the list until no
//                  remaining U can change any row, and CHECKS that every row's result (its K-th
//                  largest value for the sort neuron) reaches tau.  Outputs that do not are recorded;
//   prune_redo     evaluates the recorded outputs over all columns.
// The result is exact whatever the data: the thresholds only decide how many columns are read.  Where
// too many lists overflow (inputs spread as wide as the weights), nothing is walked and prune_redo evaluates
// the layer as a whole with register tiles.
#pragma once
#include "common.cuh"
#include "launch.h"

namespace snb {

struct PruneProblem {
    // inputs: x [B, CI] (compact over ci when given) and / or the ends of a box xl, xu [B, W_CI]
    const float* x = nullptr;
    const float* xl = nullptr;
    const float* xu = nullptr;
    const float* w = nullptr;   // [W_CO, W_CI]
    const int* ci = nullptr;    // [S, CI] kept columns per sub-batch, or null
    const int* co = nullptr;    // [S, CO] kept rows of W per sub-batch, or null
    int B = 0, CO = 0, CI = 0, W_CO = 0, W_CI = 0;
    // outputs [B, CO]; positions optional
    float* y = nullptr;
    float* yl = nullptr;
    float* yu = nullptr;
    int* pos = nullptr;         // x: argmax words ([K][B][CO] for the sort neuron)
    int* posl = nullptr;        // box: words of both bounds
    int* posu = nullptr;
    int K = 1;                  // 1: maximum; 2..25: sort neuron of that many values
    float q = 0.f;

    // Chain form (csrc/mlp.cu): one layer hands its result to the next without a row-major copy in between.
    // Input: xt [S][W_CI][tensors][32] and the order codes of its column ranges, as prune_prep leaves them (x, xl, xu
    // then only say which tensors there are; ci and co are null); kept = columns that every sub-batch holds.
    const float* xt = nullptr;
    const unsigned* hi = nullptr;
    const unsigned* nlo = nullptr;
    int kept = 0;
    // Output: yt [S][CO][tensors][32], NaN in rows past the batch and in outputs that `keep` [S][CO] drops; ranges
    // (zeroed before), sums over the rows of a sub-batch in row order [S][CO], words [S][CO][32]
    // (SNB_NO_GRAD_ID where dropped).  y = (y - mean[j]) + bias[j] before it is written anywhere (either may be null).
    float* yt = nullptr;
    unsigned* yhi = nullptr;
    unsigned* ynlo = nullptr;
    float* part = nullptr;
    int* post = nullptr;
    const unsigned char* keep = nullptr;
    const int* out_list = nullptr;      // [S][out_kept] the outputs that `keep` keeps (null without `keep`)
    int out_kept = 0;
    const float* mean = nullptr;
    const float* bias = nullptr;
    unsigned* counters = nullptr;       // four zeroed counters of the caller's, or null: those in the workspace
    const int* kept_list = nullptr;     // [S][kept] kept columns: the first one is the position of an output at its floor
    bool leave = false;                 // maxima of points, no positions: a layer that would be evaluated as a whole is left to the caller (prune_left)
};

// Transposes x (or x and the box [max(x - eps, down), min(x + eps, up)], or given box ends) to the chain form.
struct PrunePrep {
    const float* x = nullptr;
    const float* xl = nullptr;
    const float* xu = nullptr;
    const int* ci = nullptr;
    int* inv = nullptr;         // with ci: -1 before
    int B = 0, CI = 0, W_CI = 0;
    bool box = false;           // make xl, xu from x
    float eps = 0.f, down = 0.f, up = 0.f;
    float* xt = nullptr;
    unsigned* hi = nullptr;     // zeroed before
    unsigned* nlo = nullptr;
    unsigned* general = nullptr;    // with ci: flags of what its lists are not (zeroed before)
};
cudaError_t prune_prepare(const PrunePrep& q, cudaStream_t st);

// Order-preserving codes of floats; 0 stands for "no value" (NaN).
__device__ __forceinline__ unsigned order_code(float f) {
    const unsigned b = __float_as_uint(f);
    return f != f ? 0u : ((b & 0x80000000u) ? ~b : (b | 0x80000000u));
}
__device__ __forceinline__ float decode(unsigned e) {   // 0 -> NaN
    return __uint_as_float((e & 0x80000000u) ? (e ^ 0x80000000u) : ~e);
}

// Above 1 / 32 of overflowed lists the layer is evaluated as a whole: one output by itself costs about 12 times its part
// of the whole (512 x 5120 x 5120 with positions).
__host__ __device__ __forceinline__ bool prune_gives_up(unsigned overflowed, int W_CO) { return (long long)overflowed * 32 > W_CO; }

// What the counters of a problem count, at the start of its workspace (unless they are the caller's): outputs left over by the walks; rows of W whose list
// overflowed; what the column lists are not: in ascending order, or (the transposed input has one place per column) without an entry that
// comes twice.
enum { FAILED = 0, OVERFLOWED = 1, GENERAL = 2 };
constexpr unsigned LIST_ORDER = 1u, LIST_TWICE = 2u;
__device__ __forceinline__ bool prune_left(const unsigned* counters, bool column_lists, int W_CO) {
    return (column_lists && (counters[GENERAL] & LIST_TWICE)) || prune_gives_up(counters[OVERFLOWED], W_CO);
}

// y and pos of a sort neuron by the kernels of sort_neuron.cu if the layer is to be evaluated as a whole, nothing otherwise.
cudaError_t sort_positions_if(const PruneProblem& p, const unsigned* overflowed, cudaStream_t st);

// Whether the pruned evaluation takes this problem (sizes only), and its scratch.
bool prune_applies(const PruneProblem& p);
size_t prune_workspace_bytes(const PruneProblem& p);
// ws: prune_workspace_bytes(p) bytes, 16-byte aligned.
cudaError_t prune_forward(const PruneProblem& p, void* ws, cudaStream_t st);
inline bool prune_fits(const PruneProblem& p, const void* ws, size_t ws_bytes) {
    return ws && aligned16(ws) && prune_applies(p) && ws_bytes >= prune_workspace_bytes(p);
}

}  // namespace snb
