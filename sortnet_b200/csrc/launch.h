// Host-side helpers shared by the entry points.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <mutex>

namespace snb {

// Records the last CUDA runtime error seen by an entry point of this thread.
void set_last_cuda_error(cudaError_t e);

// Called after every launch (or n of them): counts them (snb_launch_count) and returns the launch error, if any.
cudaError_t launched(int n = 1);

// Number of SMs of the current device (cached per device).
int sm_count();

// Lets KERN launch with up to MOST bytes of dynamic shared memory on the current device.  The attribute belongs to the
// function, not to a launch, and is shared by all host threads: it is set once, to the most that any launch
// of KERN asks for, so that threads with different sizes cannot take each other's limit away.
template <auto KERN, int MOST>
inline cudaError_t allow_smem() {
    static std::atomic<bool> done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (done[dev & 63].load(std::memory_order_acquire)) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(KERN, cudaFuncAttributeMaxDynamicSharedMemorySize, MOST);
    if (e == cudaSuccess) done[dev & 63].store(true, std::memory_order_release);
    return e;
}
constexpr int MOST_SMEM = 227 * 1024;        // what a CTA of sm_100a may have

// Launches KERN so that its CTAs may be set up while the kernel before it in the stream ends.  Every thread of it calls after_previous()
// (common.cuh) before it touches what that kernel writes or may still read.  For chains of kernels of 10 to 40 us, where 2 to 3 us from
// the end of one to the first loads of the next count: interval bounds of seven layers (24 launches) 540 -> 500 us, a training pass of
// six 777 -> 765 us, sort neurons with gradients 995 -> 953 us.
// share: percent of an SM's memory that shared memory should have, the rest being L1 (l1_share below); negative: as the kernel before left it.
template <typename... Params, typename... Args>
inline cudaError_t launch_next_with(int share, void (*kern)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const Args&... args) {
    cudaLaunchAttribute attributes[2];
    attributes[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attributes[0].val.programmaticStreamSerializationAllowed = 1;
    attributes[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attributes[1].val.sharedMemCarveout = share > 0 ? (unsigned)share : 0u;
    cudaLaunchConfig_t config = {};
    config.gridDim = grid, config.blockDim = block, config.dynamicSmemBytes = smem, config.stream = st;
    config.attrs = attributes, config.numAttrs = share < 0 ? 1 : 2;
    const cudaError_t e = cudaLaunchKernelEx(&config, kern, static_cast<Params>(args)...);
    const cudaError_t last = launched();                     // takes a failed launch's error away, so that no later call reports it
    return e != cudaSuccess ? e : last;
}
template <typename... Params, typename... Args>
inline cudaError_t launch_next(void (*kern)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, const Args&... args) {
    return launch_next_with(-1, kern, grid, block, smem, st, args...);
}

// The share with which `ctas` CTAs of `bytes` of shared memory fit an SM and the rest is L1, for a grid of `grid` CTAs.  Left alone, an SM stays as the
// kernel before wanted it, and in a chain that is a filter with its stages: the list walks behind it, which live on L1, took 50 instead of
// 43 us per layer of a training pass.  A grid of less than `from` CTAs per SM is left alone: it has little to gain, and dividing the memory anew
// takes 1 to 2 us (four layers of 28 rows and 832 outputs 95 us, with all of them divided 98).
inline int l1_share(int ctas, int bytes, long long grid, float from) {
    const int room = ctas * (bytes + 1024), all = 228 * 1024;
    return (float)grid < from * (float)sm_count() ? -1 : room >= all ? 100 : (100 * room + all - 1) / all;
}

// Values with positions of small problems by one launch of a warp per row and four outputs, instead of tiles, partial results and a
// second pass.  B200, launches inside a graph, tiles / warps.  Points: 18.4 / 2.5 us at 9 x 97 x 33, 11.5 / 2.7 at 32 x 256 x 128,
// 11.7 / 4.5 at 64 x 256 x 256, 11.1 / 6.1 at 16 x 512 x 1024, 12.3 / 7.2 at 32 x 1000 x 250; boxes: 44.2 / 3.1 at 9 x 97 x 33, 82.4 / 5.3
// at 32 x 256 x 128, 324 / 15 at 9 x 1000 x 200.  The limits: outputs, each of which ends in a reduction over its warp (128 K of them at
// 64 columns 13.9 / 13.2 and 22.8 / 17.9; 262 K at 8 columns 15.4 / 21.6 and 12.7 / 27.9); terms (12.1 / 9.3 at 64 x 1024 x 256, but 18.0 / 28.1
// at 512 x 128 x 512); and, for points, whose tiles share long rows out, the columns (4 x 5120 x 64: 12.2 / 19.5, boxes 1602 / 63).
constexpr long long SMALL_TERMS = 8ll << 20, SMALL_OUTPUTS = 32ll << 10;
constexpr int SMALL_COLUMNS = 1024;

inline bool small_problem(int B, int CO, int CI) { return (long long)B * CO <= SMALL_OUTPUTS && (long long)B * CO * CI <= SMALL_TERMS; }

inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace snb

#define SNB_CUDA(...)                          \
    do {                                       \
        cudaError_t _e = (__VA_ARGS__);        \
        if (_e != cudaSuccess) {               \
            snb::set_last_cuda_error(_e);      \
            return SNB_ERR_CUDA;               \
        }                                      \
    } while (0)
