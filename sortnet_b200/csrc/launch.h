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
