// Launches of the per-cell kernels, one translation unit per precision.
#pragma once

#include <cuda_runtime.h>

#include <atomic>
#include <utility>
#include <vector>

#include "solve.h"

namespace wcb {

// Start/end events of the four per-cell kernels (LoS+transmission,
// reflection, diffraction, finalize), each recorded on the kernel's stream.
struct ComponentEvents {
    cudaEvent_t start[4] = {nullptr, nullptr, nullptr, nullptr};
    cudaEvent_t end[4] = {nullptr, nullptr, nullptr, nullptr};
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> vis;  // around each diffraction visibility launch
};

// Raises a kernel's dynamic shared memory limit to `bytes`, once per device: the
// attribute belongs to the device that is current when it is set.  `done` holds
// a bit per device.
inline void raise_shared_limit(const void* kernel, int bytes, std::atomic<unsigned long long>& done) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return;
    const unsigned long long bit = 1ull << (device & 63);
    if (done.load(std::memory_order_acquire) & bit) return;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess)
        done.fetch_or(bit, std::memory_order_release);
}

struct DiffractionPlan {
    int chunk = 0;           // edges per chunk
    int chunks = 0;          // chunks covering the scene's edge count
    unsigned* words = nullptr;
    void* carry = nullptr;   // running per-cell sums between chunks (chunks > 1)
    bool run_vis = true;     // false when this frequency block reuses the words
};

// Per-cell kernels of `nf` frequencies (1 to 4), instantiated for float and
// double in solve_f32.cu and solve_f64.cu.
template <typename T>
void launch_components(const MainParams& q, int nf, unsigned blocks, int sdepth, size_t stack_bytes, cudaStream_t stream,
                       cudaStream_t side, ComponentEvents* evs, const DiffractionPlan& dp);

}  // namespace wcb
