// Grid-wide barrier of persistent cooperative kernels: every CTA is resident
// (cooperative launch), one atomic add per CTA, one polling thread per CTA.
// The wait is bounded; a wait that runs out reports failure to every thread
// of its CTA, which then leaves the kernel (the others' waits run out too).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace hyt::dev {

constexpr uint32_t kGridSpinLimit = 1u << 25;  // polls of ~0.5 us: far above any phase of an in-HBM solve

// `count` grows by gridDim.x per barrier and starts at 0; `round` counts the
// barriers passed so far (the same in every thread).  The fences make every
// thread's earlier writes visible to all threads after the barrier, also
// through L1 (plain loads; read-only-path loads of such data are not allowed).
__device__ __forceinline__ bool grid_sync(uint32_t *count, uint32_t &round) {
    __syncthreads();
    bool ok = true;
    if (threadIdx.x == 0) {
        __threadfence();
        const uint32_t want = (round + 1) * gridDim.x;
        uint32_t seen = atomicAdd(count, 1u) + 1u;
        uint32_t polls = 0;
        while (static_cast<int32_t>(seen - want) < 0) {
            if (++polls > kGridSpinLimit) {
                ok = false;
                break;
            }
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(count) : "memory");
        }
        __threadfence();
    }
    ++round;
    return __syncthreads_and(ok) != 0;
}

}  // namespace hyt::dev
