// The meeting of a cooperative launch's blocks between the steps of an iteration.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace mars {

constexpr long long kBarrierCycles = 4000000000ll;  // ~2 s

// All blocks arrive, then leave: the counter only grows during a launch.  A wait that runs out
// sets the error word and the counter's top bit, which lets everybody through.
__device__ __forceinline__ void grid_meet(uint32_t* counter, uint32_t target, int* err) {
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
        const long long t0 = clock64();
        for (;;) {
            uint32_t v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(counter) : "memory");
            if (v >= target) break;
            if (clock64() - t0 > kBarrierCycles) {
                atomicOr(err, 256);
                atomicOr(counter, 0x80000000u);
                break;
            }
        }
    }
    __syncthreads();
}

// A launch's last words: the last block through leaves both words (arrivals, blocks through) as
// they were, zero.
__device__ __forceinline__ void grid_leave(uint32_t* sync) {
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (atomicAdd(sync + 1, 1u) == gridDim.x - 1) {
            sync[0] = 0u;
            sync[1] = 0u;
        }
    }
}

}  // namespace mars
