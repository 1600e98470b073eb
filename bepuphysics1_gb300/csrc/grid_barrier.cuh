// Bounded grid barrier for the cooperative kernels.
#pragma once

#include <cuda_runtime.h>

#include "../../include/bepugpu.h"

namespace bepugpu {

// Thread 0 of each block arrives on a counter; the last arrival resets it and
// bumps the generation.  A wait that outlives kBarrierSpinLimit polls sets
// *err and the kernel returns.  Writes before the barrier are visible after it
// to loads that do not come from a stale L1 line.
constexpr long long kBarrierSpinLimit = 1ll << 24;
__device__ __forceinline__ bool GridBarrier(unsigned int* counter, volatile unsigned int* generation,
                                            unsigned int& localGen, volatile int* err) {
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned int g = localGen;
        __threadfence();
        unsigned int arrived = atomicAdd(counter, 1u);
        if (arrived == gridDim.x - 1) {
            atomicExch(counter, 0u);
            __threadfence();
            atomicAdd((unsigned int*)generation, 1u);
        } else {
            long long spins = 0;
            while (*generation == g) {
                if (++spins > kBarrierSpinLimit) {
                    *err = BEPUGPU_TIMEOUT;
                    break;
                }
                if (*err) break;
                __nanosleep(64);
            }
        }
        __threadfence();
    }
    localGen++;
    __syncthreads();
    return *err == 0;
}

}  // namespace bepugpu
