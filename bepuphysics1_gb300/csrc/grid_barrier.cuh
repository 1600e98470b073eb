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

// The same for a kernel that knows its number of barriers: `counter` only
// counts up while it runs, so a block that has arrived waits for the counter
// itself, with no reset and no generation behind the last arrival.  `arrived`
// is the blocks' total before this barrier.  FinishGridBarriers, on every
// block's way out, lets the last one put the counter back to zero.
__device__ __forceinline__ bool CountBarrier(unsigned int* counter, unsigned int& arrived, volatile int* err) {
    arrived += gridDim.x;
    bool ok = true;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(counter, 1u);
        for (long long spins = 1; *(volatile unsigned int*)counter < arrived; spins++) {
            if (spins > kBarrierSpinLimit) *err = BEPUGPU_TIMEOUT;
            // another block's error is looked for now and then: a load a poll is a trip through L2
            if ((spins & 63) == 0 && *err) {
                ok = false;
                break;
            }
        }
        __threadfence();
    }
    return __syncthreads_and(ok);
}
__device__ __forceinline__ void FinishGridBarriers(unsigned int* counter, unsigned int arrived) {
    if (threadIdx.x == 0 && atomicAdd(counter, 1u) == arrived + gridDim.x - 1) atomicExch(counter, 0u);
}

}  // namespace bepugpu
