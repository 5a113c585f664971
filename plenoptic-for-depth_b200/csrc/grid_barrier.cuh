// grid_barrier.cuh -- barrier over the blocks of a cooperative launch.
#pragma once
#include <cuda_runtime.h>
#include "pm_kernels.h"

namespace pfd {

// Every thread of the grid calls it; bar counts arrivals from zero, target is the number
// of blocks times the calls so far.  The wait is bounded (about 2^22 polls): a block that
// gives up records PFD_DEVERR_TMA_TIMEOUT and gets false.
__device__ __forceinline__ bool grid_barrier(unsigned int* bar, unsigned int target, int* err)
{
    __syncthreads();
    int ok = 1;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(bar, 1u);
        ok = 0;
        for (unsigned int it = 0; it < (1u << 22); ++it) {
            if (*(volatile unsigned int*)bar >= target) { ok = 1; break; }
            if (it > 32) __nanosleep(64);
        }
        __threadfence();
        if (!ok) atomicOr(err, PFD_DEVERR_TMA_TIMEOUT);
    }
    return __syncthreads_and(ok) != 0;
}

}  // namespace pfd
