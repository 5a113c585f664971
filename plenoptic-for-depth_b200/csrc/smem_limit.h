// smem_limit.h -- dynamic shared memory above the default 48 KB.
#pragma once
#include <cuda_runtime.h>

namespace pfd {

// Lets kernel k be launched with `smem` bytes.  The limit belongs to the kernel, not to a
// launch: one made for each call's own size would be taken back by another thread's smaller
// call before this one's launch.  So it stays as it is up to the default 48 KB, and goes to
// all that one CTA may have above, for good.
inline cudaError_t allow_dynamic_smem(const void* k, int smem)
{
    cudaFuncAttributes a;
    const cudaError_t e = cudaFuncGetAttributes(&a, k);
    if (e != cudaSuccess) return e;
    if (smem + (int)a.sharedSizeBytes <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - (int)a.sharedSizeBytes);
}

}  // namespace pfd
