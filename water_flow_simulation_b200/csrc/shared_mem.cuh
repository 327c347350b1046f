// shared_mem.cuh -- dynamic shared memory beyond the default of a launch, for both translation units.
#pragma once
#include <cuda_runtime.h>

#include <mutex>

namespace wfs {
// Lets launches of `kern` in the current context take `bytes` of dynamic shared memory.  The allowance
// is the context's, so it is looked up there (another device, or a host's own context, has its own);
// it is only ever raised, so threads that launch the kernel with different sizes do not lower each
// other's.  Clears the error it returns.
template <typename K>
cudaError_t allow_shared(K kern, size_t bytes)
{
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    cudaFuncAttributes now;
    cudaError_t e = cudaFuncGetAttributes(&now, kern);
    if (e == cudaSuccess && now.maxDynamicSharedSizeBytes < (int)bytes)
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}
}  // namespace wfs
