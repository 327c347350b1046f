// shared_mem.cuh -- dynamic shared memory beyond the default of a launch, for both translation units.
// The allowance belongs to the CUDA context (another device, or a host's own context, has its own), so
// both functions ask for it at every launch.  They clear the error that they return.
#pragma once
#include <cuda_runtime.h>

#include <mutex>

namespace wfs {
// Launches of `kern` may take `bytes`, the same at every call for one kernel (57 ns).
template <typename K>
cudaError_t allow_shared(K kern, size_t bytes)
{
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) cudaGetLastError();
    return e;
}

// The same for kernels whose size differs from call to call: looked up (280 ns) and only ever raised, so
// that threads with different sizes do not lower each other's.
template <typename K>
cudaError_t raise_shared(K kern, size_t bytes)
{
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    cudaFuncAttributes now;
    cudaError_t e = cudaFuncGetAttributes(&now, kern);
    if (e == cudaSuccess && now.maxDynamicSharedSizeBytes >= (int)bytes) return e;
    if (e == cudaSuccess) return allow_shared(kern, bytes);
    cudaGetLastError();
    return e;
}
}  // namespace wfs
