// tensor_map.cuh -- the driver's tensor-map encoder.
#pragma once
#include <cuda.h>
#include <cuda_runtime_api.h>

namespace wfs {
using PfnEncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                    const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                    CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
// cuTensorMapEncodeTiled through the runtime's driver entry point (the library links no libcuda).
// Threads that ask while the first one is still looking it up wait for it.
inline PfnEncodeTiled encode_tiled()
{
    static const PfnEncodeTiled fn = [] {
        void* p = nullptr;
        const bool found = cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault,
                                                            nullptr) == cudaSuccess;
        return found ? reinterpret_cast<PfnEncodeTiled>(p) : nullptr;
    }();
    return fn;
}
}  // namespace wfs
