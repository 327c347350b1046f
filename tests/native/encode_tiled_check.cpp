// Host-side check of encode_tiled (tensor_map.cuh) with a driver entry point that takes a while to be
// found: eight threads ask for the first time at once, and every one must get it.  Prints how many did.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <cstring>
#include <thread>
#include <vector>
#include "../../water_flow_simulation_b200/csrc/tensor_map.cuh"

static CUresult found(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                      const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                      CUtensorMapL2promotion, CUtensorMapFloatOOBfill)
{
    return CUDA_SUCCESS;
}
extern "C" cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** fn, unsigned int, unsigned long long,
                                                        cudaDriverEntryPointQueryResult*)
{
    std::this_thread::sleep_for(std::chrono::milliseconds(200));
    *fn = std::strcmp(name, "cuTensorMapEncodeTiled") ? nullptr : reinterpret_cast<void*>(&found);
    return cudaSuccess;
}

int main()
{
    std::atomic<int> ready{0}, got{0};
    std::vector<std::thread> all;
    for (int t = 0; t < 8; ++t)
        all.emplace_back([&] {
            ++ready;
            while (ready < 8) std::this_thread::yield();
            if (wfs::encode_tiled() == &found) ++got;
        });
    for (auto& t : all) t.join();
    std::printf("%d\n", got.load());
    return 0;
}
