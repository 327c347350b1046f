// channels.cuh -- channels of one voxel of a channels-last grid, in memory and as floats.
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

namespace wfs {
// N channels of a voxel as floats and back: one 16- or 2 x 16-byte access for N = 8 (aligned rows of a
// multiple of 8 channels), one element for N = 1.  Wide accesses are to memory only: a local float array
// is aligned to 4 bytes.
template <int N>
__device__ __forceinline__ void load_n(float (&v)[N], const __nv_bfloat16* p)
{
    if constexpr (N == 8) {
        const uint4 u = __ldg(reinterpret_cast<const uint4*>(p));
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            v[2 * j] = __uint_as_float(w[j] << 16);
            v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
        }
    } else {
        v[0] = __bfloat162float(*p);
    }
}
template <int N>
__host__ __device__ __forceinline__ void load_n(float (&v)[N], const float* p)
{
    if constexpr (N == 8) {
        const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
        v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
        v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
        v[0] = *p;
    }
}
template <int N>
__host__ __device__ __forceinline__ void store_n(__nv_bfloat16* p, const float (&v)[N])
{
    if constexpr (N == 8) {
        __align__(16) __nv_bfloat16 h[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) h[j] = __float2bfloat16_rn(v[j]);
        *reinterpret_cast<uint4*>(p) = *reinterpret_cast<uint4*>(h);
    } else {
        *p = __float2bfloat16_rn(v[0]);
    }
}
template <int N>
__host__ __device__ __forceinline__ void store_n(float* p, const float (&v)[N])
{
    if constexpr (N == 8) {
        reinterpret_cast<float4*>(p)[0] = make_float4(v[0], v[1], v[2], v[3]);
        reinterpret_cast<float4*>(p)[1] = make_float4(v[4], v[5], v[6], v[7]);
    } else {
        *p = v[0];
    }
}
}  // namespace wfs
