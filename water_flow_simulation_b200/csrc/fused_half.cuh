// fused_half.cuh -- the split (work-list) pipeline over 16-bit population storage.
// Included inside the anonymous namespace of lbm_kernels.cu, after fused_split.cuh.
//
// Storage: h_i = fp16_rn((f_i - w_i) * scale) in the SoA layout of the float path
// (h[i*cells + c]), scale a per-lattice power of two.  Collision stays in FP32.  A step
// moves 2 x 19 x 2 = 76 bytes per cell instead of 152.
//
// Work lists are built over row segments of 32*cpl cells (cpl = cells_per_lane 2, 4 or 8:
// 64, 128 or 256 cells), and pitch is a multiple of 8 so every 8-cell group is one aligned
// 16-byte vector.
//   k_rows_h_plain    plain segments: a lane moves VP = 4 (or 8) cells with one 8-byte (16-byte)
//                     load/store per direction, 32*cpl/VP lanes per segment; the +-1 x
//                     neighbours are one shuffle and VP/2 byte permutes on the packed halves;
//                     the collision works on deviations directly (moments of f - w), two
//                     cells at a time in packed float32 (collide2).
//   k_edge            edge segments (fused_edge.cuh) and
//   k_cells           special segments (fused_cells.cuh), on populations.
#pragma once

// Pull of direction I for the VP cells (VP = 4 or 8) of a lane in an interior row, packed:
// word j of h[I] holds cells 2j (low half) and 2j+1 (high half).  A +x mover takes element
// x-1: word j = (high half of source word j-1, low half of source word j); word -1 is the
// left lane's last word (at a segment's first lane: the 4-byte word just left of the
// segment).  A -x mover takes element x+1 symmetrically, word VP/2 from the right lane.
// G lanes share a segment (shuffles of width G).  All loads are issued, in order, before the
// first shuffle waits for one: left to the compiler, the 16-bit kernel waited for early loads
// with later ones not yet issued (VP = 8: 366 us against 404 on the 36M-cell reach).
template <int VP> struct HVec;
template <> struct HVec<4> {
    static __device__ __forceinline__ void store(__half* p, const uint32_t (&t)[2])
    {
        *reinterpret_cast<uint2*>(p) = make_uint2(t[0], t[1]);
    }
};
// Stores are plain write-back stores: for this kernel they measured 2.7 % faster than
// streaming (.cs) stores on reach36m, while the float32 kernels keep .cs stores (6 % slower
// without).
template <> struct HVec<8> {
    static __device__ __forceinline__ void store(__half* p, const uint32_t (&t)[4])
    {
        *reinterpret_cast<uint4*>(p) = make_uint4(t[0], t[1], t[2], t[3]);
    }
};

// Coherent packed loads of VP cells and of one 4-byte word (hcoh; __half goes through ld_ordered).
template <int VP>
__device__ __forceinline__ void hload(uint32_t (&t)[VP / 2], const hcoh* p)
{
    if constexpr (VP == 8) {
        const uint4 v = __ldcg(reinterpret_cast<const uint4*>(p));
        t[0] = v.x; t[1] = v.y; t[2] = v.z; t[3] = v.w;
    } else {
        const uint2 v = __ldcg(reinterpret_cast<const uint2*>(p));
        t[0] = v.x; t[1] = v.y;
    }
}
__device__ __forceinline__ uint32_t hword(const hcoh* p) { return __ldcg(reinterpret_cast<const unsigned int*>(p)); }

template <int I, int VP, typename T>
__device__ __forceinline__ void hpull_load(uint32_t (&h)[Q][VP / 2], uint32_t (&e)[Q], const T* __restrict__ own_ptr,
                                           const PullOffsets& po, int gl, int G, bool lid)
{
    const T* src = own_ptr + pull_offset<I>(po, lid);
    e[I] = 0;
    if constexpr (std::is_same<T, __half>::value) {
        ld_ordered(h[I], src);
        if constexpr (cx(I) == 1) ld_ordered_if(gl == 0, e[I], src - 2);
        if constexpr (cx(I) == -1) ld_ordered_if(gl == G - 1, e[I], src + VP);
    } else {
        hload<VP>(h[I], src);
        if constexpr (cx(I) == 1) if (gl == 0) e[I] = hword(src - 2);
        if constexpr (cx(I) == -1) if (gl == G - 1) e[I] = hword(src + VP);
    }
}
template <int I, int VP, int G>
__device__ __forceinline__ void hpull_shift(uint32_t (&h)[Q][VP / 2], const uint32_t (&e)[Q], int gl)
{
    constexpr int NW = VP / 2;
    if constexpr (cx(I) == 1) {
        uint32_t prev = __shfl_up_sync(0xffffffffu, h[I][NW - 1], 1, G);
        if (gl == 0) prev = e[I];
#pragma unroll
        for (int j = NW - 1; j > 0; --j) h[I][j] = __byte_perm(h[I][j - 1], h[I][j], 0x5432);
        h[I][0] = __byte_perm(prev, h[I][0], 0x5432);
    } else if constexpr (cx(I) == -1) {
        uint32_t next = __shfl_down_sync(0xffffffffu, h[I][0], 1, G);
        if (gl == G - 1) next = e[I];
#pragma unroll
        for (int j = 0; j < NW - 1; ++j) h[I][j] = __byte_perm(h[I][j], h[I][j + 1], 0x5432);
        h[I][NW - 1] = __byte_perm(h[I][NW - 1], next, 0x5432);
    }
}
template <int VP, int G, typename T, int... Is>
__device__ __forceinline__ void hpull_all(std::integer_sequence<int, Is...>, uint32_t (&h)[Q][VP / 2],
                                          const T* __restrict__ own_ptr, const PullOffsets& po, int gl,
                                          bool lid)
{
    uint32_t e[Q];
    (hpull_load<Is, VP, T>(h, e, own_ptr, po, gl, G, lid), ...);
    (hpull_shift<Is, VP, G>(h, e, gl), ...);
}

// One plain segment (row-segment id `id`) for the G lanes of a group: lane gl of the group
// moves VP cells.  Every lane of the warp calls it together (shuffles); `store` false: the
// group recomputes a segment another group owns and writes nothing.
template <int VP, int G, bool OUT, bool AVG, typename T = __half>
__device__ __forceinline__ void h_plain_segment(const lbm_lattice& L, const PullOffsets& po,
                                                const T* __restrict__ fs, T* __restrict__ fd, float scale,
                                                uint32_t id, int gl, bool store)
{
    constexpr int NW = VP / 2, SEG = VP * G;
    const int nseg = (L.pitch + SEG - 1) / SEG;
    const long long S = L.cells;
    const float inv_scale = 1.0f / scale;
    int seg, y, z;
    decode_row(id, nseg, L.ny, seg, y, z);
    const long long own = ((long long)z * L.ny + y) * L.pitch + seg * SEG + gl * VP;
    uint32_t h[Q][NW];
    hpull_all<VP, G, T>(std::make_integer_sequence<int, Q>{}, h, fs + own, po, gl, z == L.nz - 1);
    float R[VP], UX[VP], UY[VP], UZ[VP];
#pragma unroll
    for (int p = 0; p < NW; ++p) {
        float2 d[Q], r2, ux2, uy2, uz2;
#pragma unroll
        for (int i = 0; i < Q; ++i) d[i] = half2_bits_to_float2(h[i][p]);
        collide2<true, AVG>(d, scale, inv_scale, L.tau0, L.csmag2, r2, ux2, uy2, uz2);
        R[2 * p] = r2.x; UX[2 * p] = ux2.x; UY[2 * p] = uy2.x; UZ[2 * p] = uz2.x;
        R[2 * p + 1] = r2.y; UX[2 * p + 1] = ux2.y; UY[2 * p + 1] = uy2.y; UZ[2 * p + 1] = uz2.y;
#pragma unroll
        for (int i = 0; i < Q; ++i) h[i][p] = float2_to_half2_bits(d[i].x, d[i].y);
    }
    if (!store) return;
#pragma unroll
    for (int i = 0; i < Q; ++i) HVec<VP>::store(reinterpret_cast<__half*>(fd) + (long long)i * S + own, h[i]);
    if constexpr (OUT) {
        store_fields<VP, AVG>(L, own, R, UX, UY, UZ);
        bool bad = false;
#pragma unroll
        for (int k = 0; k < VP; ++k) bad |= !(R[k] > 0.f && R[k] < 3.4e38f);
        if (bad) atomicOr(L.status, 1);
    }
}

// Plain list over segments of VP*G cells: a warp takes 32/G consecutive list entries per
// pass, G lanes (VP cells each) per segment.  In the last pass, groups past the end of the
// list repeat the pass's first segment and store nothing (every lane still takes part in
// the shuffles).  One pass per warp unless the grid is held down (lbm_tile.ctas_per_sm): CTAs
// that come and go sweep the list in order, 4 % faster than a resident grid striding over it
// (347 against 360 us on the 27.3M plain cells of the 36M-cell reach, 5.98 TB/s of 76 B a cell).
// VP = 4 keeps 20 warps per SM (96 registers), VP = 8 12 (168, 345 us there, but half the warps
// where a case is small).
template <int VP, int G, bool OUT, bool AVG>
__global__ void __launch_bounds__(128, VP == 8 ? 3 : 5) k_rows_h_plain(const lbm_lattice L, const PullOffsets po,
                                                                      const uint32_t* __restrict__ list, int nlist,
                                                                      const __half* __restrict__ fs,
                                                                      __half* __restrict__ fd, float scale)
{
    constexpr int PER_WARP = 32 / G;
    const int lane = threadIdx.x & 31, gl = lane % G, grp = lane / G;
    const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), W = (int)((gridDim.x * blockDim.x) >> 5);
    for (long long b = (long long)gw * PER_WARP; b < nlist; b += (long long)W * PER_WARP) {
        const bool valid = b + grp < nlist;
        const uint32_t id = __ldg(list + (valid ? b + grp : b));
        h_plain_segment<VP, G, OUT, AVG>(L, po, fs, fd, scale, id, gl, valid);
    }
}

// float populations <-> 16-bit storage, n = 19*cells elements (direction i = element / cells).
__global__ void k_pack_populations(const float* __restrict__ f, __half* __restrict__ h, long long cells, float scale)
{
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long long)Q * cells) return;
    const int i = (int)(e / cells);
    const float w = i == 0 ? wgt(0) : (i < 7 ? wgt(1) : wgt(7));
    h[e] = __float2half_rn(__fmul_rn(__fsub_rn(f[e], w), scale));
}
__global__ void k_unpack_populations(const __half* __restrict__ h, float* __restrict__ f, long long cells,
                                     float inv_scale)
{
    const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= (long long)Q * cells) return;
    const int i = (int)(e / cells);
    const float w = i == 0 ? wgt(0) : (i < 7 ? wgt(1) : wgt(7));
    f[e] = __fadd_rn(w, __fmul_rn(__half2float(h[e]), inv_scale));
}
