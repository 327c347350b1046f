// fused_cells.cuh -- special segments of the split pipeline, one cell per lane.
// Included inside the anonymous namespace of lbm_kernels.cu, after fused_half.cuh.
//
// A warp pass covers 32 consecutive cells of one row; a lane owns one cell and pulls its 19
// populations with one scalar load each.  What bounds these segments is instruction issue and
// latency, not bytes: per cell a flag word, then 19 populations and (under the wall function) six
// more values, and about 1000 instructions, a third of them the float64 wall function's.  So the
// pull is branch-free -- the address of every direction is selected first (the own cell's
// opposite population at a wall, the own population at an x edge, the mirrored one under the
// lid, else the neighbour's) -- and all 19 loads, and the wall function's, are in flight together
// after the one flag word.  One cell per lane fits 96 registers, 20 warps per SM; the scalar
// accesses of a warp still fall into whole 32-byte sectors.  On the special segments of the
// 36M-cell reach 92 us with 16-bit storage and 114 with float32, against 136 and 262 for two and
// four cells per lane with a branch, and a dependent load, per bounced direction.
#pragma once

// One stored population as it lies in memory, and its value as float.
template <typename T> struct Stored {
    using type = uint16_t;
    static __device__ __forceinline__ float value(uint16_t v) { return __half2float(__ushort_as_half(v)); }
};
template <> struct Stored<float> {
    using type = float;
    static __device__ __forceinline__ float value(float v) { return v; }
};
template <typename T>
__device__ __forceinline__ void load_cell(typename Stored<T>::type& v, const T* p) { ld_ordered(v, p); }
__device__ __forceinline__ void load_cell(uint16_t& v, const hcoh* p)
{
    v = __half_as_ushort(__ldcg(reinterpret_cast<const __half*>(p)));
}

template <typename T, typename Int, int... Is>
__device__ __forceinline__ void pull_cell_all(std::integer_sequence<int, Is...>, float (&f)[Q],
                                              const T* __restrict__ fs, Int own, Int plane, int pitch,
                                              long long S, uint32_t fk, bool lid, bool x_first, bool x_last)
{
    typename Stored<T>::type v[Q];
    (load_cell(v[Is], fs + pull_element<Is, Int>(own, plane, pitch, S, fk, lid, x_first, x_last)), ...);
    ((f[Is] = Stored<T>::value(v[Is])), ...);
}

// Streaming store of one cell's population of direction I.
template <int I>
__device__ __forceinline__ void store_cell(float* p, float v, float) { __stcs(p, v); }
template <int I>
__device__ __forceinline__ void store_cell(__half* p, float v, float scale)
{
    *p = __float2half_rn(fma_rn(v, scale, -wgt(I) * scale));   // (v - w) scale: the scale is a power of two
}
template <int I>
__device__ __forceinline__ void store_cell(hcoh* p, float v, float scale)
{
    store_cell<I>(reinterpret_cast<__half*>(p), v, scale);
}
template <typename T, int... Is>
__device__ __forceinline__ void store_cell_all(std::integer_sequence<int, Is...>, T* fd, long long own, long long S,
                                               const float (&f)[Q], float scale)
{
    (store_cell<Is>(fd + Is * S + own, f[Is], scale), ...);
}

// Outlet cells at the start of a pass: when x = nx-1 is a multiple of 32 but not of `join` cells
// (the list's segment length, at most 128), the lane that holds x = nx-2 (lane 31 of the pass
// before, same segment, so the same arithmetic) also writes the outlet cell, from the unrounded
// populations it holds, and the outlet cell's own lane keeps its populations.  At a multiple of
// `join` a separate pass (bc_row) writes the outlet from the stored populations.
__device__ __forceinline__ bool outlet_across_passes(const lbm_lattice& L, int join)
{
    return (L.nx - 1) % 32 == 0 && (L.nx - 1) % join != 0;
}

// One warp pass over the cells x = xa + lane of row (y, z) of a special segment
// (floodsim/lbm3d.py:42-138): `fk` is the lane's flag word (FLAG_SOLID past the pitch), JOIN as in
// outlet_across_passes, Int as in pull_element.  Called by all lanes of the warp.
template <int JOIN, bool OUT, bool UCOL, bool AVG, typename T, typename Int = long long>
__device__ __forceinline__ void cell_pass(const lbm_lattice& L, const T* __restrict__ fs, T* __restrict__ fd,
                                          float scale, float inv_scale, int xa, int y, int z, int lane, uint32_t fk)
{
    constexpr auto QS = std::make_integer_sequence<int, Q>{};
    const long long S = L.cells;
    const int x = xa + lane;
    const bool active = x < L.pitch, solid = (fk & FLAG_SOLID) != 0;
    const Int plane = (Int)L.ny * L.pitch, own = z * plane + (Int)y * L.pitch + x;
    float f[Q];
    float r = 1.f, ux = 0.f, uy = 0.f, uz = 0.f;
    if (!solid) {
        pull_cell_all<T, Int>(QS, f, fs, own, plane, L.pitch, S, fk, z == L.nz - 1, x == 0, x == L.nx - 1);
        float U = 0.f, cf = 0.f;
        if (fk & FLAG_WALLFN) {
            if constexpr (UCOL) U = (fk & FLAG_BEDWALL) ? L.colU[(long long)y * L.pitch + x] : 0.f;
            else U = L.uref[own];
            cf = L.cfw[own];
            ux = L.ux[own]; uy = L.uy[own]; uz = L.uz[own]; r = L.rho[own];
        }
        raw_to_pop<T>(f, inv_scale);
        if (fk & FLAG_WALLFN) wall_function(f, fk & FLAG_WALLS, cf, ux, uy, uz, r, U);
        const float tau0 = sponge_tau0(L, x);
        if (fk & FLAG_FORCE)
            collide<true>(f, L.Fx[own] * L.force_scale, L.Fy[own] * L.force_scale, L.Fz[own] * L.force_scale, tau0,
                          L.csmag2, r, ux, uy, uz);
        else
            collide<false>(f, 0.f, 0.f, 0.f, tau0, L.csmag2, r, ux, uy, uz);
    } else {
#pragma unroll
        for (int i = 0; i < Q; ++i) f[i] = wgt(i);
    }
    bool keep = !active;                                   // lanes that store no populations
    const int out_lane = L.nx - 1 - xa;                    // the outlet cell's lane
    if (xa == 0 || (out_lane >= 0 && out_lane <= 32)) {    // warp-uniform
        const bool across = out_lane == 32 && outlet_across_passes(L, JOIN);
        if (out_lane == 0 && outlet_across_passes(L, JOIN))
            keep |= lane == 0 && !solid && !(L.flags[own - 1] & FLAG_SOLID);
#pragma unroll 1
        for (int end = 0; end < 2; ++end) {                // inlet x = 0 from 1, outlet x = nx-1 from nx-2
            const int b = end == 0 ? (xa == 0 ? 0 : -1) : across ? 31 : out_lane > 0 && out_lane < 32 ? out_lane : -1;
            if (b < 0) continue;
            const int from = end == 0 ? lane + 1 : across ? lane : lane - 1;
            float g[Q];
#pragma unroll
            for (int i = 0; i < Q; ++i) g[i] = __shfl_sync(0xffffffffu, f[i], from);
            const bool from_solid = __shfl_sync(0xffffffffu, solid, from);
            if (lane == b && !solid && !from_solid && !(end && across && (L.flags[own + 1] & FLAG_SOLID))) {
                float o[Q];
                nebb(end == 0, g, o, end == 0 ? L.uin[y + (long long)L.ny * z] : 0.f, L.rho_out);
                if (end && across) {
                    store_cell_all<T>(QS, fd, own + 1, S, o, scale);
                } else {
#pragma unroll
                    for (int i = 0; i < Q; ++i) f[i] = o[i];
                }
            }
        }
    }
    if (!keep) store_cell_all<T>(QS, fd, own, S, f, scale);
    if (!active) return;
    if constexpr (OUT) {
        if (!solid && !(r > 0.f && r < 3.4e38f)) atomicOr(L.status, 1);
        const float R[1] = {r}, UX[1] = {ux}, UY[1] = {uy}, UZ[1] = {uz};
        store_fields<1, AVG>(L, own, R, UX, UY, UZ);
    } else if (fk & FLAG_WALLFN) {                         // the wall function reads these next step
        L.rho[own] = r; L.ux[own] = ux; L.uy[own] = uy; L.uz[own] = uz;
    }
}

// Flag word of the cell x of a row for cell_pass (FLAG_SOLID past the pitch).
__device__ __forceinline__ uint32_t pass_flags(const lbm_lattice& L, int x, int y, int z)
{
    return x < L.pitch ? __ldg(L.flags + ((long long)z * L.ny + y) * L.pitch + x) : FLAG_GHOST | FLAG_SOLID;
}

// Special list: pass t of the launch is 32-cell part t % CPL of entry t / CPL (segments of 32*CPL cells).
template <int CPL, bool OUT, bool UCOL, bool AVG, typename T>
__global__ void __launch_bounds__(128, 5) k_cells(const lbm_lattice L, const uint32_t* __restrict__ special,
                                                           int n_special, const T* __restrict__ fs, T* __restrict__ fd,
                                                           float scale)
{
    constexpr int SEG = 32 * CPL, JOIN = SEG < 128 ? SEG : 128;
    const int lane = threadIdx.x & 31;
    const long long W = ((long long)gridDim.x * blockDim.x) >> 5, total = (long long)n_special * CPL;
    const int nseg = (L.pitch + SEG - 1) / SEG;
    const float inv_scale = 1.0f / scale;
    for (long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < total; t += W) {
        int seg, y, z;
        decode_row(__ldg(special + t / CPL), nseg, L.ny, seg, y, z);
        const int xa = seg * SEG + (int)(t % CPL) * 32;
        if (xa >= L.pitch) continue;                       // warp-uniform
        cell_pass<JOIN, OUT, UCOL, AVG, T>(L, fs, fd, scale, inv_scale, xa, y, z, lane, pass_flags(L, xa + lane, y, z));
    }
}
