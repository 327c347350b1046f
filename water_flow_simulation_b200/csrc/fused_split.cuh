// fused_split.cuh -- work-list pipeline of the fused step (lbm_tile.pipeline = 3).
// Included inside the anonymous namespace of lbm_kernels.cu, after fused_reg.cuh.
//
// The lattice is cut into row segments of 32*V cells (V = 4: 128 cells).  Once per
// geometry (lbm_build_worklists) every segment is classified and compacted, in order,
// into one of four lists:
//   plain   -- open row (1 <= y <= ny-2, 1 <= z <= nz-1: the row under the lid included),
//              clear of the x edges and of padding, no cell solid, walled, forced or under
//              the wall function;
//   edge    -- the same, except that the segment holds x = 0 (inlet) or x = nx-1 (outlet)
//              and possibly padding: the first and last segment of an open row;
//   solid   -- every cell solid (or padding);
//   special -- everything else (walls, bed, lid, banks, hulls, forcing).
// A step then runs k_all_lists (fused_all.cuh), the passes of the three moving lists in one launch;
// an output step, an overlapped one or one with its grid held down runs a kernel per list:
//   k_rows          over the plain list: 19 V-wide pulls at constant offsets (the +-1 x
//                   neighbours by warp shuffle), collision with no force, 19 V-wide
//                   streaming stores -- no flag word is read; this is where the cells are;
//   k_cells         (fused_cells.cuh) over the special list: flag words, y walls, bed, lid,
//                   bounce-back, x edges, wall function, forcing, inlet/outlet, one cell per lane;
//   k_edge          (fused_edge.cuh) over the edge list: the plain pull, the x-edge copies, the
//                   inlet and outlet extrapolation and rest-state padding, without flag words;
//   k_solid_out     on output steps only: the fields of solid segments;
//   k_column_mean   on output steps with the column-mean wall model: the depth-mean speed
//                   of every (y, x) column, summed over z in order.
// Solid segments move no populations: solid cells are never read and both population
// buffers hold their rest state from the start.
#pragma once

// Row-segment id: (z * ny + y) * nseg + seg.
__device__ __forceinline__ void decode_row(uint32_t id, int nseg, int ny, int& seg, int& y, int& z)
{
    seg = (int)(id % (uint32_t)nseg);
    const uint32_t yz = id / (uint32_t)nseg;
    y = (int)(yz % (uint32_t)ny);
    z = (int)(yz / (uint32_t)ny);
}

// Streaming stores of the V cells' 19 populations.
template <int I, int V>
__device__ __forceinline__ void store_pop(float* p, const float (&f)[V][Q])
{
    float v[V];
#pragma unroll
    for (int k = 0; k < V; ++k) v[k] = f[k][I];
    vstore<V>(p, v);
}
template <int V, int... Is>
__device__ __forceinline__ void store_pops(std::integer_sequence<int, Is...>, float* fd, long long S, long long own,
                                           const float (&f)[V][Q])
{
    (store_pop<Is, V>(fd + (long long)Is * S + own, f), ...);
}

// Output-step fields of V cells and, with AVG, their time-average sums
// (floodsim/reach3d.py:443-451: ux, uy, uz, rho, speed, ux^2).  UX2: as in collide().
template <int V, bool AVG, bool UX2 = (V > 1)>
__device__ __forceinline__ void store_fields(const lbm_lattice& L, long long own, const float (&R)[V],
                                             const float (&UX)[V], const float (&UY)[V], const float (&UZ)[V])
{
    const long long S = L.cells;
    vstore_plain<V>(L.rho + own, R);
    vstore_plain<V>(L.ux + own, UX);
    vstore_plain<V>(L.uy + own, UY);
    vstore_plain<V>(L.uz + own, UZ);
    if constexpr (AVG) {
        if (!L.avg) return;                // a batched lattice outside its averaging window
        float a[V], s[V];
#define WFS_ACC(M, EXPR)                                                   \
        vload_plain<V>(a, L.avg + (long long)(M) * S + own);               \
        _Pragma("unroll") for (int k = 0; k < V; ++k) {                   \
            s[k] = a[k] + (EXPR);                                         \
        }                                                                 \
        vstore_plain<V>(L.avg + (long long)(M) * S + own, s);
        WFS_ACC(0, UX[k])
        WFS_ACC(1, UY[k])
        WFS_ACC(2, UZ[k])
        WFS_ACC(3, R[k])
        WFS_ACC(4, sqrtf(fma_rn(UZ[k], UZ[k], UX2 ? fma_rn(UY[k], UY[k], mul_rn(UX[k], UX[k]))
                                              : fma_rn(UX[k], UX[k], mul_rn(UY[k], UY[k])))))
        WFS_ACC(5, UX[k] * UX[k])
#undef WFS_ACC
    }
}

// Relaxation time at zero strain of column x: tau0, or inside the optional outlet sponge
// tau0 + (sponge_tau - tau0) s^2 (explicitly rounded, so every kernel computes the same value).
__device__ __forceinline__ float sponge_tau0(const lbm_lattice& L, int x)
{
    const int x0 = L.nx - L.sponge_cols;
    if (L.sponge_cols <= 0 || x < x0) return L.tau0;
    const float s = __fdiv_rn((float)(x - x0 + 1), (float)L.sponge_cols);
    return __fadd_rn(L.tau0, __fmul_rn(__fsub_rn(L.sponge_tau, L.tau0), __fmul_rn(s, s)));
}

// One plain segment of 32*V cells (row-segment id `id`), V cells per lane.
template <int V, bool OUT, bool AVG>
__device__ __forceinline__ void plain_segment(const lbm_lattice& L, const PullOffsets& po, const float* __restrict__ fs,
                                              float* __restrict__ fd, uint32_t id, int lane)
{
    constexpr int SEG = 32 * V;
    int seg, y, z;
    decode_row(id, (L.pitch + SEG - 1) / SEG, L.ny, seg, y, z);
    const long long own = ((long long)z * L.ny + y) * L.pitch + seg * SEG + lane * V;
    float f[V][Q];
    float R[V], UX[V], UY[V], UZ[V];
    pull_fast_all<V>(std::make_integer_sequence<int, Q>{}, f, fs + own, po, lane, z == L.nz - 1);
#pragma unroll
    for (int k = 0; k < V; k += 2) {
        float2 d[Q], r2, ux2, uy2, uz2;
#pragma unroll
        for (int i = 0; i < Q; ++i) d[i] = make_float2(f[k][i], f[k + 1][i]);
        collide2<false, AVG>(d, 1.f, 1.f, L.tau0, L.csmag2, r2, ux2, uy2, uz2);
#pragma unroll
        for (int i = 0; i < Q; ++i) { f[k][i] = d[i].x; f[k + 1][i] = d[i].y; }
        R[k] = r2.x; UX[k] = ux2.x; UY[k] = uy2.x; UZ[k] = uz2.x;
        R[k + 1] = r2.y; UX[k + 1] = ux2.y; UY[k + 1] = uy2.y; UZ[k + 1] = uz2.y;
    }
    store_pops<V>(std::make_integer_sequence<int, Q>{}, fd, L.cells, own, f);
    if constexpr (OUT) {
        store_fields<V, AVG>(L, own, R, UX, UY, UZ);
        bool bad = false;
#pragma unroll
        for (int k = 0; k < V; ++k) bad |= !(R[k] > 0.f && R[k] < 3.4e38f);
        if (bad) atomicOr(L.status, 1);
    }
}

// Plain list: a warp pass per segment of 32*V cells, one pass per warp unless the grid is held
// down (lbm_tile.ctas_per_sm).  Bound by HBM: with V = 4, 16 warps per SM (118 registers) and all
// of a pass's 19 16-byte loads issued before anything waits, 155 KB are in flight per SM, and CTAs
// that come and go sweep the list in order; 605 us on the 36M-cell reach, against 734 for a
// resident grid of 12 warps per SM and the scalar collision.
template <int V, bool OUT, bool AVG>
__global__ void __launch_bounds__(128, V == 4 ? 4 : 6) k_rows(const lbm_lattice L, const PullOffsets po,
                                                              const uint32_t* __restrict__ list, int nlist,
                                                              const float* __restrict__ fs, float* __restrict__ fd)
{
    const int lane = threadIdx.x & 31;
    const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), W = (int)((gridDim.x * blockDim.x) >> 5);
    for (int w = gw; w < nlist; w += W) plain_segment<V, OUT, AVG>(L, po, fs, fd, __ldg(list + w), lane);
}

// Output step: fields of one solid segment's V cells per lane (rho = 1, u = 0) and their
// time-average sums.
template <int V, bool AVG>
__device__ __forceinline__ void solid_segment(const lbm_lattice& L, uint32_t id, int lane)
{
    constexpr int SEG = 32 * V;
    const int nseg = (L.pitch + SEG - 1) / SEG;
    const long long S = L.cells;
    int seg, y, z;
    decode_row(id, nseg, L.ny, seg, y, z);
    const int x0 = seg * SEG + lane * V;
    if (x0 >= L.pitch) return;
    const long long own = ((long long)z * L.ny + y) * L.pitch + x0;
    float one[V], zero[V];
#pragma unroll
    for (int k = 0; k < V; ++k) { one[k] = 1.f; zero[k] = 0.f; }
    vstore_plain<V>(L.rho + own, one);
    vstore_plain<V>(L.ux + own, zero);
    vstore_plain<V>(L.uy + own, zero);
    vstore_plain<V>(L.uz + own, zero);
    if constexpr (AVG) {
        if (!L.avg) return;
        float a[V];
        vload_plain<V>(a, L.avg + 3 * S + own);
#pragma unroll
        for (int k = 0; k < V; ++k) a[k] += 1.f;
        vstore_plain<V>(L.avg + 3 * S + own, a);
    }
}

template <int V, bool AVG>
__global__ void k_solid_out(const lbm_lattice L, const uint32_t* __restrict__ list, int nlist)
{
    const int lane = threadIdx.x & 31;
    const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), W = (int)((gridDim.x * blockDim.x) >> 5);
    for (int w = gw; w < nlist; w += W) solid_segment<V, AVG>(L, __ldg(list + w), lane);
}

// Depth-mean speed of column q = x + pitch*y (floodsim/reach3d.py:412-417): the sums of ux
// and uy over the column's fluid cells, taken in z order, then sqrt(sx^2 + sy^2) / n.
// COH: read the velocities through coherent loads (the persistent batch chunk, where other
// CTAs wrote them earlier in the same launch).
template <bool COH = false>
__device__ __forceinline__ void column_mean_at(const lbm_lattice& L, long long q)
{
    if (q >= (long long)L.ny * L.pitch) return;
    const int x = (int)(q % L.pitch);
    if (x >= L.nx) return;
    const long long plane = (long long)L.ny * L.pitch;
    float sx = 0.f, sy = 0.f, n = 0.f;
    for (int z = 0; z < L.nz; ++z) {
        const long long c = q + plane * z;
        if (!(L.flags[c] & FLAG_SOLID)) {
            sx += COH ? __ldcg(L.ux + c) : L.ux[c];
            sy += COH ? __ldcg(L.uy + c) : L.uy[c];
            n += 1.f;
        }
    }
    L.colU[q] = sqrtf(sx * sx + sy * sy) / fmaxf(n, 1.f);
}

__global__ void k_column_mean(const lbm_lattice L)
{
    column_mean_at(L, (long long)blockIdx.x * blockDim.x + threadIdx.x);
}
