// fused_edge.cuh -- edge segments of the split pipeline, four cells per lane.
// Included inside the anonymous namespace of lbm_kernels.cu, after fused_half.cuh.
//
// An edge segment is the first or last of an open row: plain cells but for x = 0, x = nx-1 and
// padding.  It takes the plain kernels' pull (one 16- or 8-byte load per direction, x neighbours
// by shuffle) and the packed collision on populations; the two end cells then cost a few
// predicated loads and one lane's inlet/outlet extrapolation per segment.  51 us on the edge
// segments of the 36M-cell reach with 16-bit storage (71 for two cells per lane and 4-byte
// loads), 149 with float32, whose segments are twice as long; those segments lie 3 or 6 KB apart.
#pragma once

// Two cells' stored populations of one direction: float2, or two 16-bit values in a word.
template <typename T> struct PairOf { using type = uint32_t; };
template <> struct PairOf<float> { using type = float2; };

// Direction I of the four cells of lane gl of a group of G lanes (a row segment of 4*G cells).
template <int I, int G>
__device__ __forceinline__ void edge_pull(float (&t)[Q][4], float (&e)[Q], const float* __restrict__ own_ptr,
                                          const PullOffsets& po, int gl, bool lid)
{
    const float* src = own_ptr + pull_offset<I>(po, lid);
    e[I] = 0.f;
    ld_ordered(t[I], src);
    if constexpr (cx(I) == 1) ld_ordered_if(gl == 0, e[I], src - 1);
    if constexpr (cx(I) == -1) ld_ordered_if(gl == G - 1, e[I], src + 4);
}
template <int I, int G>
__device__ __forceinline__ void edge_shift(float2 (&h)[Q][2], const float (&t)[Q][4], const float (&e)[Q], int gl)
{
    if constexpr (cx(I) == 0) {
        h[I][0] = make_float2(t[I][0], t[I][1]);
        h[I][1] = make_float2(t[I][2], t[I][3]);
    } else if constexpr (cx(I) == 1) {
        const float p = __shfl_up_sync(0xffffffffu, t[I][3], 1, G);
        h[I][0] = make_float2(gl == 0 ? e[I] : p, t[I][0]);
        h[I][1] = make_float2(t[I][1], t[I][2]);
    } else {
        const float n = __shfl_down_sync(0xffffffffu, t[I][0], 1, G);
        h[I][0] = make_float2(t[I][1], t[I][2]);
        h[I][1] = make_float2(t[I][3], gl == G - 1 ? e[I] : n);
    }
}
template <int G, int... Is>
__device__ __forceinline__ void edge_pull_all(std::integer_sequence<int, Is...>, float2 (&h)[Q][2],
                                              const float* __restrict__ p, const PullOffsets& po, int gl, bool lid)
{
    float t[Q][4], e[Q];
    (edge_pull<Is, G>(t, e, p, po, gl, lid), ...);
    (edge_shift<Is, G>(h, t, e, gl), ...);
}
template <int G, typename T, int... Is>
__device__ __forceinline__ void edge_pull_all(std::integer_sequence<int, Is...> s, uint32_t (&h)[Q][2],
                                              const T* __restrict__ p, const PullOffsets& po, int gl, bool lid)
{
    hpull_all<4, G, T>(s, h, p, po, gl, lid);
}

// Populations of a stored pair and back; one element of a pair replaced by a population.
__device__ __forceinline__ float2 pair_pop(float2 h, int, float) { return h; }
__device__ __forceinline__ float2 pair_pop(uint32_t h, int i, float inv_scale)
{
    return fma2(half2_bits_to_float2(h), both(inv_scale), both(wgt(i)));
}
__device__ __forceinline__ void pair_set(float2& h, float2 v, int, float) { h = v; }
__device__ __forceinline__ void pair_set(uint32_t& h, float2 v, int i, float scale)
{
    const float2 s = fma2(v, both(scale), both(-wgt(i) * scale));
    h = float2_to_half2_bits(s.x, s.y);
}
__device__ __forceinline__ void pair_set_x(float2& h, float v, int, float) { h.x = v; }
__device__ __forceinline__ void pair_set_x(uint32_t& h, float v, int i, float scale)
{
    h = __byte_perm(float2_to_half2_bits(fma_rn(v, scale, -wgt(i) * scale), 0.f), h, 0x7610);
}

template <int... Is>
__device__ __forceinline__ void edge_store_all(std::integer_sequence<int, Is...>, float* p, long long S,
                                               const float2 (&h)[Q][2])
{
    (Vec<4>::store(p + Is * S, h[Is][0].x, h[Is][0].y, h[Is][1].x, h[Is][1].y), ...);
}
template <typename T, int... Is>
__device__ __forceinline__ void edge_store_all(std::integer_sequence<int, Is...>, T* p, long long S,
                                               const uint32_t (&h)[Q][2])
{
    (HVec<4>::store(reinterpret_cast<__half*>(p + Is * S), h[Is]), ...);
}

// The cells x0 .. x0+3 (x0 a multiple of 4) of lane gl of a G-lane group in an open row.  `store`
// false: the group repeats another group's segment and writes nothing.  Loads stay inside the
// population array: an open row has rows on both sides.  When x = nx-1 is a multiple of 4*G its
// neighbour is in another segment, and a separate pass (bc_row) writes the outlet.
template <int G, bool OUT, bool AVG, typename T>
__device__ __forceinline__ void edge_lane(const lbm_lattice& L, const PullOffsets& po, const T* __restrict__ fs,
                                          T* __restrict__ fd, float scale, float inv_scale, int x0, int y, int z,
                                          int gl, bool store)
{
    constexpr auto QS = std::make_integer_sequence<int, Q>{};
    const long long S = L.cells, rowc = ((long long)z * L.ny + y) * L.pitch;
    const bool active = x0 < L.pitch;
    const long long own = rowc + (active ? x0 : L.pitch - 4);
    typename PairOf<T>::type h[Q][2];
    edge_pull_all<G>(QS, h, fs + own, po, gl, z == L.nz - 1);
    // a direction whose source lies outside [0, nx) keeps the cell's own population
    // (floodsim/lbm3d.py:48-49): cx = +1 at x = 0, cx = -1 at x = nx-1
    const bool first = x0 == 0, last = x0 <= L.nx - 1 && L.nx - 1 < x0 + 4;
    const int kl = (L.nx - 1) & 3;                         // the outlet cell's place in its lane
    float in_own[Q], out_own[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        if (cx(i) == 1) in_own[i] = first ? ld1(fs + i * S + rowc) : 0.f;
        if (cx(i) == -1) out_own[i] = last ? ld1(fs + i * S + rowc + L.nx - 1) : 0.f;
    }
    float R[4], UX[4], UY[4], UZ[4], g1[Q];
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        float2 d[Q], r, ux, uy, uz;
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            d[i] = pair_pop(h[i][p], i, inv_scale);
            const float w = std::is_same<T, float>::value ? 0.f : wgt(i);
            const float is = std::is_same<T, float>::value ? 1.f : inv_scale;
            if (cx(i) == 1 && p == 0) d[i].x = first ? fma_rn(in_own[i], is, w) : d[i].x;
            if (cx(i) == -1) {
                d[i].x = last && kl == 2 * p ? fma_rn(out_own[i], is, w) : d[i].x;
                d[i].y = last && kl == 2 * p + 1 ? fma_rn(out_own[i], is, w) : d[i].y;
            }
        }
        collide2<false, false>(d, 1.f, 1.f, L.tau0, L.csmag2, r, ux, uy, uz);
        const bool padx = x0 + 2 * p >= L.nx, pady = x0 + 2 * p + 1 >= L.nx;     // padding: at rest
#pragma unroll
        for (int i = 0; i < Q; ++i) d[i] = make_float2(padx ? wgt(i) : d[i].x, pady ? wgt(i) : d[i].y);
        R[2 * p] = padx ? 1.f : r.x;
        R[2 * p + 1] = pady ? 1.f : r.y;
        UX[2 * p] = padx ? 0.f : ux.x; UX[2 * p + 1] = pady ? 0.f : ux.y;
        UY[2 * p] = padx ? 0.f : uy.x; UY[2 * p + 1] = pady ? 0.f : uy.y;
        UZ[2 * p] = padx ? 0.f : uz.x; UZ[2 * p + 1] = pady ? 0.f : uz.y;
        if (p == 0) {
            // inlet x = 0 from x = 1; outlet at place 1 from place 0
            const bool o1 = last && kl == 1;
            if (first || o1) {
                float g[Q], o[Q];
#pragma unroll
                for (int i = 0; i < Q; ++i) g[i] = first ? d[i].y : d[i].x;
                nebb(first, g, o, first ? L.uin[y + (long long)L.ny * z] : 0.f, L.rho_out);
#pragma unroll
                for (int i = 0; i < Q; ++i) {
                    if (first) d[i].x = o[i];
                    else d[i].y = o[i];
                }
            }
#pragma unroll
            for (int i = 0; i < Q; ++i) g1[i] = d[i].y;
        } else {
            // outlet at place 3 from 2, at 2 from 1, at 0 from the left lane's 3
            float g[Q], o[Q];
            if (__any_sync(0xffffffffu, last && kl == 0)) {
#pragma unroll
                for (int i = 0; i < Q; ++i) {
                    const float left = __shfl_up_sync(0xffffffffu, d[i].y, 1, G);
                    g1[i] = kl == 0 ? left : g1[i];
                }
            }
            if (last && kl != 1 && (kl != 0 || gl > 0)) {
#pragma unroll
                for (int i = 0; i < Q; ++i) g[i] = kl == 3 ? d[i].x : g1[i];
                nebb(false, g, o, 0.f, L.rho_out);
#pragma unroll
                for (int i = 0; i < Q; ++i) {
                    if (kl == 3) d[i].y = o[i];
                    else if (kl == 2) d[i].x = o[i];
                    else pair_set_x(h[i][0], o[i], i, scale);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < Q; ++i) pair_set(h[i][p], d[i], i, scale);
    }
    if (!active || !store) return;
    edge_store_all(QS, fd + own, S, h);
    if constexpr (OUT) {
        store_fields<4, AVG, false>(L, own, R, UX, UY, UZ);
        bool bad = false;
#pragma unroll
        for (int k = 0; k < 4; ++k) bad |= !(R[k] > 0.f && R[k] < 3.4e38f);
        if (bad) atomicOr(L.status, 1);
    }
}

// Edge list: entries are segments of 32*CPL cells; a warp pass takes two entries of 64 cells
// each, one of 128, or half of one of 256.
__host__ __device__ constexpr int edge_passes(int cpl, int nlist) { return cpl == 2 ? (nlist + 1) / 2 : nlist * (cpl / 4); }

template <int CPL, bool OUT, bool AVG, typename T>
__device__ __forceinline__ void edge_pass(const lbm_lattice& L, const PullOffsets& po, const uint32_t* __restrict__ list,
                                          int nlist, const T* __restrict__ fs, T* __restrict__ fd, float scale, int t,
                                          int lane)
{
    constexpr int G = CPL == 2 ? 16 : 32, PER_WARP = 32 / G, SEG = 32 * CPL, PASSES = SEG / (4 * G);
    const int gl = lane % G, grp = lane / G, b = t / PASSES * PER_WARP;
    const bool valid = b + grp < nlist;
    int seg, y, z;
    decode_row(__ldg(list + (valid ? b + grp : b)), (L.pitch + SEG - 1) / SEG, L.ny, seg, y, z);
    const int x0 = seg * SEG + t % PASSES * 4 * G + gl * 4;
    edge_lane<G, OUT, AVG, T>(L, po, fs, fd, scale, 1.0f / scale, x0, y, z, gl, valid);
}

template <int CPL, bool OUT, bool AVG, typename T>
__global__ void __launch_bounds__(128, std::is_same<T, float>::value ? 3 : 4)
    k_edge(const lbm_lattice L, const PullOffsets po, const uint32_t* __restrict__ list, int nlist,
           const T* __restrict__ fs, T* __restrict__ fd, float scale)
{
    const int lane = threadIdx.x & 31, W = (int)((gridDim.x * blockDim.x) >> 5), total = edge_passes(CPL, nlist);
    for (int t = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5); t < total; t += W)
        edge_pass<CPL, OUT, AVG, T>(L, po, list, nlist, fs, fd, scale, t, lane);
}
