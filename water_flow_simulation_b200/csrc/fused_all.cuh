// fused_all.cuh -- the three lists of the split pipeline's step in one launch.
// Included inside the anonymous namespace of lbm_kernels.cu, after fused_edge.cuh.
//
// What bounds a step differs by list: instruction issue and latency for the special segments, HBM
// for the plain ones, and on small lattices the launches themselves (about 5 us a kernel, with
// every warp of it resident at once).  In one launch the lists run beside one another and share one
// tail.  Occupancy is that of the 16-bit plain kernel (5 CTAs, 96 registers) or the float32 one (4,
// 128): the edge passes then spill some 170 bytes a thread, which costs less than the CTAs would
// (8M cells in 16-bit storage: 150 us a step at 5 CTAs, 153 at 4, 162 in three launches).
//
//   us a step          three launches   one launch
//   192 x 50 x 12    f32     12.9          9.0
//   333 x 61 x 17    f16     20.9         13.1
//   577 x 203 x 25   f16     77.4         69.4
//   493 x 263 x 41   f16      119          107
//   701 x 305 x 37   f32      229          209
//   1500 x 602 x 40  f32      910          894
//   1500 x 602 x 40  f16      548          547
// (a twentieth of an averaged window of 20 steps, whose output step keeps its launches per list)
#pragma once

// Warp passes of the special list first (the longest chain of dependent loads and arithmetic), then
// the edge list's, then the plain list's; the code of each pass is that of k_cells, k_edge, k_rows
// and k_rows_h_plain, and the lists' passes do not read what another writes.  `nspread` > 0: the
// first nspread CTAs' worth of passes (special and edge) are spread evenly over the grid.
template <int CPL, bool UCOL, bool EARLY, typename T>
__global__ void __launch_bounds__(128, std::is_same<T, float>::value ? 4 : 5)
    k_all_lists(const lbm_lattice L, const PullOffsets po, const T* __restrict__ fs, T* __restrict__ fd, float scale,
                int nspread)
{
    constexpr int SEG = 32 * CPL, G = SEG / 4 < 32 ? SEG / 4 : 32;
    constexpr bool F32 = std::is_same<T, float>::value;
    // steps launched early are those of small lattices (kEarlyLaunchCells): 32-bit indexes (pull_element)
    using Int = std::conditional_t<EARLY, int, long long>;
    const int lane = threadIdx.x & 31, nseg = (L.pitch + SEG - 1) / SEG;
    const float inv_scale = 1.0f / scale;
    if constexpr (EARLY) {
        // launched while the step before is in its last wave (launch_all_lists): nothing is read or written
        // until that step has ended, and the next one may start once every CTA of this one has
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    }
    int cta = (int)blockIdx.x;
    if (nspread > 0) {
        const int before = (int)((long long)cta * nspread / gridDim.x);
        cta = (int)((long long)(cta + 1) * nspread / gridDim.x) > before ? before : nspread + cta - before;
    }
    int t = cta * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5);
    const int ncells = L.n_special * CPL;
    if (t < ncells) {
        int seg, y, z;
        decode_row(__ldg(L.rows_special + t / CPL), nseg, L.ny, seg, y, z);
        const int xa = seg * SEG + t % CPL * 32;
        if (xa < L.pitch)
            cell_pass<SEG < 128 ? SEG : 128, false, UCOL, false, T, Int>(L, fs, fd, scale, inv_scale, xa, y, z, lane,
                                                                         pass_flags(L, xa + lane, y, z));
        return;
    }
    t -= ncells;
    const int nedge = edge_passes(CPL, L.n_edge);
    if (t < nedge) {
        edge_pass<CPL, false, false, T>(L, po, L.rows_edge, L.n_edge, fs, fd, scale, t, lane);
        return;
    }
    t -= nedge;
    if constexpr (F32) {
        if (t < L.n_plain) plain_segment<CPL, false, false>(L, po, fs, fd, __ldg(L.rows_plain + t), lane);
    } else {
        const int b = t * (32 / G), grp = lane / G;
        if (b < L.n_plain) {
            const bool valid = b + grp < L.n_plain;
            h_plain_segment<4, G, false, false>(L, po, fs, fd, scale, __ldg(L.rows_plain + (valid ? b + grp : b)),
                                                lane % G, valid);
        }
    }
}
