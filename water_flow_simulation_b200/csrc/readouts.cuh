// readouts.cuh -- FP64 device reductions of the along-stream profiles (floodsim/reach3d.py:545-568).
// Included inside the anonymous namespace of lbm_kernels.cu.
//
// Per x station, over the fluid cells of the cross-section (y, z), in float64:
//   PROF_Q        sum ux                      (discharge / (dx^2 * velocity scale))
//   PROF_UXX      sum ux^2                    (momentum flux)
//   PROF_DRHO     sum (rho - 1)               (pressure part of the momentum balance)
//   PROF_MASS     sum rho
//   PROF_NFLUID   fluid cells
//   PROF_TOP_N    fluid cells of the top layer (z = nz-1, under the rigid lid)
//   PROF_TOP_DRHO sum (rho - 1) over the top layer   (lid water level)
//   PROF_TOP_UX   sum ux over the top layer          (surface speed)
//   PROF_UMAX     max |u|
// and per (y, x) column the largest |u|^2 of a fluid cell whose lower neighbour is solid
// or the bed (the bed-shear cell of floodsim/reach3d.py:562-566).  The fields are either
// the time-average sums (avg, scaled by inv_navg: ux, uy, uz, rho, |u|, ux^2 at m*cells)
// or, without avg, the instantaneous rho/ux/uy/uz.  The sums are deterministic: pass 1
// writes per-chunk partials, pass 2 adds the chunks in a fixed order.
#pragma once

enum ProfField {
    PROF_Q = 0, PROF_UXX, PROF_DRHO, PROF_MASS, PROF_NFLUID, PROF_TOP_N, PROF_TOP_DRHO, PROF_TOP_UX, PROF_UMAX,
    PROF_NF
};

struct CellFields {
    double rho, ux, sp, uxx;
};

// v: the time-average sums of ux, rho, |u| and ux^2 (AVG), or ux, rho, uy and uz.
template <bool AVG>
__device__ __forceinline__ CellFields cell_fields(const float (&v)[4], double inv_navg)
{
    CellFields r;
    if constexpr (AVG) {
        r.ux = (double)v[0] * inv_navg;
        r.rho = (double)v[1] * inv_navg;
        r.sp = (double)v[2] * inv_navg;
        r.uxx = (double)v[3] * inv_navg;
    } else {
        const double u = v[0], w1 = v[2], w2 = v[3];
        r.ux = u;
        r.rho = v[1];
        r.sp = sqrt(u * u + w1 * w1 + w2 * w2);
        r.uxx = u * u;
    }
    return r;
}

// Pass 1: thread = x station, blockIdx.y = chunk of `per_chunk` columns y, each summed over z, so that
// one pass over the flags and fields makes the partials and the bed speeds.  Bound by the bytes (a
// flag and four fields a cell): kProfAhead layers' flags and fields are requested together, not a
// field after its flag; a warp holds 20 loads in flight and there is a warp per 32 columns.  7.9M cells:
// 41 us, 3.9 TB/s, with the bed speeds, which took a second pass over the flags.  Profiles and force
// sums of that case together, with their copies to the host: 590 us before, 400 now.
constexpr int kProfAhead = 4;

template <bool AVG>
__global__ void __launch_bounds__(128) k_profile_partials(const lbm_lattice L, double inv_navg, int per_chunk,
                                                          double* __restrict__ part, double* __restrict__ sp2)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= L.nx) return;
    const int y0 = blockIdx.y * per_chunk, y1 = min(y0 + per_chunk, L.ny);
    const long long plane = (long long)L.ny * L.pitch, S = L.cells;
    // the four fields: time-average sums of ux, rho, |u| and ux^2, or ux, rho, uy and uz
    const float* const fld[4] = {AVG ? L.avg : L.ux, AVG ? L.avg + 3 * S : L.rho, AVG ? L.avg + 4 * S : L.uy,
                                 AVG ? L.avg + 5 * S : L.uz};
    double acc[PROF_NF];
#pragma unroll
    for (int k = 0; k < PROF_NF; ++k) acc[k] = 0.0;
    for (int y = y0; y < y1; ++y) {
        const long long col = (long long)y * L.pitch + x;
        double bed = 0.0;
        bool below_solid = true;                           // z = 0 sits on the bed
        for (int z0 = 0; z0 < L.nz; z0 += kProfAhead) {
            uint32_t fk[kProfAhead];
            float v[kProfAhead][4];
#pragma unroll
            for (int j = 0; j < kProfAhead; ++j) {
                const bool in = z0 + j < L.nz;
                const long long c = col + (in ? z0 + j : z0) * plane;
                fk[j] = in ? __ldg(L.flags + c) : FLAG_SOLID;
#pragma unroll
                for (int k = 0; k < 4; ++k) v[j][k] = __ldg(fld[k] + c);
            }
#pragma unroll
            for (int j = 0; j < kProfAhead; ++j) {
                const bool solid = fk[j] & FLAG_SOLID;
                if (!solid) {
                    const CellFields f = cell_fields<AVG>(v[j], inv_navg);
                    acc[PROF_Q] += f.ux;
                    acc[PROF_UXX] += f.uxx;
                    acc[PROF_DRHO] += f.rho - 1.0;
                    acc[PROF_MASS] += f.rho;
                    acc[PROF_NFLUID] += 1.0;
                    acc[PROF_UMAX] = fmax(acc[PROF_UMAX], f.sp);
                    if (z0 + j == L.nz - 1) {
                        acc[PROF_TOP_N] += 1.0;
                        acc[PROF_TOP_DRHO] += f.rho - 1.0;
                        acc[PROF_TOP_UX] += f.ux;
                    }
                    if (below_solid) bed = fmax(bed, f.sp * f.sp);
                }
                below_solid = solid;
            }
        }
        sp2[(long long)y * L.nx + x] = bed;
    }
#pragma unroll
    for (int k = 0; k < PROF_NF; ++k) part[((long long)blockIdx.y * PROF_NF + k) * L.nx + x] = acc[k];
}

// Pass 2: prof[k*nx + x] = the chunks' partials added (max for PROF_UMAX): 8 threads a value, each a run
// of the chunks in order, then the runs in order.  One thread a value waited for 256 loads in turn.
__global__ void __launch_bounds__(256) k_profile_sum(const double* __restrict__ part, int nchunks, int nx,
                                                     double* __restrict__ prof)
{
    __shared__ double run[8][32];
    const long long n = (long long)PROF_NF * nx, i = (long long)blockIdx.x * 32 + threadIdx.x;   // k*nx + x
    const bool most = i / nx == PROF_UMAX;
    const int per = (nchunks + 7) / 8, c0 = threadIdx.y * per, c1 = min(c0 + per, nchunks);
    double s = 0.0;
    if (i < n) {
#pragma unroll 8
        for (int ch = c0; ch < c1; ++ch) {
            const double v = __ldg(part + ch * n + i);
            s = most ? fmax(s, v) : s + v;
        }
    }
    run[threadIdx.y][threadIdx.x] = s;
    __syncthreads();
    if (threadIdx.y || i >= n) return;
    for (int r = 1; r < 8; ++r) s = most ? fmax(s, run[r][threadIdx.x]) : s + run[r][threadIdx.x];
    prof[i] = s;
}

// ---------------------------------------------------------------------------------------------
// FP64 force sums: the force on each body (hull) by momentum exchange, and the body force the
// lattice applies (propellers, jets).  No counterpart in the reference, which infers the boats'
// net force from the momentum-flux difference along the reach (floodsim/reach3d.py:604-609).
//
// From a state (f = the stored post-collision populations of the last step, rho/u its fields,
// colU or uref the wall-model speed) the next step pulls, at a fluid cell x whose source
// x - c_i is a solid cell of body k, the bounced f_opp(i)(x) as f_i(x), corrected by the wall
// function (floodsim/lbm3d.py:61-101); body k then receives -c_i (f_opp(i)(x) + f_i(x)) over
// that link -- its horizontal part only where the source was mirrored by the rigid lid
// (a -z mover under the lid, floodsim/lbm3d.py:54), the lid taking the vertical part.  acc[3*(k-1) + d]: the sum for body k (1..nbody); acc[3*nbody + d]: the applied
// body force, sum of F * force_scale over forced fluid cells.  Lattice units (momentum per
// cell volume per step).  A grid of kBodyBlocks blocks, each thread summing its cells in order,
// then each block and the blocks in fixed orders: deterministic.
// ---------------------------------------------------------------------------------------------
constexpr int kMaxBodies = 16;
constexpr int kBodyBlocks = 1024;
constexpr int kBodyThreads = 256;

// What it adds up for one fluid cell with a force or walls (flag word fk).
template <typename T>
__device__ __forceinline__ void body_force_cell(const lbm_lattice& L, const T* __restrict__ f, float inv_scale,
                                                const uint8_t* __restrict__ body, int nbody, bool ucol, long long c,
                                                uint32_t fk, double* acc)
{
    const long long plane = (long long)L.ny * L.pitch;
    if (fk & FLAG_FORCE) {
        acc[3 * nbody + 0] += (double)(L.Fx[c] * L.force_scale);
        acc[3 * nbody + 1] += (double)(L.Fy[c] * L.force_scale);
        acc[3 * nbody + 2] += (double)(L.Fz[c] * L.force_scale);
    }
    const uint32_t wm = fk & FLAG_WALLS;
    if (!wm || nbody == 0) return;
    const uint32_t row = (uint32_t)(c / L.pitch);
    const int x = (int)(c - (long long)row * L.pitch), y = (int)(row % (uint32_t)L.ny), z = (int)(row / (uint32_t)L.ny);
    int bk[Q];
    bool any = false;
#pragma unroll
    for (int i = 1; i < Q; ++i) {                    // all sources' bytes requested together
        const bool lid = z - cz(i) >= L.nz;          // mirrored into the own layer (the lid's rule)
        const int xs = x - cx(i), ys = y - cy(i), zs = lid ? z : z - cz(i);
        const bool in = (wm & (1u << i)) && zs >= 0 && ys >= 0 && ys < L.ny && xs >= 0 && xs < L.nx;   // bed, y walls, x edges
        bk[i] = in ? (int)__ldg(body + zs * plane + (long long)ys * L.pitch + xs) : 0;
    }
#pragma unroll
    for (int i = 1; i < Q; ++i) {
        if (bk[i] > nbody) bk[i] = 0;
        any |= bk[i] > 0;
        if (z - cz(i) >= L.nz) bk[i] = -bk[i];
    }
    if (!any) return;
    float fw[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i)
        fw[i] = (i > 0 && (wm & (1u << i))) ? ldpop(f + (long long)opp(i) * L.cells + c, i, inv_scale) : 0.f;
    float bounced[Q];
#pragma unroll
    for (int i = 0; i < Q; ++i) bounced[i] = fw[i];
    if (fk & FLAG_WALLFN) {
        const float U = ucol ? ((fk & FLAG_BEDWALL) ? L.colU[(long long)y * L.pitch + x] : 0.f) : L.uref[c];
        wall_function(fw, wm, L.cfw[c], L.ux[c], L.uy[c], L.uz[c], L.rho[c], U);
    }
#pragma unroll
    for (int i = 1; i < Q; ++i)
        if (bk[i]) {
            const double m = (double)bounced[i] + (double)fw[i];
            double* a = acc + 3 * ((bk[i] < 0 ? -bk[i] : bk[i]) - 1);
            a[0] -= cx(i) * m;
            a[1] -= cy(i) * m;
            if (bk[i] > 0) a[2] -= cz(i) * m;      // through the lid: the lid takes the vertical part
        }
}

// Bound by the flags, 4 bytes a cell: a thread reads kBodyAhead quads of them at once (cell by cell where
// they are not 16-byte aligned) and looks closer only at fluid cells with a force or walls, three
// blocks per SM (7.9M cells: 74 us; 77 with two).
constexpr int kBodyAhead = 4;

template <typename T>
__global__ void __launch_bounds__(kBodyThreads, 3) k_body_forces(const lbm_lattice L, const T* __restrict__ f,
                                                                 float inv_scale, const uint8_t* __restrict__ body,
                                                                 int nbody, bool ucol, double* __restrict__ part)
{
    __shared__ double red[kBodyThreads / 32][3 * kMaxBodies + 3];
    const int nacc = 3 * nbody + 3, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double acc[3 * kMaxBodies + 3];
    for (int k = 0; k < nacc; ++k) acc[k] = 0.0;
    const bool vec = (reinterpret_cast<uintptr_t>(L.flags) & 15) == 0;
    const long long quads = L.cells / 4, step = (long long)gridDim.x * blockDim.x;   // pitch: a multiple of 4
    for (long long q0 = (long long)blockIdx.x * blockDim.x + threadIdx.x; q0 < quads; q0 += kBodyAhead * step) {
        uint4 v[kBodyAhead];
#pragma unroll
        for (int j = 0; j < kBodyAhead; ++j) {
            const long long q = q0 + j * step;
            v[j] = make_uint4(FLAG_SOLID, FLAG_SOLID, FLAG_SOLID, FLAG_SOLID);
            if (q < quads && vec) v[j] = __ldg(reinterpret_cast<const uint4*>(L.flags) + q);
            else if (q < quads) v[j] = make_uint4(L.flags[4 * q], L.flags[4 * q + 1], L.flags[4 * q + 2], L.flags[4 * q + 3]);
        }
#pragma unroll 1
        for (int k = 0; k < 4 * kBodyAhead; ++k) {
            uint32_t fk = 0;
#pragma unroll
            for (int j = 0; j < kBodyAhead; ++j)
                if (k / 4 == j) fk = k % 4 == 0 ? v[j].x : k % 4 == 1 ? v[j].y : k % 4 == 2 ? v[j].z : v[j].w;
            if (!(fk & FLAG_SOLID) && (fk & (FLAG_FORCE | FLAG_WALLS)))
                body_force_cell<T>(L, f, inv_scale, body, nbody, ucol, 4 * (q0 + k / 4 * step) + k % 4, fk, acc);
        }
    }
    for (int k = 0; k < nacc; ++k) {
        double s = acc[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) red[warp][k] = s;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < nacc; k += blockDim.x) {
        double s = red[0][k];
        for (int w = 1; w < kBodyThreads / 32; ++w) s += red[w][k];
        part[(long long)k * gridDim.x + blockIdx.x] = s;
    }
}

// out[k] = the blocks' partials of component k: a block per component, each thread every 256th partial
// in order, then a fixed tree.  One thread a component waited for 1024 loads in turn.
__global__ void __launch_bounds__(256) k_body_forces_sum(const double* __restrict__ part, int nblocks, double* __restrict__ out)
{
    __shared__ double red[8];
    const int k = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double s = 0.0;
    for (int b = threadIdx.x; b < nblocks; b += blockDim.x) s += part[(long long)k * nblocks + b];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) red[warp] = s;
    __syncthreads();
    if (threadIdx.x) return;
    for (int w = 1; w < 8; ++w) s += red[w];
    out[k] = s;
}
