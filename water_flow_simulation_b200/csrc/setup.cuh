// setup.cuh -- kernels that open a case: row padding, cell flags, work lists, start state.
// Included inside the anonymous namespace of lbm_kernels.cu.
//
// Each runs once per case (or after a change of forces or friction) and is bound by the bytes
// of the per-cell arrays it reads and writes once, so a thread takes four cells with vector
// accesses, a warp reads a segment's flags together, and the ordered compaction runs on all SMs.
#pragma once

// A thread's row and first cell where blocks of 128 threads, four cells each, cover rows of `pitch`
// cells (row_grid): no 64-bit division per cell.  False: nothing to do.
__device__ __forceinline__ bool row_of(long long rows, int pitch, long long& row, int& x)
{
    row = (long long)blockIdx.z * gridDim.y + blockIdx.y;
    x = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    return row < rows && x < pitch;
}
dim3 row_grid(long long rows, int pitch)
{
    const unsigned gy = (unsigned)(rows < 65535 ? rows : 65535);
    return dim3((unsigned)((pitch / 4 + 127) / 128), gy, (unsigned)((rows + gy - 1) / gy));
}

// Rows of nx elements (1 or 4 bytes each) to rows of `pitch`, the rest filled with `pad`.  A thread takes
// four cells of kPitchRows consecutive rows, all requested together: with one row a thread the
// blocks came and went 30 deep, each waiting for one load (36M cells: bytes 40 -> 25 us, floats 58 -> 46).
constexpr int kPitchRows = 4;

template <typename T>
__global__ void __launch_bounds__(128) k_pitch_rows(const T* __restrict__ src, T* __restrict__ dst, int nx, int pitch,
                                                    long long rows, T pad)
{
    long long group;
    int x;
    if (!row_of((rows + kPitchRows - 1) / kPitchRows, pitch, group, x)) return;
    const long long row0 = group * kPitchRows;
    struct __align__(4) Four { T v[4]; } o[kPitchRows];
#pragma unroll
    for (int j = 0; j < kPitchRows; ++j)
#pragma unroll
        for (int k = 0; k < 4; ++k)
            o[j].v[k] = row0 + j < rows && x + k < nx ? __ldg(src + (row0 + j) * nx + x + k) : pad;
#pragma unroll
    for (int j = 0; j < kPitchRows; ++j)
        if (row0 + j < rows) *reinterpret_cast<Four*>(dst + (row0 + j) * pitch + x) = o[j];
}

// Cell flags from unvectorised accesses: arrays at any alignment.
template <int I>
__device__ __forceinline__ void flag_dir(uint32_t& wm, const uint8_t* __restrict__ solid, const lbm_lattice& L,
                                         int x, int y, int z)
{
    const int xs = x - cx(I), ys = y - cy(I);
    int zs = z - cz(I);
    if (xs < 0 || xs >= L.nx) return;
    if (zs >= L.nz) zs = z;
    bool wall = (ys < 0 || ys >= L.ny || zs < 0);
    if (!wall) wall = solid[xs + (long long)L.pitch * (ys + (long long)L.ny * zs)] != 0;
    if (wall) wm |= (1u << I);
}
template <int... Is>
__device__ __forceinline__ void flag_all(std::integer_sequence<int, Is...>, uint32_t& wm,
                                         const uint8_t* __restrict__ solid, const lbm_lattice& L, int x, int y, int z)
{
    (flag_dir<Is>(wm, solid, L, x, y, z), ...);
}

// The flag word of a fluid cell: its wall mask, force, wall function (friction, and a usable wall
// normal and face) and bed/bank bits.
__host__ __device__ __forceinline__ uint32_t fluid_flags(uint32_t wm, float fx, float fy, float fz, float cf, bool bedwall)
{
    constexpr uint32_t PX = dir_mask([](int i) { return cx(i) == 1; }), NX = dir_mask([](int i) { return cx(i) == -1; });
    constexpr uint32_t PY = dir_mask([](int i) { return cy(i) == 1; }), NY = dir_mask([](int i) { return cy(i) == -1; });
    constexpr uint32_t PZ = dir_mask([](int i) { return cz(i) == 1; }), NZ = dir_mask([](int i) { return cz(i) == -1; });
    uint32_t fw = wm;
    if (fx != 0.f || fy != 0.f || fz != 0.f) fw |= FLAG_FORCE;
    if (wm && cf > 0.f) {
        const bool normal = popc32(wm & PX) != popc32(wm & NX) || popc32(wm & PY) != popc32(wm & NY) ||
                            popc32(wm & PZ) != popc32(wm & NZ);
        if (normal && (wm & 0x7Eu)) fw |= FLAG_WALLFN;
    }
    if (bedwall) fw |= FLAG_BEDWALL;
    return fw;
}

__global__ void k_build_flags(const lbm_lattice L, const uint8_t* __restrict__ solid,
                              const uint8_t* __restrict__ bedwall, uint32_t* __restrict__ flags)
{
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= L.cells) return;
    const int x = (int)(c % L.pitch), y = (int)((c / L.pitch) % L.ny), z = (int)(c / ((long long)L.pitch * L.ny));
    if (x >= L.nx) { flags[c] = FLAG_GHOST | FLAG_SOLID; return; }
    if (solid[c]) { flags[c] = FLAG_SOLID; return; }
    uint32_t wm = 0;
    flag_all(std::make_integer_sequence<int, Q>{}, wm, solid, L, x, y, z);
    flags[c] = fluid_flags(wm, L.Fx[c], L.Fy[c], L.Fz[c], L.cfw[c], bedwall && bedwall[c]);
}

// The same for four cells per thread (x0 a multiple of 4; 16-byte aligned float arrays and flags,
// 4-byte aligned masks).  The solid cells x0-1 .. x0+4 of each of the nine source rows are six
// bits, and every direction's four wall bits a shift of one of them: 36M cells in 246 us against
// 845 with 18 bounds checks and byte loads per cell.
__global__ void __launch_bounds__(128) k_build_flags4(const lbm_lattice L, const uint8_t* __restrict__ solid,
                                                      const uint8_t* __restrict__ bedwall, uint32_t* __restrict__ flags)
{
    long long row;
    int x0;
    if (!row_of((long long)L.ny * L.nz, L.pitch, row, x0)) return;
    const int y = (int)((uint32_t)row % (uint32_t)L.ny), z = (int)((uint32_t)row / (uint32_t)L.ny);
    const long long c = row * L.pitch + x0;
    uint32_t inside = 0;                                   // bit j: x0 - 1 + j lies in [0, nx)
#pragma unroll
    for (int j = 0; j < 6; ++j) inside |= (x0 - 1 + j >= 0 && x0 - 1 + j < L.nx) ? 1u << j : 0u;
    uint32_t rows[3][3];                                   // [sy + 1][sz + 1]: source row (y + sy, z + sz)
#pragma unroll
    for (int sy = -1; sy <= 1; ++sy)
#pragma unroll
        for (int sz = -1; sz <= 1; ++sz) {
            const int ys = y + sy, zs = z + sz >= L.nz ? z : z + sz;       // the lid mirrors
            uint32_t m = 0x3Fu;                                            // y walls and the bed
            if (ys >= 0 && ys < L.ny && zs >= 0) {
                const uint8_t* s = solid + ((long long)zs * L.ny + ys) * L.pitch + x0;
                const uint32_t w = __vcmpne4(__ldg(reinterpret_cast<const uint32_t*>(s)), 0u) & 0x08040201u;
                m = ((w * 0x01010101u) >> 24) << 1;
                if (inside & 1u) m |= __ldg(s - 1) ? 1u : 0u;
                if (inside & 0x20u) m |= __ldg(s + 4) ? 0x20u : 0u;
            }
            rows[sy + 1][sz + 1] = m & inside;
        }
    const float4 fx = __ldg(reinterpret_cast<const float4*>(L.Fx + c)), fy = __ldg(reinterpret_cast<const float4*>(L.Fy + c));
    const float4 fz = __ldg(reinterpret_cast<const float4*>(L.Fz + c)), cf = __ldg(reinterpret_cast<const float4*>(L.cfw + c));
    const uint32_t bw = bedwall ? __ldg(reinterpret_cast<const uint32_t*>(bedwall + c)) : 0u;
    const float f[3][4] = {{fx.x, fx.y, fx.z, fx.w}, {fy.x, fy.y, fy.z, fy.w}, {fz.x, fz.y, fz.z, fz.w}};
    const float cfs[4] = {cf.x, cf.y, cf.z, cf.w};
    uint32_t out[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        uint32_t wm = 0;
#pragma unroll
        for (int i = 1; i < Q; ++i) wm |= ((rows[1 - cy(i)][1 - cz(i)] >> (k + 1 - cx(i))) & 1u) << i;
        if (x0 + k >= L.nx) out[k] = FLAG_GHOST | FLAG_SOLID;
        else if ((rows[1][1] >> (k + 1)) & 1u) out[k] = FLAG_SOLID;
        else out[k] = fluid_flags(wm, f[0][k], f[1][k], f[2][k], cfs[k], (bw >> (8 * k)) & 0xffu);
    }
    *reinterpret_cast<uint4*>(flags + c) = make_uint4(out[0], out[1], out[2], out[3]);
}

// Four flags: one access, or one flag at a time where they are not 16-byte aligned.
__device__ __forceinline__ void load_flags4(uint32_t (&fk)[4], const uint32_t* p, bool vec)
{
    if (vec) {
        const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
        fk[0] = v.x; fk[1] = v.y; fk[2] = v.z; fk[3] = v.w;
    } else {
        for (int k = 0; k < 4; ++k) fk[k] = __ldg(p + k);
    }
}

// 0 plain, 1 solid, 2 special, 3 edge (see fused_split.cuh): 8*V lanes (at most 32) of four flags each
// per segment of 32*V cells, kClassAhead segments in flight per thread (36M cells: 75 us, 99
// with one).
constexpr int kClassAhead = 4;
__global__ void __launch_bounds__(256) k_classify(const lbm_lattice L, int V, uint8_t* __restrict__ cls)
{
    const int SEG = 32 * V, G = V >= 4 ? 32 : 8 * V, lane = threadIdx.x & 31, gl = lane % G;
    const int nseg = (L.pitch + SEG - 1) / SEG;
    const long long n = (long long)nseg * L.ny * L.nz;
    const long long id0 = ((long long)blockIdx.x * blockDim.x + threadIdx.x) / G, step = (long long)gridDim.x * blockDim.x / G;
    const bool vec = (reinterpret_cast<uintptr_t>(L.flags) & 15) == 0;
    const unsigned group = (G == 32 ? 0xffffffffu : ((1u << G) - 1u) << (lane - gl));
    uint32_t fk[kClassAhead][4];                           // the first four flags of each segment, requested together
#pragma unroll
    for (int j = 0; j < kClassAhead; ++j) {
        const uint32_t id = id0 + j * step < n ? (uint32_t)(id0 + j * step) : 0u;            // ids are 32-bit
        const int x = (int)(id % (uint32_t)nseg) * SEG + 4 * gl;
#pragma unroll
        for (int k = 0; k < 4; ++k) fk[j][k] = FLAG_GHOST | FLAG_SOLID;
        if (x < L.pitch) load_flags4(fk[j], L.flags + (long long)(id / (uint32_t)nseg) * L.pitch + x, vec);
    }
#pragma unroll
    for (int j = 0; j < kClassAhead; ++j) {
        const long long id = id0 + j * step;
        const bool valid = id < n;
        const uint32_t id32 = valid ? (uint32_t)id : 0u, yz = id32 / (uint32_t)nseg;
        const int seg = (int)(id32 % (uint32_t)nseg), y = (int)(yz % (uint32_t)L.ny), z = (int)(yz / (uint32_t)L.ny);
        const int xa = seg * SEG, xb = min(xa + SEG, L.pitch);
        bool fluid_seen = false, any_special = false;
        for (int x = xa + 4 * gl; x < xb; x += 4 * G) {
            if (x != xa + 4 * gl) load_flags4(fk[j], L.flags + (long long)yz * L.pitch + x, vec);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                fluid_seen |= (fk[j][k] & FLAG_SOLID) == 0;
                if (x + k < L.nx) any_special |= (fk[j][k] & (FLAG_SOLID | FLAG_WALLS | FLAG_WALLFN | FLAG_FORCE)) != 0;
            }
        }
        const bool all_solid = (__ballot_sync(0xffffffffu, fluid_seen) & group) == 0;
        any_special = (__ballot_sync(0xffffffffu, any_special) & group) != 0;
        // open rows: clear of the y walls and the bed; the row under the lid counts (its -z movers
        // read the own row's mirrored populations at constant offsets)
        if (L.sponge_cols > 0 && xb > L.nx - L.sponge_cols) any_special = true;   // per-cell relaxation time
        const bool interior_row = y >= 1 && y <= L.ny - 2 && z >= 1 && z <= L.nz - 1;
        const bool clear_of_edges = seg > 0 && xa + SEG < L.nx;
        int c = 2;
        if (all_solid) c = 1;
        else if (interior_row && !any_special) c = clear_of_edges ? 0 : 3;
        if (valid && gl == 0) cls[id] = (uint8_t)c;
    }
}

// Ordered stream compaction of the four classes.  CTA b takes `chunk` entries (a multiple of 16)
// from b*chunk on; where its entries go follows from the counts of every class before them,
// which it makes itself from the class bytes (all of them are a few hundred KB of L2): no pass in
// between, no scratch.  One CTA alone took 1151 us on the 578k segments of the 36M-cell reach;
// all SMs take 36.  counts[c] receives the number of segments of class c, lists[c] their ids in order.
__global__ void __launch_bounds__(1024) k_compact(const uint8_t* __restrict__ cls, long long n, long long chunk,
                                                  uint32_t* __restrict__ plain, uint32_t* __restrict__ solid,
                                                  uint32_t* __restrict__ special, uint32_t* __restrict__ edge,
                                                  int* __restrict__ counts)
{
    constexpr int NC = 4;
    __shared__ int warp_tot[NC][32];
    __shared__ int base[NC];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const long long first = blockIdx.x * chunk, last = min(first + chunk, n);
    uint32_t* const lists[NC] = {plain, solid, special, edge};
    int before[NC] = {0, 0, 0, 0};
    if ((reinterpret_cast<uintptr_t>(cls) & 15) == 0) {
        for (long long i = tid; i < first / 16; i += blockDim.x) {
            const uint4 v = __ldg(reinterpret_cast<const uint4*>(cls) + i);
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int k = 0; k < NC; ++k) before[k] += __popc(__vcmpeq4(w[j], 0x01010101u * k)) >> 3;
        }
    } else {
        for (long long i = tid; i < first; i += blockDim.x)
#pragma unroll
            for (int k = 0; k < NC; ++k) before[k] += cls[i] == k;
    }
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        const int t = __reduce_add_sync(0xffffffffu, before[k]);
        if (lane == 0) warp_tot[k][warp] = t;
    }
    __syncthreads();
    if (tid < NC) {
        int sum = 0;
        for (int w = 0; w < nwarps; ++w) sum += warp_tot[tid][w];
        base[tid] = sum;
    }
    __syncthreads();
    for (long long start = first; start < last; start += blockDim.x) {
        const long long i = start + tid;
        const int c = i < last ? cls[i] : NC;
        int rank[NC];
#pragma unroll
        for (int k = 0; k < NC; ++k) {
            const unsigned m = __ballot_sync(0xffffffffu, c == k);
            rank[k] = __popc(m & ((1u << lane) - 1u));
            if (lane == 0) warp_tot[k][warp] = __popc(m);
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < NC; ++k)
            if (c == k) {
                int acc = base[k];
                for (int w = 0; w < warp; ++w) acc += warp_tot[k][w];
                lists[k][acc + rank[k]] = (uint32_t)i;
            }
        __syncthreads();
        if (tid < NC) {
            int sum = 0;
            for (int w = 0; w < nwarps; ++w) sum += warp_tot[tid][w];
            base[tid] += sum;
        }
        __syncthreads();
    }
    if (tid < NC && last == n) counts[tid] = base[tid];
}

// f = feq(1, (u,0,0)) of direction i evaluated with the operation order and float64/float32 mix of
// the reference's NumPy start (floodsim/lbm3d.py:377-384): cu = (3*c_x)*u and the quadratic in
// float64, 1.5*u*u in float32, rounded once to float32 at the end.
__device__ __forceinline__ float start_value(int cxi, double w, float u)
{
    const double ud = (double)u;
    const float q = __fmul_rn(__fmul_rn(1.5f, u), u);
    const double cu = __dmul_rn((double)(3 * cxi), ud);
    const double poly = __dsub_rn(__dadd_rn(__dadd_rn(1.0, cu), __dmul_rn(__dmul_rn(0.5, cu), cu)), (double)q);
    return __double2float_rn(__dmul_rn(w, poly));
}
__device__ __forceinline__ float stored_start(float f, float, float, float*) { return f; }
__device__ __forceinline__ __half stored_start(float f, float w, float scale, __half*)
{
    return __float2half_rn(__fmul_rn(__fsub_rn(f, w), scale));
}

// Start state by rows:
// inside a row every fluid cell starts alike and every other cell at rest, so the 19 stored values
// of either are made once per block and a thread writes four cells of each direction with one
// access.  T = float, or __half for 16-bit storage (scaled deviations from the weights).
// 36M cells with 16-bit storage: 247 us, 6.1 TB/s, against 380 for one cell per thread.
template <typename T>
__global__ void __launch_bounds__(128) k_start_rows(const lbm_lattice L, T* __restrict__ f, float scale)
{
    __shared__ T value[2][Q];
    long long row;
    int x;
    const bool active = row_of((long long)L.ny * L.nz, L.pitch, row, x);
    if (row >= (long long)L.ny * L.nz) return;             // the whole block
    const int z = (int)(row / L.ny), y = (int)(row % L.ny);
    if (threadIdx.x < 2 * Q) {
        const int i = threadIdx.x % Q, fluid = threadIdx.x / Q;
        const double w64 = i == 0 ? wgt64(0) : (i < 7 ? wgt64(1) : wgt64(7));
        const float w = i == 0 ? wgt(0) : (i < 7 ? wgt(1) : wgt(7));
        value[fluid][i] = stored_start(start_value(cx(i), w64, fluid ? L.uin[y + (long long)L.ny * z] : 0.f), w, scale,
                                       (T*)nullptr);
    }
    __syncthreads();
    if (!active) return;
    const long long c = row * L.pitch + x;
    const uint4 fl = __ldg(reinterpret_cast<const uint4*>(L.flags + c));
    const bool fluid[4] = {x < L.nx && !(fl.x & FLAG_SOLID), x + 1 < L.nx && !(fl.y & FLAG_SOLID),
                           x + 2 < L.nx && !(fl.z & FLAG_SOLID), x + 3 < L.nx && !(fl.w & FLAG_SOLID)};
    struct __align__(4 * sizeof(T)) Four { T v[4]; };
#pragma unroll
    for (int i = 0; i < Q; ++i) {
        Four o;
#pragma unroll
        for (int k = 0; k < 4; ++k) o.v[k] = fluid[k] ? value[1][i] : value[0][i];
        *reinterpret_cast<Four*>(f + (long long)i * L.cells + c) = o;
    }
}

// The same for arrays at any alignment, one cell per thread.
template <typename T>
__global__ void k_start_cells(const lbm_lattice L, T* __restrict__ f, float scale)
{
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= L.cells) return;
    const int x = (int)(c % L.pitch), y = (int)((c / L.pitch) % L.ny), z = (int)(c / ((long long)L.pitch * L.ny));
    const bool fluid = x < L.nx && !(L.flags[c] & FLAG_SOLID);
    const float u = fluid ? L.uin[y + (long long)L.ny * z] : 0.f;
#pragma unroll
    for (int i = 0; i < Q; ++i)
        f[(long long)i * L.cells + c] = stored_start(start_value(cx(i), wgt64(i), u), wgt(i), scale, (T*)nullptr);
}
