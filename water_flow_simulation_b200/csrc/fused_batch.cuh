// fused_batch.cuh -- many lattices of one 16-bit run, stepped by one launch over all their lists.
// Included inside the anonymous namespace of lbm_kernels.cu, after fused_half.cuh and bc_row.
//
// A batch holds K lattices (boat cases of any sizes) in device memory: their lattice
// descriptors, pull-offset tables, 16-bit storage scales and both population buffers of each.
// Work-list entries carry the case in their top 8 bits and the row-segment id (of that case's
// own 64-cell segments, cells_per_lane 2) in the low 24.  One step of the whole batch is then one
// launch over the concatenated lists and one for the outlet rows (output steps: a launch per list, and
// the solid-field and column-mean passes), whatever the sizes of the cases: small
// cases no longer leave the GPU idle between launches or in short tails, and the launch
// count of a step does not grow with the number of cases.  Population buffers alternate by
// step parity, so a chunk of an even number of steps can be captured once as a CUDA graph
// and replayed.
#pragma once

constexpr int kBatchCaseShift = 24;
constexpr uint32_t kBatchSegMask = (1u << kBatchCaseShift) - 1u;
constexpr int kBatchMaxCases = 256;

struct BatchDesc {
    const lbm_lattice* lat;    // K lattice descriptors
    const PullOffsets* po;     // K pull-offset tables
    const float* scale;        // K storage scales
    __half* const* pop0;       // K first population buffers
    __half* const* pop1;       // K second population buffers
};

struct BatchItem {
    int c;
    uint32_t id;
    const __half* fs;
    __half* fd;
};

__device__ __forceinline__ BatchItem batch_item(const BatchDesc& B, int parity, uint32_t e)
{
    BatchItem it;
    it.c = (int)(e >> kBatchCaseShift);
    it.id = e & kBatchSegMask;
    it.fs = parity ? B.pop1[it.c] : B.pop0[it.c];
    it.fd = parity ? B.pop0[it.c] : B.pop1[it.c];
    return it;
}

// Pull-offset tables of the K lattices (set-up).
__global__ void k_batch_pull_offsets(const lbm_lattice* __restrict__ lat, int K, PullOffsets* __restrict__ po)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;     // case * Q + direction
    if (t >= K * Q) return;
    const int c = t / Q, i = t % Q;
    const lbm_lattice& L = lat[c];
    const long long d = (long long)i * L.cells - (long long)cz(i) * L.ny * L.pitch - (long long)cy(i) * L.pitch;
    po[c].d[i] = d;
    po[c].lid[i] = cz(i) == -1 ? (long long)mirz(i) * L.cells - (long long)cy(i) * L.pitch : d;
}

template <int VP, int G, bool OUT, bool AVG>
__global__ void __launch_bounds__(128, VP == 8 ? 3 : 5) k_batch_plain(const BatchDesc B, int parity,
                                                                     const uint32_t* __restrict__ list, int nlist)
{
    constexpr int PER_WARP = 32 / G;
    const int lane = threadIdx.x & 31, gl = lane % G, grp = lane / G;
    const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), W = (int)((gridDim.x * blockDim.x) >> 5);
    for (long long b = (long long)gw * PER_WARP; b < nlist; b += (long long)W * PER_WARP) {
        const bool valid = b + grp < nlist;
        const BatchItem it = batch_item(B, parity, __ldg(list + (valid ? b + grp : b)));
        h_plain_segment<VP, G, OUT, AVG>(B.lat[it.c], B.po[it.c], it.fs, it.fd, __ldg(B.scale + it.c), it.id, gl,
                                         valid);
    }
}

// One 32-cell pass of a batch's special entry e (64-cell segments): part 0 or 1 of it.
template <bool OUT, bool UCOL, bool AVG, typename T>
__device__ __forceinline__ void batch_cell_pass(const BatchDesc& B, int parity, uint32_t e, int part, int lane)
{
    constexpr int SEG = 64;
    const BatchItem it = batch_item(B, parity, e);
    const lbm_lattice& L = B.lat[it.c];
    const float scale = __ldg(B.scale + it.c);
    int seg, y, z;
    decode_row(it.id, (L.pitch + SEG - 1) / SEG, L.ny, seg, y, z);
    const int xa = seg * SEG + part * 32;
    if (xa >= L.pitch) return;                             // warp-uniform
    // 32-bit indexes: a case has at most 2^24 segments, 2^30 cells.  Its planes' bases lie in memory here and
    // not in uniform registers, and 64-bit sums cost 0.7 % (five cases of 1.7M cells, 20 steps: 2718 and 2703 us).
    cell_pass<SEG, OUT, UCOL, AVG, T, int>(L, reinterpret_cast<const T*>(it.fs), reinterpret_cast<T*>(it.fd), scale,
                                           1.0f / scale, xa, y, z, lane, pass_flags(L, xa + lane, y, z));
}

// A warp pass over edge entries b and b+1 of a batch, 16 lanes each.  The two may be of cases whose
// outlet cells sit at different places in their lanes, which edge_lane decides per group.
template <bool OUT, bool AVG, typename T>
__device__ __forceinline__ void batch_edge_pass(const BatchDesc& B, int parity, const uint32_t* __restrict__ list,
                                                long long b, int nlist, int lane)
{
    constexpr int SEG = 64, G = 16;
    const bool valid = b + lane / G < nlist;
    const BatchItem it = batch_item(B, parity, __ldg(list + (valid ? b + lane / G : b)));
    const lbm_lattice& L = B.lat[it.c];
    const float scale = __ldg(B.scale + it.c);
    int seg, y, z;
    decode_row(it.id, (L.pitch + SEG - 1) / SEG, L.ny, seg, y, z);
    edge_lane<G, OUT, AVG, T>(L, B.po[it.c], reinterpret_cast<const T*>(it.fs), reinterpret_cast<T*>(it.fd), scale,
                              1.0f / scale, seg * SEG + lane % G * 4, y, z, lane % G, valid);
}

template <bool OUT, bool UCOL, bool AVG>
__global__ void __launch_bounds__(128, 4) k_batch_cells(const BatchDesc B, int parity,
                                                                 const uint32_t* __restrict__ special, int n_special)
{
    const int lane = threadIdx.x & 31;
    const long long W = ((long long)gridDim.x * blockDim.x) >> 5, total = 2LL * n_special;
    for (long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < total; t += W)
        batch_cell_pass<OUT, UCOL, AVG, __half>(B, parity, __ldg(special + (t >> 1)), (int)(t & 1), lane);
}

template <bool OUT, bool AVG>
__global__ void __launch_bounds__(128, 4) k_batch_edge(const BatchDesc B, int parity,
                                                                const uint32_t* __restrict__ edge, int n_edge)
{
    const int lane = threadIdx.x & 31;
    const long long W = ((long long)gridDim.x * blockDim.x) >> 5;
    for (long long b = 2 * (((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5); b < n_edge; b += 2 * W)
        batch_edge_pass<OUT, AVG, __half>(B, parity, edge, b, n_edge, lane);
}

// The three lists of a step in one launch (as k_all_lists): special passes, edge passes, plain passes.
// Five cases of 1.7M cells: 134 us a step against 145 in three launches (137 at 4 CTAs per SM).
template <bool UCOL>
__global__ void __launch_bounds__(128, 5) k_batch_all(const BatchDesc B, int parity, const lbm_batch b)
{
    const int lane = threadIdx.x & 31;
    int t = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (t < 2 * b.n_special) {
        batch_cell_pass<false, UCOL, false, __half>(B, parity, __ldg(b.rows_special + (t >> 1)), t & 1, lane);
        return;
    }
    t -= 2 * b.n_special;
    if (2 * t < b.n_edge) {
        batch_edge_pass<false, false, __half>(B, parity, b.rows_edge, 2LL * t, b.n_edge, lane);
        return;
    }
    t -= (b.n_edge + 1) / 2;
    const int p = 2 * t, grp = lane >> 4;
    if (p < b.n_plain) {
        const bool valid = p + grp < b.n_plain;
        const BatchItem it = batch_item(B, parity, __ldg(b.rows_plain + (valid ? p + grp : p)));
        h_plain_segment<4, 16, false, false>(B.lat[it.c], B.po[it.c], it.fs, it.fd, __ldg(B.scale + it.c), it.id,
                                             lane & 15, valid);
    }
}

template <bool AVG>
__global__ void k_batch_solid_out(const BatchDesc B, const uint32_t* __restrict__ list, int nlist)
{
    const int lane = threadIdx.x & 31;
    const int gw = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), W = (int)((gridDim.x * blockDim.x) >> 5);
    for (int w = gw; w < nlist; w += W) {
        const uint32_t e = __ldg(list + w);
        solid_segment<2, AVG>(B.lat[e >> kBatchCaseShift], e & kBatchSegMask, lane);
    }
}

// blockIdx.y = case
__global__ void k_batch_column_mean(const BatchDesc B)
{
    column_mean_at(B.lat[blockIdx.y], (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

// Outlet rows of the cases whose x = nx-2 and x = nx-1 fall in different segments; blockIdx.y = case.
__global__ void k_batch_bc_rows(const BatchDesc B, int parity)
{
    const lbm_lattice& L = B.lat[blockIdx.y];
    if ((L.nx - 1) % 64 != 0) return;
    __half* fd = parity ? B.pop0[blockIdx.y] : B.pop1[blockIdx.y];
    bc_row<__half>(L, fd, 2, __ldg(B.scale + blockIdx.y), (long long)blockIdx.x * blockDim.x + threadIdx.x);
}

// ---------------------------------------------------------------------------------------------
// Persistent chunk: `nsteps` steps of the whole batch in ONE cooperative launch.  Every CTA stays
// resident for the chunk; a step is two phases separated by grid barriers:
//   phase 1  the step's segment tasks, statically interleaved over all warps of the grid in one
//            task space [special | edge | plain groups]: a special task is half a 64-cell segment
//            (one cell per lane), an edge task two segments (16 lanes of 4 cells each), a plain
//            task four (8 lanes of 8 cells each); so every warp works through some of each kind and the
//            latency-bound special segments run beside the bandwidth-bound plain ones;
//   phase 2  the outlet rows of cases whose x = nx-2 and nx-1 lie in different segments, and on
//            the chunk's last (output) step the solid segments' fields and the column means.
// The per-segment device functions are those of the per-kernel batch step, so both give the
// same populations bit for bit.  Barrier waits are bounded by kBarrierTimeoutNs of the global
// timer: a CTA that runs out raises an abort flag in the sync words, every CTA then leaves the
// chunk, and bit 1 of every case's status word is set (the state is not to be trusted).
// sync: 4 uint32 of device memory, zeroed by the host before the launch (count, generation,
// abort flag, spare).
// ---------------------------------------------------------------------------------------------
constexpr unsigned long long kBarrierTimeoutNs = 2000000000ULL;

__device__ __forceinline__ unsigned long long global_timer_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid-wide barrier of a cooperative launch; false when a wait ran out (here or in another CTA).
__device__ bool grid_barrier(uint32_t* sync, unsigned nblocks)
{
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        volatile uint32_t* vgen = sync + 1;
        volatile uint32_t* vabort = sync + 2;
        const uint32_t g = *vgen;
        __threadfence();
        const uint32_t arrived = atomicAdd(sync, 1u);
        if (arrived == nblocks - 1) {
            atomicExch(sync, 0u);
            __threadfence();
            atomicAdd(sync + 1, 1u);
        } else {
            const unsigned long long t0 = global_timer_ns();
            while (*vgen == g) {
                if (*vabort) { ok = 0; break; }
                if (global_timer_ns() - t0 > kBarrierTimeoutNs) {
                    atomicExch(sync + 2, 1u);
                    ok = 0;
                    break;
                }
                __nanosleep(256);
            }
        }
        __threadfence();
    }
    __syncthreads();
    return ok != 0;
}

template <bool OUT, bool UCOL, bool AVG>
__device__ __forceinline__ void batch_tasks(const BatchDesc& B, int parity, const uint32_t* __restrict__ special,
                                            int n_special, const uint32_t* __restrict__ edge, int n_edge,
                                            const uint32_t* __restrict__ plain, int n_plain)
{
    constexpr int VP = 8, G = 8, PER_WARP = 32 / G;
    const int lane = threadIdx.x & 31;
    const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const long long W = ((long long)gridDim.x * blockDim.x) >> 5;
    const long long n_pgroups = (n_plain + PER_WARP - 1) / PER_WARP;
    const long long ns = 2LL * n_special, ne = (n_edge + 1LL) / 2, total = ns + ne + n_pgroups;
    for (long long t = gw; t < total; t += W) {
        // populations are read with coherent loads (hcoh): this launch wrote them in earlier steps
        if (t < ns) {
            batch_cell_pass<OUT, UCOL, AVG, hcoh>(B, parity, __ldg(special + (t >> 1)), (int)(t & 1), lane);
        } else if (t < ns + ne) {
            batch_edge_pass<OUT, AVG, hcoh>(B, parity, edge, 2 * (t - ns), n_edge, lane);
        } else {
            const long long b = (t - ns - ne) * PER_WARP;
            const int gl = lane % G, grp = lane / G;
            const bool valid = b + grp < n_plain;
            const BatchItem it = batch_item(B, parity, __ldg(plain + (valid ? b + grp : b)));
            h_plain_segment<VP, G, OUT, AVG, hcoh>(B.lat[it.c], B.po[it.c], reinterpret_cast<const hcoh*>(it.fs),
                                                   reinterpret_cast<hcoh*>(it.fd), __ldg(B.scale + it.c), it.id, gl,
                                                   valid);
        }
    }
}

template <bool UCOL, bool AVG_LAST>
__global__ void __launch_bounds__(128, 3) k_batch_chunk(const BatchDesc B, int K, int parity0, int nsteps,
                                                      const uint32_t* __restrict__ special, int n_special,
                                                      const uint32_t* __restrict__ edge, int n_edge,
                                                      const uint32_t* __restrict__ plain, int n_plain,
                                                      const uint32_t* __restrict__ solid, int n_solid,
                                                      int max_rows, int max_columns, uint32_t* sync)
{
    const unsigned nblocks = gridDim.x;
    const long long gtid = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long nthreads = (long long)gridDim.x * blockDim.x;
    for (int s = 0; s < nsteps; ++s) {
        const int parity = (parity0 + s) & 1;
        const bool last = s == nsteps - 1;
        if (last) batch_tasks<true, UCOL, AVG_LAST>(B, parity, special, n_special, edge, n_edge, plain, n_plain);
        else batch_tasks<false, UCOL, false>(B, parity, special, n_special, edge, n_edge, plain, n_plain);
        bool ok = grid_barrier(sync, nblocks);
        if (ok) {
            // outlet rows of the cases that need their own pass (the fields they write are not
            // read by the solid-field or column-mean work of this phase)
            for (long long j = gtid; j < (long long)K * max_rows; j += nthreads) {
                const int c = (int)(j / max_rows);
                const lbm_lattice& L = B.lat[c];
                if ((L.nx - 1) % 64 != 0) continue;
                hcoh* fd = reinterpret_cast<hcoh*>(parity ? B.pop0[c] : B.pop1[c]);
                bc_row<hcoh>(L, fd, 2, __ldg(B.scale + c), j % max_rows);
            }
            if (last) {
                const int lane = threadIdx.x & 31;
                for (long long w = gtid >> 5; w < n_solid; w += nthreads >> 5) {
                    const uint32_t e = __ldg(solid + w);
                    solid_segment<2, AVG_LAST>(B.lat[e >> kBatchCaseShift], e & kBatchSegMask, lane);
                }
                if (UCOL)
                    for (long long j = gtid; j < (long long)K * max_columns; j += nthreads)
                        column_mean_at<true>(B.lat[j / max_columns], j % max_columns);
            }
            if (!last) ok = grid_barrier(sync, nblocks);
        }
        if (!ok) {
            if (gtid < K) atomicOr(B.lat[gtid].status, 2);
            return;
        }
    }
}
