// surrogate.cu -- BF16 tensor-core kernels of the learned warm start (sm_100a, tcgen05).
//
// The network is a small 3D convolutional encoder-decoder on a coarse copy of the lattice.
// Every convolution, forward and backward, is a product on 5th-generation tensor cores:
//   D[M x N] = A[M x K] * B[N x K]^T      A, B bf16, both K-major; accumulation f32 in TMEM
// finished by fused epilogues (bias, ReLU, bf16 store).  k_conv_fwd and k_conv_back read the
// grids in place (no column matrix), k_conv_in that of the first layer (8 channels); the weight gradients
// go through gather kernels (k_im2col_t, transposes) and lbm_gemm_bf16, whose kernel is chosen per call:
//   k_gemm_ws    products with >= 1024 rows and >= 128 columns (none of the network's): persistent,
//                warp-specialised, TMA ring + MMA thread + epilogue warps, accumulator transposed in TMEM;
//   k_gemm_tma   smaller products (the weight gradients): one tile per CTA, TMA ring, MMA warp;
//   k_gemm_bf16  when no tensor map can be made: the register-staged kernel described here.
//
// k_gemm_bf16 tile: one CTA computes 128 rows x BN columns.  Per 64-wide K step, the 4 warps copy
// the A and B tiles (16-byte vectors, zero-filled past M, N, K) into shared memory in the
// 128-byte-swizzled K-major layout the UMMA matrix descriptors describe; one elected thread
// then issues four tcgen05.mma (K = 16 each) accumulating into TMEM and commits them to an
// mbarrier that every thread waits on (bounded: on timeout the block sets an error flag,
// skips the rest, still frees its TMEM and returns).  The epilogue reads the accumulator
// with tcgen05.ld (warp w owns TMEM lanes 32w..32w+31 = tile rows) and applies bias/ReLU.
#include <cuda.h>
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "channels.cuh"
#include "errors.cuh"
#include "shared_mem.cuh"
#include "tensor_map.cuh"
#include "../../include/lbm_b200.h"

using namespace wfs;

namespace {

constexpr int GM = 128;                     // tile rows = tcgen05.mma M
constexpr int GK = 64;                      // K per shared tile: one 128-byte row of bf16
constexpr long long kWaitPolls = 1LL << 22; // mbarrier polls before a block gives up

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Matrix descriptor of a K-major operand tile in the 128-byte swizzle: rows of 128 bytes,
// groups of 8 rows 1024 bytes apart (fields as in the PTX tcgen05 shared-memory descriptor).
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr)
{
    return (uint64_t)((saddr & 0x3FFFFu) >> 4)      // start address, 16-byte units
         | ((uint64_t)1 << 16)                      // leading byte offset (16 B; unused when swizzled)
         | ((uint64_t)(1024 >> 4) << 32)            // stride byte offset: 8 rows x 128 B
         | ((uint64_t)1 << 46)                      // descriptor version
         | ((uint64_t)2 << 61);                     // 128-byte swizzle
}

// Instruction descriptor: kind::f16 with bf16 A and B, f32 D, both K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t idesc_bf16(int n)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(GM >> 4) << 24);
}

// Byte offset of 16-byte chunk j (0..7) of row r in a 128-byte-swizzled tile.
__device__ __forceinline__ uint32_t sw128(int r, int j)
{
    return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + ((j ^ (r & 7)) << 4));
}

__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
        :
        : "r"(tmem), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity)
{
    for (long long i = 0; i < kWaitPolls; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done)
            : "r"(mbar), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

// The convolutions' and k_gemm_tma's loading and MMA warps stay converged and let one elected lane issue,
// with descriptors made by adding to one word: under a branch on the lane number each operand of a
// tcgen05 or TMA instruction is moved to a uniform register on its own.  Convolutions 128 -> 128 and
// 128 -> 64 on 15k voxels 30.3 -> 25.8 and 28.0 -> 22.8 us, weight gradients over 12k voxels 68 -> 64.
__device__ __forceinline__ bool elect_one()
{
    uint32_t on;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(on));
    return on != 0;
}
// A whole warp's bounded wait; false if it ran out or `failed` (in shared memory) is set.
__device__ __forceinline__ bool warp_wait(uint32_t mbar, uint32_t parity, const int* failed)
{
    return __all_sync(0xffffffffu, mbar_wait(mbar, parity) && *(const volatile int*)failed == 0);
}
// The four MMAs (K = 16 each) of one K tile, operands at shared addresses a and b (K-major, 128-byte
// swizzle).  The low descriptor word holds the address in 16-byte units, so a K step of 32 bytes adds 2.
__device__ __forceinline__ void mma_ktile(uint32_t tmem, uint32_t a, uint32_t b, uint32_t idesc, uint32_t acc)
{
    constexpr uint32_t HI = (uint32_t)(1024 >> 4) | (1u << 14) | (2u << 29);      // as in umma_desc
    const uint32_t la = (a >> 4) | (1u << 16), lb = (b >> 4) | (1u << 16);
#pragma unroll
    for (int kk = 0; kk < GK / 16; ++kk)
        asm volatile(
            "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
            "mov.b64 da, {%1, %5};\n\tmov.b64 db, {%2, %5};\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}\n"
            ::"r"(tmem), "r"(la + 2 * kk), "r"(lb + 2 * kk), "r"(idesc), "r"(kk ? 1u : acc), "n"(HI));
}
__device__ __forceinline__ void mma_commit(uint32_t mbar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}
// Stage and phase parity of a ring of S stages.
template <int S>
struct RingPos {
    int s = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void next()
    {
        if (++s == S) {
            s = 0;
            phase ^= 1u;
        }
    }
};

enum GemmEpi { EPI_F32 = 0, EPI_F32_ADD = 1, EPI_BF16_BIAS = 2, EPI_BF16_BIAS_RELU = 3, EPI_F32_BIAS = 4 };

template <int BN, int EPI>
__global__ void __launch_bounds__(128, 1) k_gemm_bf16(const __nv_bfloat16* __restrict__ A, int lda,
                                                      const __nv_bfloat16* __restrict__ B, int ldb, int M, int N,
                                                      int K, void* __restrict__ D, int ldd,
                                                      const float* __restrict__ bias, int* __restrict__ err)
{
    static_assert(BN == 32 || BN == 64 || BN == 128 || BN == 256, "TMEM allocation is a power of two >= 32");
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* tA = sm;                       // 128 x 128 B
    uint8_t* tB = sm + GM * 128;            // BN x 128 B
    __shared__ __align__(8) uint64_t mbar;
    __shared__ uint32_t tmem_slot;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * GM, n0 = blockIdx.y * BN;
    const uint32_t mb = smem_u32(&mbar);
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mb) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");   // visible to the commit's arrive
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    const uint32_t idesc = idesc_bf16(BN);
    const int nk = (K + GK - 1) / GK;
    uint32_t parity = 0;
    bool failed = false;
    for (int kt = 0; kt < nk; ++kt) {
        const int k0 = kt * GK;
        for (int c = tid; c < GM * 8; c += blockDim.x) {
            const int r = c >> 3, j = c & 7, m = m0 + r, k = k0 + 8 * j;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (m < M && k < K) v = *reinterpret_cast<const uint4*>(A + (size_t)m * lda + k);
            *reinterpret_cast<uint4*>(tA + sw128(r, j)) = v;
        }
        for (int c = tid; c < BN * 8; c += blockDim.x) {
            const int r = c >> 3, j = c & 7, n = n0 + r, k = k0 + 8 * j;
            uint4 v = make_uint4(0, 0, 0, 0);
            if (n < N && k < K) v = *reinterpret_cast<const uint4*>(B + (size_t)n * ldb + k);
            *reinterpret_cast<uint4*>(tB + sw128(r, j)) = v;
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // shared writes -> tensor core reads
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int kk = 0; kk < GK / 16; ++kk)
                mma_bf16(tmem, umma_desc(smem_u32(tA) + 32 * kk), umma_desc(smem_u32(tB) + 32 * kk), idesc,
                         (kt | kk) != 0);
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mb)
                         : "memory");
        }
        const bool ok = mbar_wait(mb, parity);                // the tiles are reused next K step
        parity ^= 1u;
        if (__syncthreads_or(!ok)) { failed = true; break; }
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (failed) {
        if (tid == 0) atomicExch(err, 1);
    } else if (nk > 0) {
        const int m = m0 + warp * 32 + lane;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 16) {
            uint32_t r[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                "%14, %15}, [%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                  "=r"(r[15])
                : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (m < M) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int n = n0 + c0 + j;
                    if (n >= N) continue;
                    const float v = __uint_as_float(r[j]);
                    if constexpr (EPI == EPI_F32) {
                        static_cast<float*>(D)[(size_t)m * ldd + n] = v;
                    } else if constexpr (EPI == EPI_F32_ADD) {
                        static_cast<float*>(D)[(size_t)m * ldd + n] += v;
                    } else if constexpr (EPI == EPI_F32_BIAS) {
                        static_cast<float*>(D)[(size_t)m * ldd + n] = v + (bias ? bias[n] : 0.f);
                    } else {
                        float o = v + (bias ? bias[n] : 0.f);
                        if constexpr (EPI == EPI_BF16_BIAS_RELU) o = fmaxf(o, 0.f);
                        static_cast<__nv_bfloat16*>(D)[(size_t)m * ldd + n] = __float2bfloat16_rn(o);
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN) : "memory");
}

// ---------------------------------------------------------------------------------------------
// Pipelined GEMM: the same product and epilogues as k_gemm_bf16, with the operand tiles brought
// in by the Tensor Memory Accelerator.  A ring of S stages (A tile 128 x 64 and B tile BN x 64,
// bf16, 128-byte swizzled -- the layout the UMMA descriptors describe) is filled by one thread
// issuing cp.async.bulk.tensor loads (no multicast) that complete on the stage's `full` mbarrier;
// one thread of another warp waits on `full`, issues the four tcgen05.mma of the stage and
// commits them to the stage's `empty` mbarrier, which the loading thread waits on before it
// refills the stage; the last commit goes to `done`, on which the four warps wait before the
// epilogue reads TMEM.  Every wait is bounded: a thread that runs out sets `err`, the others'
// waits run out in turn, the loading thread waits (bounded) for the copies it issued, and the
// block frees its TMEM and returns.  Tile rows and columns past M, N and K come in as zeros
// (the tensor map's out-of-bounds fill).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t mbar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t mbar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(mbar)
        : "memory");
}

template <int BN, int EPI, int S>
__global__ void __launch_bounds__(128, 1) k_gemm_tma(const __grid_constant__ CUtensorMap tmA,
                                                     const __grid_constant__ CUtensorMap tmB, int M, int N, int K,
                                                     void* __restrict__ D, int ldd, const float* __restrict__ bias,
                                                     int* __restrict__ err)
{
    static_assert(BN == 32 || BN == 64 || BN == 128 || BN == 256, "TMEM allocation is a power of two >= 32");
    constexpr uint32_t A_BYTES = GM * 128, B_BYTES = BN * 128, STAGE = A_BYTES + B_BYTES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full[S], empty[S], done;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * GM, n0 = blockIdx.y * BN;
    const int nk = (K + GK - 1) / GK;
    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        mbar_init(smem_u32(&done), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        failed = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    if (warp == 0) {
        // loader: stage s = kt % S takes K tile kt once the MMAs of K tile kt - S have read it
        int issued = 0;
        RingPos<S> r;
        for (int kt = 0; kt < nk; ++kt, ++issued, r.next()) {
            if (kt >= S && !warp_wait(smem_u32(&empty[r.s]), r.phase ^ 1u, &failed)) {
                atomicExch(err, 1);
                failed = 1;
                break;
            }
            if (elect_one()) {
                const uint32_t a = smem_u32(sm) + r.s * STAGE, fb = smem_u32(&full[r.s]);
                mbar_expect_tx(fb, STAGE);
                tma_load_2d(a, &tmA, kt * GK, m0, fb);
                tma_load_2d(a + A_BYTES, &tmB, kt * GK, n0, fb);
            }
            __syncwarp();
        }
        // the copies of the last min(S, issued) K tiles must have landed before the block can
        // leave (on success the MMA warp has waited for all of them already)
        for (int kt = (issued > S ? issued - S : 0); kt < issued; ++kt)
            mbar_wait(smem_u32(&full[kt % S]), (uint32_t)((kt / S) & 1));
    } else if (warp == 1) {
        const uint32_t idesc = idesc_bf16(BN);
        RingPos<S> r;
        for (int kt = 0; kt < nk; ++kt, r.next()) {
            if (!warp_wait(smem_u32(&full[r.s]), r.phase, &failed)) {
                atomicExch(err, 1);
                failed = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
                const uint32_t a = smem_u32(sm) + r.s * STAGE;
                mma_ktile(tmem, a, a + A_BYTES, idesc, kt != 0);
                mma_commit(smem_u32(&empty[r.s]));
                if (kt == nk - 1) mma_commit(smem_u32(&done));
            }
            __syncwarp();
        }
    }
    __syncwarp();
    const bool ok = nk > 0 && mbar_wait(smem_u32(&done), 0u);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (__syncthreads_or(!ok || failed)) {
        if (tid == 0 && nk > 0) atomicExch(err, 1);
    } else {
        const int m = m0 + warp * 32 + lane;
#pragma unroll 1
        for (int c0 = 0; c0 < BN; c0 += 16) {
            uint32_t r[16];
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                "%14, %15}, [%16];"
                : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                  "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                  "=r"(r[15])
                : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0));
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
            if (m < M) {
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int n = n0 + c0 + j;
                    if (n >= N) continue;
                    const float v = __uint_as_float(r[j]);
                    if constexpr (EPI == EPI_F32) {
                        static_cast<float*>(D)[(size_t)m * ldd + n] = v;
                    } else if constexpr (EPI == EPI_F32_ADD) {
                        static_cast<float*>(D)[(size_t)m * ldd + n] += v;
                    } else if constexpr (EPI == EPI_F32_BIAS) {
                        static_cast<float*>(D)[(size_t)m * ldd + n] = v + (bias ? bias[n] : 0.f);
                    } else {
                        float o = v + (bias ? bias[n] : 0.f);
                        if constexpr (EPI == EPI_BF16_BIAS_RELU) o = fmaxf(o, 0.f);
                        static_cast<__nv_bfloat16*>(D)[(size_t)m * ldd + n] = __float2bfloat16_rn(o);
                    }
                }
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN) : "memory");
}

template <int BN, int EPI>
int launch_gemm(const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb, int M, int N, int K, void* D, int ldd,
                const float* bias, int* err, cudaStream_t st)
{
    auto kern = k_gemm_bf16<BN, EPI>;
    const int smem = GM * 128 + BN * 128 + 1024;
    if (const cudaError_t e = allow_shared(kern, smem))
        return fail(LBM_ERR_CUDA, "k_gemm_bf16: %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
    dim3 grid((unsigned)((M + GM - 1) / GM), (unsigned)((N + BN - 1) / BN));
    kern<<<grid, 128, smem, st>>>(A, lda, B, ldb, M, N, K, D, ldd, bias, err);
    return check_launch("k_gemm_bf16");
}

// Tensor map of a rows x K bf16 matrix with row stride ld (elements), boxes of 64 (K) x box_rows,
// 128-byte swizzle, zero fill out of bounds.
bool bf16_tile_map(CUtensorMap* map, const __nv_bfloat16* base, int rows, int K, int ld, int box_rows)
{
    PfnEncodeTiled enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)GK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

constexpr int kGemmStages = 3, kGemmDeepStages = 8;

// The pipelined kernel when the tensor maps can be made; false: the caller runs k_gemm_bf16.
template <int BN, int EPI, int S = kGemmStages>
bool launch_gemm_tma(const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb, int M, int N, int K, void* D,
                     int ldd, const float* bias, int* err, cudaStream_t st, int* status)
{
    CUtensorMap ta, tb;
    if (!bf16_tile_map(&ta, A, M, K, lda, GM) || !bf16_tile_map(&tb, B, N, K, ldb, BN)) return false;
    auto kern = k_gemm_tma<BN, EPI, S>;
    const int smem = S * (GM * 128 + BN * 128) + 1024;
    if (allow_shared(kern, smem) != cudaSuccess) return false;
    dim3 grid((unsigned)((M + GM - 1) / GM), (unsigned)((N + BN - 1) / BN));
    kern<<<grid, 128, smem, st>>>(ta, tb, M, N, K, D, ldd, bias, err);
    *status = check_launch("k_gemm_tma");
    return true;
}

template <int EPI>
int launch_gemm_bn(int bn, const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb, int M, int N, int K,
                   void* D, int ldd, const float* bias, int* err, cudaStream_t st)
{
    int status = LBM_OK;
    switch (bn) {
    case 32:
        if (launch_gemm_tma<32, EPI>(A, lda, B, ldb, M, N, K, D, ldd, bias, err, st, &status)) return status;
        return launch_gemm<32, EPI>(A, lda, B, ldb, M, N, K, D, ldd, bias, err, st);
    case 64:
        if (launch_gemm_tma<64, EPI>(A, lda, B, ldb, M, N, K, D, ldd, bias, err, st, &status)) return status;
        return launch_gemm<64, EPI>(A, lda, B, ldb, M, N, K, D, ldd, bias, err, st);
    case 128:
        if (launch_gemm_tma<128, EPI>(A, lda, B, ldb, M, N, K, D, ldd, bias, err, st, &status)) return status;
        return launch_gemm<128, EPI>(A, lda, B, ldb, M, N, K, D, ldd, bias, err, st);
    default:
        if (launch_gemm_tma<256, EPI>(A, lda, B, ldb, M, N, K, D, ldd, bias, err, st, &status)) return status;
        return launch_gemm<256, EPI>(A, lda, B, ldb, M, N, K, D, ldd, bias, err, st);
    }
}

// ---------------------------------------------------------------------------------------------
// Persistent warp-specialised GEMM for products with many rows and N >= 128 (a caller's; the network's own
// have at most 128 rows, and its convolutions read the grids in place).  The accumulator is held transposed: tcgen05.mma with M = 128 takes a
// 128-row block of B (output channels n0..n0+127) as its A operand and a BV-row block of A
// (voxels m0..m0+BV-1, BV = 128..256) as its B operand, so TMEM lane l holds channel n0 + l and
// column j voxel m0 + j.  The epilogue thread of lane l then writes 32 voxels of one channel,
// and a warp's store covers 32 consecutive channels of one output row (64 or 128 contiguous
// bytes) instead of one element of 32 rows.  Each operand block is read from L2 once per tile
// of 128 x BV outputs, and BV is chosen so the tiles fill the SMs in as few waves as possible
// (32768 rows: BV = 224, 147 tiles on 148 SMs).
//
// One CTA of 6 warps per SM walks the tiles t = blockIdx.x, + gridDim.x, ...:
//   warp 0, one thread: TMA loads of both blocks into a ring of S stages (no multicast),
//     completing on full[s], refilling a stage once empty[s] says its MMAs are done;
//   warp 1, one thread: per stage four tcgen05.mma (K = 16) into accumulator buffer
//     tc & 1 (two buffers of 256 TMEM columns), commit to empty[s]; per tile commit to
//     acc_full[b] after waiting for acc_empty[b] (the epilogue has read the buffer);
//   warps 2-5: wait acc_full[b], tcgen05.ld 32 columns at a time from their lane quarter
//     (warp & 3), release the buffer to the MMA thread, apply the epilogue and store.
// The epilogue of one tile thus runs while the next tile's loads and MMAs proceed.  Every
// wait is bounded; a role that runs out sets `failed` and `err`, the others leave their loops,
// the MMA thread waits (bounded) for its issued MMAs, the loading thread for its copies, and
// the block frees TMEM and returns.
// ---------------------------------------------------------------------------------------------
constexpr int kWsThreads = 192;
constexpr int kWsMaxStages = 8, kWsShared = 225 * 1024;     // shared memory of a CTA at most
constexpr uint32_t kWsChBytes = GM * 128;   // channel block: 128 rows x 64 bf16

template <int EPI>
__global__ void __launch_bounds__(kWsThreads, 1) k_gemm_ws(const __grid_constant__ CUtensorMap tmA,
                                                           const __grid_constant__ CUtensorMap tmB, int M, int N,
                                                           int K, int BV, int S, void* __restrict__ D, int ldd,
                                                           const float* __restrict__ bias, int* __restrict__ err)
{
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full[kWsMaxStages], empty[kWsMaxStages], acc_full[2], acc_empty[2], drain;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t stage_bytes = kWsChBytes + (uint32_t)BV * 128u;
    const int nk = (K + GK - 1) / GK;
    const int tiles_m = (M + BV - 1) / BV, tiles = tiles_m * ((N + GM - 1) / GM);
    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full[b]), 1);
            mbar_init(smem_u32(&acc_empty[b]), 4);
        }
        mbar_init(smem_u32(&drain), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        failed = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    volatile int* vfailed = &failed;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t it = 0;
            for (int t = blockIdx.x; t < tiles && !*vfailed; t += gridDim.x) {
                const int m0 = (t % tiles_m) * BV, n0 = (t / tiles_m) * GM;
                for (int kt = 0; kt < nk; ++kt, ++it) {
                    const uint32_t s = it % (uint32_t)S, r = it / (uint32_t)S;
                    if (it >= (uint32_t)S && !mbar_wait(smem_u32(&empty[s]), (r - 1) & 1u)) {
                        atomicExch(err, 1);
                        *vfailed = 1;
                    }
                    if (*vfailed) break;
                    const uint32_t base = smem_u32(sm + (size_t)s * stage_bytes), fb = smem_u32(&full[s]);
                    mbar_expect_tx(fb, stage_bytes);
                    tma_load_2d(base, &tmB, kt * GK, n0, fb);
                    tma_load_2d(base + kWsChBytes, &tmA, kt * GK, m0, fb);
                }
            }
            // copies of the last min(S, it) stages filled must have landed before the block leaves
            for (uint32_t j = (it > (uint32_t)S ? it - (uint32_t)S : 0u); j < it; ++j)
                mbar_wait(smem_u32(&full[j % (uint32_t)S]), (j / (uint32_t)S) & 1u);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = idesc_bf16(BV);
            uint32_t it = 0, tc = 0;
            for (int t = blockIdx.x; t < tiles && !*vfailed; t += gridDim.x, ++tc) {
                const uint32_t b = tc & 1u, u = tc >> 1;
                if (tc >= 2 && !mbar_wait(smem_u32(&acc_empty[b]), (u - 1) & 1u)) {
                    atomicExch(err, 1);
                    *vfailed = 1;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + b * 256u;
                bool ok = true;
                for (int kt = 0; kt < nk; ++kt, ++it) {
                    const uint32_t s = it % (uint32_t)S, r = it / (uint32_t)S;
                    if (!mbar_wait(smem_u32(&full[s]), r & 1u) || *vfailed) {
                        atomicExch(err, 1);
                        *vfailed = 1;
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t base = smem_u32(sm + (size_t)s * stage_bytes);
#pragma unroll
                    for (int kk = 0; kk < GK / 16; ++kk)
                        mma_bf16(d, umma_desc(base + 32 * kk), umma_desc(base + kWsChBytes + 32 * kk), idesc,
                                 (kt | kk) != 0);
                    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                                 ::"r"(smem_u32(&empty[s]))
                                 : "memory");
                }
                if (!ok) break;
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                             ::"r"(smem_u32(&acc_full[b]))
                             : "memory");
            }
            // every MMA this thread issued has completed once `drain` does
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                         ::"r"(smem_u32(&drain))
                         : "memory");
            mbar_wait(smem_u32(&drain), 0u);
        }
    } else {
        const int q = warp & 3;                      // TMEM lanes 32q..32q+31 = channels
        uint32_t tc = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++tc) {
            const uint32_t b = tc & 1u, u = tc >> 1;
            const bool ready = mbar_wait(smem_u32(&acc_full[b]), u & 1u);
            if (__any_sync(0xffffffffu, !ready || *vfailed)) {
                if (lane == 0) {
                    atomicExch(err, 1);
                    *vfailed = 1;
                }
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const int m0 = (t % tiles_m) * BV, n = (t / tiles_m) * GM + q * 32 + lane;
            const int mend = M < m0 + BV ? M : m0 + BV;   // rows of this block (BV: a multiple of 16)
            const float bn = (EPI >= EPI_BF16_BIAS && bias && n < N) ? bias[n] : 0.f;
            for (int j0 = 0; j0 < BV; j0 += 32) {
                uint32_t r[32];
                asm volatile(
                    "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
                    "%13, %14, %15, %16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, "
                    "[%32];"
                    : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
                      "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
                      "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
                      "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]),
                      "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                    : "r"(tmem + b * 256u + ((uint32_t)(q * 32) << 16) + (uint32_t)j0));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (j0 + 32 >= BV) {
                    // the whole buffer is in registers: hand it back to the MMA thread
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0)
                        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[b]))
                                     : "memory");
                }
                if (n < N) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        const int m = m0 + j0 + j;
                        if (m >= mend) break;
                        const float v = __uint_as_float(r[j]);
                        const size_t o = (size_t)m * ldd + n;
                        if constexpr (EPI == EPI_F32) {
                            static_cast<float*>(D)[o] = v;
                        } else if constexpr (EPI == EPI_F32_ADD) {
                            static_cast<float*>(D)[o] += v;
                        } else if constexpr (EPI == EPI_F32_BIAS) {
                            static_cast<float*>(D)[o] = v + bn;
                        } else {
                            float x = v + bn;
                            if constexpr (EPI == EPI_BF16_BIAS_RELU) x = fmaxf(x, 0.f);
                            static_cast<__nv_bfloat16*>(D)[o] = __float2bfloat16_rn(x);
                        }
                    }
                }
            }
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

int sm_count()
{
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 148;
    return n;
}

// Row-block width of k_gemm_ws: the fewest waves of tiles over the SMs times the width (the
// rows one SM streams), ties to the wider block (fewer reads of B).
int ws_block_rows(int M, int N, int nsm)
{
    const int tiles_n = (N + GM - 1) / GM;
    int best = 256;
    long long best_cost = -1;
    for (int bv = 256; bv >= 128; bv -= 32) {
        const long long tiles = (long long)((M + bv - 1) / bv) * tiles_n;
        const long long cost = (tiles + nsm - 1) / nsm * bv;
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = bv;
        }
    }
    return best;
}

// k_gemm_ws for M >= 1024 rows and N >= 128 channels when the tensor maps can be made;
// false: the caller runs the one-tile-per-CTA kernels.
template <int EPI>
bool launch_gemm_ws(const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb, int M, int N, int K, void* D,
                    int ldd, const float* bias, int* err, cudaStream_t st, int* status)
{
    if (M < 1024 || N < GM) return false;
    const int nsm = sm_count();
    const int bv = ws_block_rows(M, N, nsm);
    const int stage = (int)kWsChBytes + bv * 128;
    // as many stages as 225 KB of shared memory hold (row block 224: 5, which measured 1 % above 4)
    const int stages = (kWsShared - 1024) / stage < kWsMaxStages ? (kWsShared - 1024) / stage : kWsMaxStages;
    const int smem = stages * stage + 1024;         // > half the SM's shared memory: one CTA per SM
    CUtensorMap ta, tb;
    if (!bf16_tile_map(&ta, A, M, K, lda, bv) || !bf16_tile_map(&tb, B, N, K, ldb, GM)) return false;
    auto kern = k_gemm_ws<EPI>;
    if (allow_shared(kern, kWsShared) != cudaSuccess) return false;
    const long long tiles = (long long)((M + bv - 1) / bv) * ((N + GM - 1) / GM);
    const int grid = (int)(tiles < nsm ? tiles : nsm);
    kern<<<grid, kWsThreads, smem, st>>>(ta, tb, M, N, K, bv, stages, D, ldd, bias, err);
    *status = check_launch("k_gemm_ws");
    return true;
}

template <int EPI>
int launch_gemm_any(int bn, const __nv_bfloat16* A, int lda, const __nv_bfloat16* B, int ldb, int M, int N, int K,
                    void* D, int ldd, const float* bias, int* err, cudaStream_t st)
{
    int status = LBM_OK;
    // D += products with a long K and few tiles (the weight gradients: K is the voxels): narrow tiles,
    // for as many CTAs as there are, and a ring deep enough that the one chain of MMAs never waits
    // for a load.  64 x 1728 weights over 12,288 voxels: 54 CTAs instead of 7, 64 us (the six layers of a
    // training step 88 -> 43 us on average).  Splitting K would be faster still, but moves the sums by more
    // than 2e-5.
    if constexpr (EPI == EPI_F32_ADD) {
        const long long wide = (long long)((M + GM - 1) / GM) * ((N + bn - 1) / bn);
        if (wide * 2 <= sm_count() && K >= 4 * GK &&
            launch_gemm_tma<32, EPI, kGemmDeepStages>(A, lda, B, ldb, M, N, K, D, ldd, bias, err, st, &status))
            return status;
    }
    if (launch_gemm_ws<EPI>(A, lda, B, ldb, M, N, K, D, ldd, bias, err, st, &status)) return status;
    return launch_gemm_bn<EPI>(bn, A, lda, B, ldb, M, N, K, D, ldd, bias, err, st);
}

// ---------------------------------------------------------------------------------------------
// Convolutions without a column matrix.  A 3x3x3 convolution of a channels-last grid is the same
// GEMM with A's rows read in place: the 128 rows of a tile are the voxels of a box of the grid, and
// the K tile of tap t and channels c0.. is that box shifted by the tap, one tiled TMA load whose
// coordinates outside the grid read zero.  K runs over taps, then channels, as the columns of
// k_im2col do, so the accumulation and the results are those of the GEMM on the column matrix.
// What bounds it: the 27 shifted reads of the grid now come from L2 instead of the column matrix's
// write and read in HBM (415 MB each way for 64 channels on 120k voxels).  A prediction on 120k
// voxels (10 x 80 x 150) took 389 us instead of 1069, a gradient on 12k voxels 816 instead of 1099; with the
// input layer, pooling and issue below 216 and 800 (whose loss adds 56 us of atomics).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, int c3,
                                            uint32_t mbar)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(mbar)
        : "memory");
}

// Boxes of 128 voxels over an X x Y x Z grid: box sides (powers of two) and the boxes along each axis.
struct ConvTiles {
    int X, Y, Z, bx, by, bz, nx, ny, nz;
};
// Voxel coordinates of the first voxel of box `tile`.
__device__ __forceinline__ void tile_origin(const ConvTiles& g, int tile, int& x, int& y, int& z)
{
    x = tile % g.nx * g.bx;
    y = tile / g.nx % g.ny * g.by;
    z = tile / (g.nx * g.ny) * g.bz;
}
// Voxel of row r of the box at (x, y, z), or -1 outside the grid.
__device__ __forceinline__ long long tile_voxel(const ConvTiles& g, int x, int y, int z, int r)
{
    x += r % g.bx;
    y += r / g.bx % g.by;
    z += r / (g.bx * g.by);
    return x < g.X && y < g.Y && z < g.Z ? x + (long long)g.X * (y + (long long)g.Y * z) : -1;
}

__device__ __forceinline__ void tmem_ld16(uint32_t (&r)[16], uint32_t addr)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
        "%14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Epilogue of the forward convolutions: columns n0 .. of voxel v (-1: none) from the thread's TMEM lane.
template <int EPI>
__device__ __forceinline__ void conv_store(uint32_t lane_addr, long long v, int N, int n0, int BN, void* __restrict__ D,
                                           const float* __restrict__ bias)
{
    const int cols = N - n0 < BN ? N - n0 : BN;            // a multiple of 8
#pragma unroll 1
    for (int c0 = 0; c0 < cols; c0 += 16) {
        uint32_t r[16];
        tmem_ld16(r, lane_addr + (uint32_t)c0);
#pragma unroll
        for (int q = 0; q < 16; q += 8) {
            if (v < 0 || c0 + q >= cols) continue;
            float o[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                o[j] = __uint_as_float(r[q + j]) + bias[n0 + c0 + q + j];
                if constexpr (EPI == EPI_BF16_BIAS_RELU) o[j] = fmaxf(o[j], 0.f);
            }
            const size_t at = (size_t)v * N + n0 + c0 + q;
            if constexpr (EPI == EPI_F32_BIAS) store_n<8>(static_cast<float*>(D) + at, o);
            else store_n<8>(static_cast<__nv_bfloat16*>(D) + at, o);
        }
    }
}

// Forward: D[v][n] = epilogue(sum_t sum_c x[v + off_t][c] W[n][t*C + c] + bias[n]), C a multiple of
// 64.  One box x BN channels per CTA (two CTAs per SM, so one's epilogue runs beside the other's
// loads), one loading warp, one MMA warp, a ring of S stages; waits bounded as in k_gemm_tma.
template <int BN, int EPI, int S>
__global__ void __launch_bounds__(128, 2) k_conv_fwd(const __grid_constant__ CUtensorMap tmX,
                                                     const __grid_constant__ CUtensorMap tmW, const ConvTiles g, int C,
                                                     int N, void* __restrict__ D, const float* __restrict__ bias,
                                                     int* __restrict__ err)
{
    static_assert(BN == 32 || BN == 64 || BN == 128, "TMEM allocation is a power of two >= 32");
    constexpr uint32_t A_BYTES = GM * 128, B_BYTES = BN * 128, STAGE = A_BYTES + B_BYTES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full[S], empty[S], done;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.y * BN, per_tap = C / GK, nk = 27 * per_tap;
    int x0, y0, z0;
    tile_origin(g, blockIdx.x, x0, y0, z0);
    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        mbar_init(smem_u32(&done), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        failed = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    if (warp == 0) {
        int issued = 0, t = 0, q = 0;                      // tap and channel block of K tile `issued`
        RingPos<S> r;
        for (; issued < nk; ++issued, r.next()) {
            if (issued >= S && !warp_wait(smem_u32(&empty[r.s]), r.phase ^ 1u, &failed)) {
                atomicExch(err, 1);
                failed = 1;
                break;
            }
            if (elect_one()) {
                const uint32_t a = smem_u32(sm) + r.s * STAGE, fb = smem_u32(&full[r.s]);
                mbar_expect_tx(fb, STAGE);
                tma_load_4d(a, &tmX, q * GK, x0 + t % 3 - 1, y0 + t / 3 % 3 - 1, z0 + t / 9 - 1, fb);
                tma_load_2d(a + A_BYTES, &tmW, issued * GK, n0, fb);
            }
            __syncwarp();
            if (++q == per_tap) {
                q = 0;
                ++t;
            }
        }
        // the last copies must have landed before the block can leave
        for (int kt = (issued > S ? issued - S : 0); kt < issued; ++kt)
            mbar_wait(smem_u32(&full[kt % S]), (uint32_t)((kt / S) & 1));
    } else if (warp == 1) {
        const uint32_t idesc = idesc_bf16(BN);
        RingPos<S> r;
        for (int kt = 0; kt < nk; ++kt, r.next()) {
            if (!warp_wait(smem_u32(&full[r.s]), r.phase, &failed)) {
                atomicExch(err, 1);
                failed = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
                const uint32_t a = smem_u32(sm) + r.s * STAGE;
                mma_ktile(tmem, a, a + A_BYTES, idesc, kt != 0);
                mma_commit(smem_u32(&empty[r.s]));
            }
            __syncwarp();
        }
        // `done` completes once every MMA issued has, a failed run's too
        if (elect_one()) mma_commit(smem_u32(&done));
    }
    __syncwarp();
    const bool ok = mbar_wait(smem_u32(&done), 0u);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (__syncthreads_or(!ok || failed)) {
        if (tid == 0) atomicExch(err, 1);
    } else {
        conv_store<EPI>(tmem + ((uint32_t)(warp * 32) << 16), tile_voxel(g, x0, y0, z0, warp * 32 + lane), N, n0, BN, D, bias);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN) : "memory");
}

// Forward of the input layer (8 channels, 16 bytes a voxel): eight taps make a K tile, so the 27 taps of
// 128 consecutive voxels are gathered straight into swizzled shared memory, a voxel per thread with all
// its loads in flight, and one chain of 14 MMAs follows (K order and values as on the column matrix).
// One shot per CTA; two CTAs per SM, so one's gather runs beside the other's epilogue.
// 120k voxels, 8 -> 64 channels: 28 us, against 28 for the column matrix and 98 for its product.
constexpr int kInTiles = 4, kInTaps = 28;       // K tiles of 8 taps; taps with a product (27, and one of zeros)

template <int BN, int EPI>
__global__ void __launch_bounds__(128, 2) k_conv_in(const __nv_bfloat16* __restrict__ Xin,
                                                    const __grid_constant__ CUtensorMap tmW, int X, int Y, int Z,
                                                    int N, void* __restrict__ D, const float* __restrict__ bias,
                                                    int* __restrict__ err)
{
    static_assert(BN == 32 || BN == 64, "TMEM allocation is a power of two >= 32");
    constexpr uint32_t A_BYTES = GM * 128, B_BYTES = BN * 128;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t loaded, done;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    const int tid = threadIdx.x, warp = tid >> 5;
    const int n0 = blockIdx.y * BN;
    const uint32_t V = (uint32_t)X * Y * Z, v = blockIdx.x * GM + tid;
    const uint32_t ld = smem_u32(&loaded), dn = smem_u32(&done), base = smem_u32(sm);
    if (tid == 0) {
        mbar_init(ld, 1);
        mbar_init(dn, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        failed = 0;
        mbar_expect_tx(ld, kInTiles * B_BYTES);
        for (int t = 0; t < kInTiles; ++t)
            tma_load_2d(base + kInTiles * A_BYTES + t * B_BYTES, &tmW, t * GK, n0, ld);
    }
    if (warp == 0) {
        __syncwarp();
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    const int x = (int)(v % (uint32_t)X), y = (int)(v / (uint32_t)X % (uint32_t)Y), z = (int)(v / ((uint32_t)X * Y));
    uint4 a[kInTaps];
#pragma unroll
    for (int t = 0; t < kInTaps; ++t) {
        const int xs = x + t % 3 - 1, ys = y + t / 3 % 3 - 1, zs = z + t / 9 - 1;
        a[t] = make_uint4(0, 0, 0, 0);
        if (t < 27 && v < V && xs >= 0 && xs < X && ys >= 0 && ys < Y && zs >= 0 && zs < Z)
            a[t] = __ldg(reinterpret_cast<const uint4*>(Xin) + xs + (long long)X * (ys + (long long)Y * zs));
    }
#pragma unroll
    for (int t = 0; t < kInTaps; ++t)
        *reinterpret_cast<uint4*>(sm + (t / 8) * A_BYTES + sw128(tid, t % 8)) = a[t];
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");       // shared writes -> tensor core reads
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    if (tid == 0) {
        if (mbar_wait(ld, 0u)) {
            const uint32_t idesc = idesc_bf16(BN);
#pragma unroll
            for (int k = 0; k < kInTaps / 2; ++k)
                mma_bf16(tmem, umma_desc(base + k / 4 * A_BYTES + 32 * (k % 4)),
                         umma_desc(base + kInTiles * A_BYTES + k / 4 * B_BYTES + 32 * (k % 4)), idesc, k != 0);
        } else {
            failed = 1;
            mbar_wait(ld, 0u);                             // the copies must have landed before the block leaves
        }
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(dn) : "memory");
    }
    __syncwarp();
    const bool ok = mbar_wait(dn, 0u);
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (__syncthreads_or(!ok || failed)) {
        if (tid == 0) atomicExch(err, 1);
    } else {
        conv_store<EPI>(tmem + ((uint32_t)(warp * 32) << 16), v < V ? (long long)v : -1, N, n0, BN, D, bias);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN) : "memory");
}

// Backward to the input: dX[v][c] = sum_t (sum_o g[v - off_t][o] Wt[t*C + c][o]), Wt the transposed
// weights (27*C x O).  The column-matrix form made dcol (float32, 27 C values per voxel) and gathered
// it; here a tap's product stays in one of two TMEM buffers, and the epilogue warps add it, in the
// order of the taps and in float32 as the gather did, to sums they keep in registers while the next
// tap's product is made.  Voxels outside the grid read zero and add nothing.
// Roles as in k_gemm_ws: warp 0 loads, warp 1 issues the MMAs, warps 2-5 add and store.
constexpr int kBackN = 64, kBackStages = 6;

__global__ void __launch_bounds__(kWsThreads, 1) k_conv_back(const __grid_constant__ CUtensorMap tmG,
                                                             const __grid_constant__ CUtensorMap tmW, const ConvTiles g,
                                                             int O, int C, float* __restrict__ dX, int* __restrict__ err)
{
    constexpr int S = kBackStages, BN = kBackN;
    constexpr uint32_t A_BYTES = GM * 128, B_BYTES = BN * 128, STAGE = A_BYTES + B_BYTES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    __shared__ __align__(8) uint64_t full[S], empty[S], acc_full[2], acc_empty[2], drain;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.y * BN, per_tap = (O + GK - 1) / GK;
    int x0, y0, z0;
    tile_origin(g, blockIdx.x, x0, y0, z0);
    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(smem_u32(&full[s]), 1);
            mbar_init(smem_u32(&empty[s]), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(smem_u32(&acc_full[b]), 1);
            mbar_init(smem_u32(&acc_empty[b]), 4);
        }
        mbar_init(smem_u32(&drain), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        failed = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(2 * BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;
    volatile int* vfailed = &failed;
    if (warp == 0) {
        int it = 0;
        bool ok = true;
        RingPos<S> r;
        for (int t = 0; t < 27 && ok; ++t) {
            const int u = 26 - t;                          // v - off_t is v's neighbour through tap 26 - t
            for (int q = 0; q < per_tap; ++q, ++it, r.next()) {
                if (it >= S && !warp_wait(smem_u32(&empty[r.s]), r.phase ^ 1u, &failed)) {
                    atomicExch(err, 1);
                    *vfailed = 1;
                    ok = false;
                    break;
                }
                if (elect_one()) {
                    const uint32_t a = smem_u32(sm) + r.s * STAGE, fb = smem_u32(&full[r.s]);
                    mbar_expect_tx(fb, STAGE);
                    tma_load_4d(a, &tmG, q * GK, x0 + u % 3 - 1, y0 + u / 3 % 3 - 1, z0 + u / 9 - 1, fb);
                    tma_load_2d(a + A_BYTES, &tmW, q * GK, t * C + n0, fb);
                }
                __syncwarp();
            }
        }
        for (int j = (it > S ? it - S : 0); j < it; ++j) mbar_wait(smem_u32(&full[j % S]), (uint32_t)((j / S) & 1));
    } else if (warp == 1) {
        const uint32_t idesc = idesc_bf16(BN);
        bool ok = true;
        RingPos<S> r;
        for (int t = 0; t < 27 && ok; ++t) {
            const int b = t & 1;
            if (t >= 2 && !warp_wait(smem_u32(&acc_empty[b]), (uint32_t)((t / 2 - 1) & 1), &failed)) {
                atomicExch(err, 1);
                *vfailed = 1;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int q = 0; q < per_tap; ++q, r.next()) {
                if (!warp_wait(smem_u32(&full[r.s]), r.phase, &failed)) {
                    atomicExch(err, 1);
                    *vfailed = 1;
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one()) {
                    const uint32_t a = smem_u32(sm) + r.s * STAGE;
                    mma_ktile(tmem + b * BN, a, a + A_BYTES, idesc, q != 0);
                    mma_commit(smem_u32(&empty[r.s]));
                    if (q == per_tap - 1) mma_commit(smem_u32(&acc_full[b]));
                }
                __syncwarp();
            }
        }
        // every MMA this warp issued has completed once `drain` does
        if (elect_one()) mma_commit(smem_u32(&drain));
        __syncwarp();
        mbar_wait(smem_u32(&drain), 0u);
    } else {
        const int quarter = warp & 3;                      // TMEM lanes 32 quarter .. + 31: the box's rows
        float sum[BN];
#pragma unroll
        for (int j = 0; j < BN; ++j) sum[j] = 0.f;
        bool good = true;
        for (int t = 0; t < 27; ++t) {
            const int b = t & 1;
            const bool ready = mbar_wait(smem_u32(&acc_full[b]), (uint32_t)((t / 2) & 1));
            if (__any_sync(0xffffffffu, !ready || *vfailed)) {
                if (lane == 0) {
                    atomicExch(err, 1);
                    *vfailed = 1;
                }
                good = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int c0 = 0; c0 < BN; c0 += 16) {
                uint32_t r[16];
                tmem_ld16(r, tmem + b * BN + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0);
#pragma unroll
                for (int j = 0; j < 16; ++j) sum[c0 + j] += __uint_as_float(r[j]);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0)
                asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&acc_empty[b])) : "memory");
        }
        const long long v = tile_voxel(g, x0, y0, z0, quarter * 32 + lane);
        if (good && v >= 0) {
            float* d = dX + (size_t)v * C + n0;
#pragma unroll
            for (int j = 0; j < BN; j += 4)
                if (n0 + j < C) *reinterpret_cast<float4*>(d + j) = make_float4(sum[j], sum[j + 1], sum[j + 2], sum[j + 3]);
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN) : "memory");
}

// Tensor map of a channels-last grid (C channels, bf16), boxes of 64 channels x the tile's voxels,
// 128-byte swizzle, zero outside.
bool bf16_grid_map(CUtensorMap* map, const __nv_bfloat16* base, int C, const ConvTiles& g)
{
    PfnEncodeTiled enc = encode_tiled();
    if (!enc) return false;
    const cuuint64_t dims[4] = {(cuuint64_t)C, (cuuint64_t)g.X, (cuuint64_t)g.Y, (cuuint64_t)g.Z};
    const cuuint64_t row = (cuuint64_t)C * 2;
    const cuuint64_t strides[3] = {row, row * g.X, row * g.X * g.Y};
    const cuuint32_t box[4] = {(cuuint32_t)GK, (cuuint32_t)g.bx, (cuuint32_t)g.by, (cuuint32_t)g.bz};
    const cuuint32_t estr[4] = {1, 1, 1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<__nv_bfloat16*>(base), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The box of 128 voxels that covers the grid with the fewest boxes; of equals the longest in x.
ConvTiles conv_tiles(int X, int Y, int Z)
{
    ConvTiles best{};
    long long fewest = -1;
    for (int bx = 128; bx >= 1; bx /= 2)
        for (int by = 128 / bx; by >= 1; by /= 2) {
            const int bz = 128 / (bx * by);
            const ConvTiles g{X, Y, Z, bx, by, bz, (X + bx - 1) / bx, (Y + by - 1) / by, (Z + bz - 1) / bz};
            const long long n = (long long)g.nx * g.ny * g.nz;
            if (fewest < 0 || n < fewest) {
                fewest = n;
                best = g;
            }
        }
    return best;
}

template <int BN, int EPI>
int launch_conv_bn(const __nv_bfloat16* x, int C, const ConvTiles& g, const __nv_bfloat16* W, int N, void* D,
                   const float* bias, int* err, cudaStream_t st)
{
    constexpr int S = 4;
    CUtensorMap tx, tw;
    if (!bf16_grid_map(&tx, x, C, g) || !bf16_tile_map(&tw, W, N, 27 * C, 27 * C, BN))
        return fail(LBM_ERR_CUDA, "lbm_conv3_bf16: no tensor map for this grid");
    auto kern = k_conv_fwd<BN, EPI, S>;
    const int smem = S * (GM * 128 + BN * 128) + 1024;
    if (const cudaError_t e = allow_shared(kern, smem))
        return fail(LBM_ERR_CUDA, "lbm_conv3_bf16: %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
    kern<<<dim3((unsigned)(g.nx * g.ny * g.nz), (unsigned)((N + BN - 1) / BN)), 128, smem, st>>>(tx, tw, g, C, N, D, bias, err);
    return check_launch("k_conv_fwd");
}

template <int BN, int EPI>
int launch_conv_in(const __nv_bfloat16* x, int X, int Y, int Z, const __nv_bfloat16* W, int N, void* D, const float* bias,
                   int* err, cudaStream_t st)
{
    CUtensorMap tw;
    if (!bf16_tile_map(&tw, W, N, 27 * 8, 27 * 8, BN)) return fail(LBM_ERR_CUDA, "lbm_conv3_bf16: no tensor map for the weights");
    auto kern = k_conv_in<BN, EPI>;
    const int smem = kInTiles * (GM * 128 + BN * 128) + 1024;
    if (const cudaError_t e = allow_shared(kern, smem))
        return fail(LBM_ERR_CUDA, "lbm_conv3_bf16: %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
    const long long V = (long long)X * Y * Z;
    kern<<<dim3((unsigned)((V + GM - 1) / GM), (unsigned)((N + BN - 1) / BN)), 128, smem, st>>>(x, tw, X, Y, Z, N, D, bias, err);
    return check_launch("k_conv_in");
}

// Channels per CTA: all of up to 64 (a box is then read once), in blocks of 64 beyond; of 32 where
// the boxes alone would leave most SMs without one (small grids).
template <int EPI>
int launch_conv(const __nv_bfloat16* x, int C, const ConvTiles& g, const __nv_bfloat16* W, int N, void* D,
                const float* bias, int* err, cudaStream_t st)
{
    if (C == 8)
        return N <= 32 ? launch_conv_in<32, EPI>(x, g.X, g.Y, g.Z, W, N, D, bias, err, st)
                       : launch_conv_in<64, EPI>(x, g.X, g.Y, g.Z, W, N, D, bias, err, st);
    const long long boxes = (long long)g.nx * g.ny * g.nz;
    if (N <= 32 || boxes * ((N + 63) / 64) * 2 <= sm_count()) return launch_conv_bn<32, EPI>(x, C, g, W, N, D, bias, err, st);
    return launch_conv_bn<64, EPI>(x, C, g, W, N, D, bias, err, st);
}

// ---------------------------------------------------------------------------------------------
// Network support kernels (CUDA cores).  Activations are channels-last: X[v * C + c], v = voxel
// index x + X*(y + Y*z) of a (Z, Y, X) grid.  A 3x3x3 tap t = (dz+1)*9 + (dy+1)*3 + (dx+1).
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ bool tap_src(int t, int x, int y, int z, int X, int Y, int Z, long long& v)
{
    const int xs = x + t % 3 - 1, ys = y + (t / 3) % 3 - 1, zs = z + t / 9 - 1;
    if (xs < 0 || xs >= X || ys < 0 || ys >= Y || zs < 0 || zs >= Z) return false;
    v = xs + (long long)X * (ys + (long long)Y * zs);
    return true;
}

// col[v][t*C + c] = X[neighbour t of v][c] (zero outside the grid).  One thread per (v, t, 8 channels).
__global__ void k_im2col(const __nv_bfloat16* __restrict__ Xin, int C, int X, int Y, int Z,
                         __nv_bfloat16* __restrict__ col)
{
    const long long V = (long long)X * Y * Z;
    const int C8 = C / 8;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;     // (v * 27 + t) * C8 + q
    if (i >= V * 27 * C8) return;
    const int q = (int)(i % C8);
    const long long vt = i / C8;
    const int t = (int)(vt % 27);
    const long long v = vt / 27;
    const int x = (int)(v % X), y = (int)((v / X) % Y), z = (int)(v / ((long long)X * Y));
    long long s;
    uint4 val = make_uint4(0, 0, 0, 0);
    if (tap_src(t, x, y, z, X, Y, Z, s)) val = *reinterpret_cast<const uint4*>(Xin + s * C + 8 * q);
    *reinterpret_cast<uint4*>(col + (v * 27 + t) * C + 8 * q) = val;
}

// The transpose of the column matrix, colT[t*C + c][v] = X[neighbour t of v][c], zero for v in
// [V, Vp): the weight gradients' operand, without the column matrix in between.  A block takes 64
// voxels x up to 64 channels of one tap through shared memory; Vp a multiple of 8.
__global__ void __launch_bounds__(256) k_im2col_t(const __nv_bfloat16* __restrict__ Xin, int C, int X, int Y, int Z,
                                                  long long Vp, __nv_bfloat16* __restrict__ colT)
{
    __shared__ __nv_bfloat16 tile[64][66];                 // [channel][voxel]
    const long long V = (long long)X * Y * Z, v0 = (long long)blockIdx.x * 64;
    const int t = blockIdx.y, cb = blockIdx.z * 64, nc = C - cb < 64 ? C - cb : 64;
    for (int e = threadIdx.x; e < 64 * (nc / 8); e += 256) {
        const int k = e / (nc / 8), q = e % (nc / 8);
        const long long v = v0 + k;
        uint4 val = make_uint4(0, 0, 0, 0);
        long long s;
        if (v < V && tap_src(t, (int)(v % X), (int)((v / X) % Y), (int)(v / ((long long)X * Y)), X, Y, Z, s))
            val = __ldg(reinterpret_cast<const uint4*>(Xin + s * C + cb + 8 * q));
        const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(&val);
#pragma unroll
        for (int j = 0; j < 8; ++j) tile[8 * q + j][k] = h[j];
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 8 * nc; e += 256) {
        const int c = e / 8, q = e % 8;
        if (v0 + 8 * q >= Vp) continue;
        __align__(16) __nv_bfloat16 h[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) h[j] = tile[c][8 * q + j];
        *reinterpret_cast<uint4*>(colT + ((long long)t * C + cb + c) * Vp + v0 + 8 * q) = *reinterpret_cast<uint4*>(h);
    }
}

// dX[v][c] = sum_t dcol[u][t*C + c] over the voxels u whose tap t reads v (u = v - offset_t).
__global__ void k_col2im(const float* __restrict__ dcol, int C, int X, int Y, int Z, float* __restrict__ dX)
{
    const long long V = (long long)X * Y * Z;
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;     // v * C + c
    if (i >= V * C) return;
    const int c = (int)(i % C);
    const long long v = i / C;
    const int x = (int)(v % X), y = (int)((v / X) % Y), z = (int)(v / ((long long)X * Y));
    float s = 0.f;
    for (int t = 0; t < 27; ++t) {
        long long u;
        // u reads v through tap t iff v is u's tap-t neighbour, i.e. u = v - offset_t = v's tap (26 - t)
        if (tap_src(26 - t, x, y, z, X, Y, Z, u)) s += dcol[(u * 27 + t) * C + c];
    }
    dX[i] = s;
}

// out[c][r] = in[r][c] for r < R; columns r in [R, Rp) of out are zero (K padding of the GEMMs).
__global__ void k_transpose_bf16(const __nv_bfloat16* __restrict__ in, long long R, int C, long long Rp,
                                 __nv_bfloat16* __restrict__ out)
{
    __shared__ __nv_bfloat16 tile[32][33];
    const long long r0 = (long long)blockIdx.x * 32;
    const int c0 = blockIdx.y * 32;
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const long long r = r0 + k;
        const int c = c0 + threadIdx.x;
        tile[k][threadIdx.x] = (r < R && c < C) ? in[r * C + c] : __float2bfloat16_rn(0.f);
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int c = c0 + k;
        const long long r = r0 + threadIdx.x;
        if (c < C && r < Rp) out[(long long)c * Rp + r] = tile[threadIdx.x][k];
    }
}

// Backward through ReLU: g = dY * (Y > 0) (or dY when relu == 0), as bf16, and its column sums
// (the bias gradient).  A block's threads keep one column each over its rows, so a column is one
// atomic per block instead of one per element (24 us a layer on 12,288 x 64, all on 64 addresses).
__global__ void __launch_bounds__(256) k_act_grad(const float* __restrict__ dY, const __nv_bfloat16* __restrict__ Y,
                                                  long long V, int C, int relu, __nv_bfloat16* __restrict__ g,
                                                  float* __restrict__ dbias)
{
    __shared__ float sum[256];
    const int per = 256 / C, r = threadIdx.x / C, c = threadIdx.x % C;      // rows of a pass; C <= 256
    float acc = 0.f;
    if (r < per)
        for (long long row = (long long)blockIdx.x * per + r; row < V; row += (long long)gridDim.x * per) {
            const long long i = row * C + c;
            float v = dY[i];
            if (relu && !(__bfloat162float(Y[i]) > 0.f)) v = 0.f;
            g[i] = __float2bfloat16_rn(v);
            acc += v;
        }
    sum[threadIdx.x] = acc;
    __syncthreads();
    if (r == 0) {
        for (int k = 1; k < per; ++k) acc += sum[k * C + c];
        atomicAdd(dbias + c, acc);
    }
}
// The same for any number of columns, one element per thread.
__global__ void k_act_grad_wide(const float* __restrict__ dY, const __nv_bfloat16* __restrict__ Y, long long V, int C,
                                int relu, __nv_bfloat16* __restrict__ g, float* __restrict__ dbias)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= V * C) return;
    float v = dY[i];
    if (relu && !(__bfloat162float(Y[i]) > 0.f)) v = 0.f;
    g[i] = __float2bfloat16_rn(v);
    atomicAdd(dbias + (i % C), v);
}

// Pooling and upsampling are copies with a few additions, bound by their bytes: a thread takes N = 8
// channels of a voxel where rows allow it (120k voxels x 64: pooling 12 -> 6 us, upsampling 46 -> 8), and
// its index arithmetic is 32-bit (I) where the grid is small enough.
// Thread index -> voxel of an A x B x C grid and first channel.  False: nothing to do.
template <int N, typename I>
__device__ __forceinline__ bool voxel_of(int C, int A, int B, int Z, I& v, int& c, int& x, int& y, int& z)
{
    const I i = (I)blockIdx.x * (I)blockDim.x + (I)threadIdx.x, per = (I)(C / N);
    v = i / per;
    c = (int)(i - v * per) * N;
    if (v >= (I)A * (I)B * (I)Z) return false;
    const I yz = v / (I)A;
    x = (int)(v - yz * (I)A);
    z = (int)(yz / (I)B);
    y = (int)(yz - (I)z * (I)B);
    return true;
}

// The sum over the eight children of a voxel of the half grid, in the order of their index.
template <int N, typename T>
__device__ __forceinline__ void sum_children(float (&s)[N], const T* __restrict__ in, int C, int X, int Y, int x, int y,
                                             int z, int c)
{
#pragma unroll
    for (int j = 0; j < N; ++j) s[j] = 0.f;
#pragma unroll
    for (int d = 0; d < 8; ++d) {
        const long long v = (2 * x + (d & 1)) + (long long)X * ((2 * y + ((d >> 1) & 1)) + (long long)Y * (2 * z + (d >> 2)));
        float a[N];
        load_n<N>(a, in + v * C + c);
#pragma unroll
        for (int j = 0; j < N; ++j) s[j] += a[j];
    }
}
__device__ __forceinline__ long long parent_of(int x, int y, int z, int X, int Y)
{
    return (x / 2) + (long long)(X / 2) * ((y / 2) + (long long)(Y / 2) * (z / 2));
}

// 2x2x2 average pooling of a (Z, Y, X) grid (even sizes) and its backward.
template <int N, typename I>
__global__ void __launch_bounds__(256) k_pool2(const __nv_bfloat16* __restrict__ in, int C, int X, int Y, int Z,
                                               __nv_bfloat16* __restrict__ out)
{
    I v;
    int c, x, y, z;
    if (!voxel_of<N, I>(C, X / 2, Y / 2, Z / 2, v, c, x, y, z)) return;
    float s[N];
    sum_children<N>(s, in, C, X, Y, x, y, z, c);
#pragma unroll
    for (int j = 0; j < N; ++j) s[j] *= 0.125f;
    store_n<N>(out + (long long)v * C + c, s);
}
template <int N, typename I>
__global__ void __launch_bounds__(256) k_pool2_back(const float* __restrict__ dout, int C, int X, int Y, int Z,
                                                    float* __restrict__ din, int accumulate)
{
    I v;
    int c, x, y, z;
    if (!voxel_of<N, I>(C, X, Y, Z, v, c, x, y, z)) return;
    float g[N], d[N];
    load_n<N>(g, dout + parent_of(x, y, z, X, Y) * C + c);
    float* at = din + (long long)v * C + c;
    if (accumulate) load_n<N>(d, at);
#pragma unroll
    for (int j = 0; j < N; ++j) d[j] = accumulate ? d[j] + 0.125f * g[j] : 0.125f * g[j];
    store_n<N>(at, d);
}

// out[v] = coarse[parent(v)] + skip[v] (nearest 2x upsampling plus the skip connection) and its
// backward for the coarse input: dcoarse[vh] = sum over the 8 children of dout.
template <int N, typename I>
__global__ void __launch_bounds__(256) k_up2_add(const __nv_bfloat16* __restrict__ coarse,
                                                 const __nv_bfloat16* __restrict__ skip, int C, int X, int Y, int Z,
                                                 __nv_bfloat16* __restrict__ out)
{
    I v;
    int c, x, y, z;
    if (!voxel_of<N, I>(C, X, Y, Z, v, c, x, y, z)) return;
    float a[N], b[N];
    load_n<N>(a, coarse + parent_of(x, y, z, X, Y) * C + c);
    load_n<N>(b, skip + (long long)v * C + c);
#pragma unroll
    for (int j = 0; j < N; ++j) a[j] += b[j];
    store_n<N>(out + (long long)v * C + c, a);
}
template <int N, typename I>
__global__ void __launch_bounds__(256) k_up2_back(const float* __restrict__ dout, int C, int X, int Y, int Z,
                                                  float* __restrict__ dcoarse)
{
    I v;
    int c, x, y, z;
    if (!voxel_of<N, I>(C, X / 2, Y / 2, Z / 2, v, c, x, y, z)) return;
    float s[N];
    sum_children<N>(s, dout, C, X, Y, x, y, z, c);
    store_n<N>(dcoarse + (long long)v * C + c, s);
}

// Masked mean-square error of pred[v][0..nout) (row stride Cp) against target[v][0..nout):
// loss += sum m (p - t)^2 / n, dpred = 2 m (p - t) / n (padding channels get 0); a NULL loss or dpred is
// left out.  The loss: float32 terms, summed in float64 in a fixed order by the first cluster of 8 CTAs
// (a partial of each in the first one's shared memory: no scratch, no atomics) and rounded once, so it
// is repeatable.  The other CTAs make the gradient beside it, an element a thread.
// A float32 atomic per term missed the exact sum of 12,288 voxels by 3e-6 and that of 120,000 by 9e-5,
// and a call took 78 and 737 us (this 6.5 and 18.5; 1000 voxels 8.3 and 6.5).
constexpr int kLossCtas = 8, kMseThreads = 1024;
__global__ void __cluster_dims__(kLossCtas, 1, 1) __launch_bounds__(kMseThreads)
    k_mse(const float* pred, int Cp, const float* __restrict__ target, int nout, const float* __restrict__ mask,
          long long V, float inv_n, float* dpred, float* loss)
{
    namespace cg = cooperative_groups;
    __shared__ double warps[kMseThreads / 32], ctas[kLossCtas];
    const int first = loss ? kLossCtas : 0;                // CTAs in front of the gradient's
    if ((int)blockIdx.x >= first) {
        const long long i = (long long)((int)blockIdx.x - first) * kMseThreads + threadIdx.x;     // v * Cp + c
        if (i >= V * Cp) return;
        const int c = (int)(i % Cp);
        const long long v = i / Cp;
        float g = 0.f;
        if (c < nout) {
            const float d = pred[i] - target[v * nout + c];
            g = 2.f * mask[v] * d * inv_n;
        }
        dpred[i] = g;
        return;
    }
    const cg::cluster_group cluster = cg::this_cluster();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double s = 0.0;
    for (long long v = (long long)blockIdx.x * kMseThreads + threadIdx.x; v < V; v += kLossCtas * kMseThreads) {
        const float m = mask[v];
        for (int c = 0; c < nout; ++c) {
            const float d = pred[v * Cp + c] - target[v * nout + c];
            s += (double)(m * d * d * inv_n);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) warps[warp] = s;
    __syncthreads();
    cluster.sync();                                        // every CTA has started
    if (threadIdx.x == 0) {
        for (int w = 1; w < kMseThreads / 32; ++w) s += warps[w];
        cluster.map_shared_rank(ctas, 0)[cluster.block_rank()] = s;
    }
    cluster.sync();
    if (cluster.block_rank() || threadIdx.x) return;
    s = ctas[0];
    for (int b = 1; b < kLossCtas; ++b) s += ctas[b];
    *loss = (float)((double)*loss + s);
}

// Adam step on float32 master weights, refreshing their bf16 copy.
__global__ void k_adam(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ s,
                       long long n, float lr, float b1, float b2, float eps, float c1, float c2,
                       __nv_bfloat16* __restrict__ wb)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi, si = b2 * s[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    s[i] = si;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(si / c2) + eps);
    w[i] = wi;
    if (wb) wb[i] = __float2bfloat16_rn(wi);
}

inline unsigned blocks(long long n, int t) { return (unsigned)((n + t - 1) / t); }

// Eight channels a thread: rows of a multiple of 8 channels, 16-byte aligned arrays, 32-bit indexes.
inline bool by_eights(long long elements, int C, const void* a, const void* b, const void* c = nullptr)
{
    return C % 8 == 0 && elements < (1LL << 31) &&
           ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}

}  // namespace

extern "C" {

int lbm_nn_im2col(const uint16_t* x, int C, int X, int Y, int Z, uint16_t* col, void* stream)
{
    g_err[0] = 0;
    if (!x || !col || C % 8 || X < 1 || Y < 1 || Z < 1) return fail(LBM_ERR_ARG, "lbm_nn_im2col: bad arguments");
    const long long n = (long long)X * Y * Z * 27 * (C / 8);
    k_im2col<<<blocks(n, 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const __nv_bfloat16*>(x), C, X, Y, Z, reinterpret_cast<__nv_bfloat16*>(col));
    return check_launch("k_im2col");
}

int lbm_nn_im2col_t(const uint16_t* x, int C, int X, int Y, int Z, int64_t Vp, uint16_t* colT, void* stream)
{
    g_err[0] = 0;
    const long long V = (long long)X * Y * Z;
    if (!x || !colT || C < 8 || C % 8 || X < 1 || Y < 1 || Z < 1 || Vp < V || Vp % 8)
        return fail(LBM_ERR_ARG, "lbm_nn_im2col_t: bad arguments (channels and Vp multiples of 8, Vp >= voxels)");
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(colT)) & 15)
        return fail(LBM_ERR_ARG, "lbm_nn_im2col_t: x and colT must be 16-byte aligned");
    k_im2col_t<<<dim3(blocks(Vp, 64), 27, (unsigned)((C + 63) / 64)), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const __nv_bfloat16*>(x), C, X, Y, Z, Vp, reinterpret_cast<__nv_bfloat16*>(colT));
    return check_launch("k_im2col_t");
}

int lbm_conv3_bf16(const uint16_t* x, int C, int X, int Y, int Z, const uint16_t* W, int N, void* D, int epilogue,
                   const float* bias, int* err, void* stream)
{
    g_err[0] = 0;
    if (!x || !W || !D || !bias || !err) return fail(LBM_ERR_ARG, "lbm_conv3_bf16: NULL pointer");
    if ((C != 8 && (C < 64 || C % 64)) || N < 8 || N % 8 || X < 1 || Y < 1 || Z < 1 || (long long)X * Y * Z > INT32_MAX - GM)
        return fail(LBM_ERR_ARG, "lbm_conv3_bf16: %d -> %d channels on %dx%dx%d (inputs 8 or a multiple of 64, outputs of 8)",
                    C, N, X, Y, Z);
    if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(D)) & 15)
        return fail(LBM_ERR_ARG, "lbm_conv3_bf16: x, W and D must be 16-byte aligned");
    const __nv_bfloat16* xb = reinterpret_cast<const __nv_bfloat16*>(x);
    const __nv_bfloat16* wb = reinterpret_cast<const __nv_bfloat16*>(W);
    const ConvTiles g = conv_tiles(X, Y, Z);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    switch (epilogue) {
    case EPI_BF16_BIAS: return launch_conv<EPI_BF16_BIAS>(xb, C, g, wb, N, D, bias, err, st);
    case EPI_BF16_BIAS_RELU: return launch_conv<EPI_BF16_BIAS_RELU>(xb, C, g, wb, N, D, bias, err, st);
    case EPI_F32_BIAS: return launch_conv<EPI_F32_BIAS>(xb, C, g, wb, N, D, bias, err, st);
    default: return fail(LBM_ERR_ARG, "lbm_conv3_bf16: epilogue %d (2, 3 or 4)", epilogue);
    }
}

int lbm_conv3_back(const uint16_t* g, int O, int X, int Y, int Z, const uint16_t* Wt, int C, float* dX, int* err,
                   void* stream)
{
    g_err[0] = 0;
    if (!g || !Wt || !dX || !err) return fail(LBM_ERR_ARG, "lbm_conv3_back: NULL pointer");
    if (O < 8 || O % 8 || C < 64 || C % 64 || X < 1 || Y < 1 || Z < 1)
        return fail(LBM_ERR_ARG, "lbm_conv3_back: %d -> %d channels on %dx%dx%d (outputs a multiple of 8, inputs of 64)", O, C,
                    X, Y, Z);
    if ((reinterpret_cast<uintptr_t>(g) | reinterpret_cast<uintptr_t>(Wt) | reinterpret_cast<uintptr_t>(dX)) & 15)
        return fail(LBM_ERR_ARG, "lbm_conv3_back: g, Wt and dX must be 16-byte aligned");
    const ConvTiles t = conv_tiles(X, Y, Z);
    CUtensorMap tg, tw;
    if (!bf16_grid_map(&tg, reinterpret_cast<const __nv_bfloat16*>(g), O, t) ||
        !bf16_tile_map(&tw, reinterpret_cast<const __nv_bfloat16*>(Wt), 27 * C, O, O, kBackN))
        return fail(LBM_ERR_CUDA, "lbm_conv3_back: no tensor map for this grid");
    const int smem = kBackStages * (GM * 128 + kBackN * 128) + 1024;
    if (const cudaError_t e = allow_shared(k_conv_back, smem))
        return fail(LBM_ERR_CUDA, "lbm_conv3_back: %d bytes of shared memory: %s", smem, cudaGetErrorString(e));
    k_conv_back<<<dim3((unsigned)(t.nx * t.ny * t.nz), (unsigned)(C / kBackN)), kWsThreads, smem,
                  reinterpret_cast<cudaStream_t>(stream)>>>(tg, tw, t, O, C, dX, err);
    return check_launch("k_conv_back");
}

int lbm_nn_col2im(const float* dcol, int C, int X, int Y, int Z, float* dx, void* stream)
{
    g_err[0] = 0;
    if (!dcol || !dx || C < 1 || X < 1 || Y < 1 || Z < 1) return fail(LBM_ERR_ARG, "lbm_nn_col2im: bad arguments");
    const long long n = (long long)X * Y * Z * C;
    k_col2im<<<blocks(n, 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(dcol, C, X, Y, Z, dx);
    return check_launch("k_col2im");
}

int lbm_nn_transpose(const uint16_t* in, int64_t R, int C, int64_t Rp, uint16_t* out, void* stream)
{
    g_err[0] = 0;
    if (!in || !out || R < 1 || C < 1 || Rp < R) return fail(LBM_ERR_ARG, "lbm_nn_transpose: bad arguments");
    dim3 grid(blocks(Rp, 32), blocks(C, 32));
    k_transpose_bf16<<<grid, dim3(32, 8), 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const __nv_bfloat16*>(in), R, C, Rp, reinterpret_cast<__nv_bfloat16*>(out));
    return check_launch("k_transpose_bf16");
}

int lbm_nn_act_grad(const float* dy, const uint16_t* y, int64_t V, int C, int relu, uint16_t* g, float* dbias,
                    void* stream)
{
    g_err[0] = 0;
    if (!dy || !g || !dbias || (relu && !y) || V < 1 || C < 1) return fail(LBM_ERR_ARG, "lbm_nn_act_grad: bad arguments");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const __nv_bfloat16* yb = reinterpret_cast<const __nv_bfloat16*>(y);
    __nv_bfloat16* gb = reinterpret_cast<__nv_bfloat16*>(g);
    if (C <= 256) {
        // blocks of about 8 passes each, at most 8 per SM
        const long long passes = (V + 256 / C - 1) / (256 / C);
        const long long grid = passes / 8 + 1 < 8 * sm_count() ? passes / 8 + 1 : 8 * sm_count();
        k_act_grad<<<(unsigned)grid, 256, 0, st>>>(dy, yb, V, C, relu, gb, dbias);
    } else {
        k_act_grad_wide<<<blocks(V * C, 256), 256, 0, st>>>(dy, yb, V, C, relu, gb, dbias);
    }
    return check_launch("k_act_grad");
}

int lbm_nn_pool2(const uint16_t* in, int C, int X, int Y, int Z, uint16_t* out, void* stream)
{
    g_err[0] = 0;
    if (!in || !out || C < 1 || X % 2 || Y % 2 || Z % 2 || X < 2 || Y < 2 || Z < 2)
        return fail(LBM_ERR_ARG, "lbm_nn_pool2: bad arguments (even grid sizes)");
    const long long n = (long long)X * Y * Z / 8 * C;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const __nv_bfloat16* a = reinterpret_cast<const __nv_bfloat16*>(in);
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(out);
    if (by_eights(n, C, in, out)) k_pool2<8, uint32_t><<<blocks(n / 8, 256), 256, 0, st>>>(a, C, X, Y, Z, o);
    else k_pool2<1, long long><<<blocks(n, 256), 256, 0, st>>>(a, C, X, Y, Z, o);
    return check_launch("k_pool2");
}

int lbm_nn_pool2_back(const float* dout, int C, int X, int Y, int Z, float* din, int accumulate, void* stream)
{
    g_err[0] = 0;
    if (!dout || !din || C < 1 || X % 2 || Y % 2 || Z % 2) return fail(LBM_ERR_ARG, "lbm_nn_pool2_back: bad arguments");
    const long long n = (long long)X * Y * Z * C;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (by_eights(n, C, dout, din)) k_pool2_back<8, uint32_t><<<blocks(n / 8, 256), 256, 0, st>>>(dout, C, X, Y, Z, din, accumulate);
    else k_pool2_back<1, long long><<<blocks(n, 256), 256, 0, st>>>(dout, C, X, Y, Z, din, accumulate);
    return check_launch("k_pool2_back");
}

int lbm_nn_up2_add(const uint16_t* coarse, const uint16_t* skip, int C, int X, int Y, int Z, uint16_t* out,
                   void* stream)
{
    g_err[0] = 0;
    if (!coarse || !skip || !out || C < 1 || X % 2 || Y % 2 || Z % 2)
        return fail(LBM_ERR_ARG, "lbm_nn_up2_add: bad arguments");
    const long long n = (long long)X * Y * Z * C;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const __nv_bfloat16 *a = reinterpret_cast<const __nv_bfloat16*>(coarse), *b = reinterpret_cast<const __nv_bfloat16*>(skip);
    __nv_bfloat16* o = reinterpret_cast<__nv_bfloat16*>(out);
    if (by_eights(n, C, coarse, skip, out)) k_up2_add<8, uint32_t><<<blocks(n / 8, 256), 256, 0, st>>>(a, b, C, X, Y, Z, o);
    else k_up2_add<1, long long><<<blocks(n, 256), 256, 0, st>>>(a, b, C, X, Y, Z, o);
    return check_launch("k_up2_add");
}

int lbm_nn_up2_back(const float* dout, int C, int X, int Y, int Z, float* dcoarse, void* stream)
{
    g_err[0] = 0;
    if (!dout || !dcoarse || C < 1 || X % 2 || Y % 2 || Z % 2) return fail(LBM_ERR_ARG, "lbm_nn_up2_back: bad arguments");
    const long long n = (long long)X * Y * Z / 8 * C;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    if (by_eights(n, C, dout, dcoarse)) k_up2_back<8, uint32_t><<<blocks(n / 8, 256), 256, 0, st>>>(dout, C, X, Y, Z, dcoarse);
    else k_up2_back<1, long long><<<blocks(n, 256), 256, 0, st>>>(dout, C, X, Y, Z, dcoarse);
    return check_launch("k_up2_back");
}

int lbm_nn_mse(const float* pred, int Cp, const float* target, int nout, const float* mask, int64_t V, float inv_n,
               float* dpred, float* loss, void* stream)
{
    g_err[0] = 0;
    if (!pred || !target || !mask || !dpred || !loss || nout > Cp || V < 1) return fail(LBM_ERR_ARG, "lbm_nn_mse: bad arguments");
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    const unsigned grad = (blocks(V * Cp, kMseThreads) + kLossCtas - 1) / kLossCtas * kLossCtas;     // whole clusters
    if (pred < dpred + V * Cp && dpred < pred + V * Cp) {  // in place: the loss reads pred first
        k_mse<<<kLossCtas, kMseThreads, 0, st>>>(pred, Cp, target, nout, mask, V, inv_n, nullptr, loss);
        if (int e = check_launch("k_mse")) return e;
        k_mse<<<grad, kMseThreads, 0, st>>>(pred, Cp, target, nout, mask, V, inv_n, dpred, nullptr);
    } else {
        k_mse<<<kLossCtas + grad, kMseThreads, 0, st>>>(pred, Cp, target, nout, mask, V, inv_n, dpred, loss);
    }
    return check_launch("k_mse");
}

int lbm_nn_adam(float* w, const float* g, float* m, float* s, int64_t n, float lr, float b1, float b2, float eps,
                int step, uint16_t* wbf16, void* stream)
{
    g_err[0] = 0;
    if (!w || !g || !m || !s || n < 1 || step < 1) return fail(LBM_ERR_ARG, "lbm_nn_adam: bad arguments");
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    k_adam<<<blocks(n, 256), 256, 0, reinterpret_cast<cudaStream_t>(stream)>>>(
        w, g, m, s, n, lr, b1, b2, eps, c1, c2, reinterpret_cast<__nv_bfloat16*>(wbf16));
    return check_launch("k_adam");
}

int lbm_gemm_bf16(const uint16_t* A, int lda, const uint16_t* B, int ldb, int M, int N, int K, void* D, int ldd,
                  int epilogue, const float* bias, int* err, void* stream)
{
    g_err[0] = 0;
    if (!A || !B || !D || !err) return fail(LBM_ERR_ARG, "lbm_gemm_bf16: NULL pointer");
    if (M < 1 || N < 1 || K < 1) return fail(LBM_ERR_ARG, "lbm_gemm_bf16: empty product %dx%dx%d", M, N, K);
    if (K % 8 || lda % 8 || ldb % 8 || lda < K || ldb < K)
        return fail(LBM_ERR_ARG, "lbm_gemm_bf16: K, lda and ldb must be multiples of 8 with lda, ldb >= K");
    if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15)
        return fail(LBM_ERR_ARG, "lbm_gemm_bf16: A and B must be 16-byte aligned");
    if (ldd < N) return fail(LBM_ERR_ARG, "lbm_gemm_bf16: ldd < N");
    if (epilogue < 0 || epilogue > 4) return fail(LBM_ERR_ARG, "lbm_gemm_bf16: unknown epilogue %d", epilogue);
    const int bn = N <= 32 ? 32 : N <= 64 ? 64 : N <= 128 ? 128 : 256;
    const __nv_bfloat16* a = reinterpret_cast<const __nv_bfloat16*>(A);
    const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(B);
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    switch (epilogue) {
    case EPI_F32: return launch_gemm_any<EPI_F32>(bn, a, lda, b, ldb, M, N, K, D, ldd, bias, err, st);
    case EPI_F32_ADD: return launch_gemm_any<EPI_F32_ADD>(bn, a, lda, b, ldb, M, N, K, D, ldd, bias, err, st);
    case EPI_BF16_BIAS: return launch_gemm_any<EPI_BF16_BIAS>(bn, a, lda, b, ldb, M, N, K, D, ldd, bias, err, st);
    case EPI_F32_BIAS: return launch_gemm_any<EPI_F32_BIAS>(bn, a, lda, b, ldb, M, N, K, D, ldd, bias, err, st);
    default: return launch_gemm_any<EPI_BF16_BIAS_RELU>(bn, a, lda, b, ldb, M, N, K, D, ldd, bias, err, st);
    }
}

}  // extern "C"
