// The warm-start network: a coordinate MLP (inflow parameters and cell
// position -> a converged state of the plain step), trained and evaluated
// on the GPU by this file's kernels.
//
//   gemm_tc_kernel        C[M,N] (fp32) = A[M,K] . B[N,K]^T with bf16 operands
//                         on the 5th-generation tensor cores (tcgen05.mma,
//                         fp32 accumulator in tensor memory), both operands
//                         k-contiguous: X.W^T (forward), dZ.(W^T)^T
//                         (backward, data) and (dZ^T).(H^T)^T (backward,
//                         weights; split over K into partial tiles that
//                         splitk_reduce_kernel adds in a fixed order)
//   gemm_tma_kernel       the same GEMM with the operand tiles brought in by
//                         the tensor memory accelerator (one thread issues
//                         cp.async.bulk.tensor per tile; no cluster
//                         multicast) and, for the forward layers, bias +
//                         GELU applied to the accumulator as it leaves
//                         tensor memory, the hidden layers' Z and H tiles
//                         staged in shared memory and stored by the TMA;
//                         used whenever both operands' rows are 16-byte
//                         aligned
//                         In a training step the same epilogue also stores
//                         H^T, and the backward data GEMMs (EPI 2) apply
//                         GELU' to the accumulator and store dZ, dZ^T and the
//                         tile's column sums: no fp32 dH or dZ in memory, no
//                         transpose, activation or column-sum launch
//   grad_adam_kernel      a training step's end: every gradient from its
//                         split partial sums in a fixed order, Adam, and the
//                         bf16 copies of the weights (W and W^T)
//   mse_grad_kernel       dY = 2 (Y - T) / (M N) as the last layer's dZ, dZ^T
//                         and column sums, squared error per row
// The kernels below serve networks the fused training step does not take
// (see train_fused):
//   transpose_bf16_kernel the transposed operands of the backward GEMMs
//   features_kernel       network inputs: the raw inputs, then sin / cos of
//                         2^f pi s of the last two (the cell position), bf16
//   gather_kernel         a mini-batch of rows of the training set, drawn by
//                         a counter-based hash of (seed, step, row)
//   bias_act_kernel       Z = C + bias, H = GELU(Z) (or Z), H as bf16
//   act_bwd_kernel        dZ = dH * GELU'(Z) (or dH), fp32 and bf16
//   col_sum_*_kernel      bias gradients: column sums in a fixed order
//   mse_kernel            dY = 2 (Y - T) / (M N), squared error per row
//   loss_kernel           mean squared error of the batch (fixed order)
//   adam_kernel           Adam on the fp32 master weights, bf16 copy refreshed
// GELU(x) = x Phi(x) = x/2 (1 + erf(x / sqrt 2)) through CUDA's erff; its
// derivative Phi(x) + x phi(x) through erff and expf.
#include <cuda.h>  // CUtensorMap and its enums (the encoder is looked up at run time)
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "../../include/gelios_b200.h"
#include "graph_capture.cuh"
#include "mlp_plan.cuh"

namespace gelios {
void set_error(const std::string& msg);
}  // namespace gelios
using namespace gelios;

namespace {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// 16-byte asynchronous copy global -> shared; bytes beyond src_bytes are zero
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, int src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
// all but the newest TC_STAGES - 1 commit groups have landed
__device__ __forceinline__ void cp_async_wait_ring() { asm volatile("cp.async.wait_group 3;\n" ::); }

// ---- the GEMM on the 5th-generation tensor cores (tcgen05)
// C[M][N] (fp32, rows of ldc) = sum_k A[m][k] B[n][k], A and B bf16 with k
// contiguous (rows of lda / ldb); blockIdx.z: K slice [z kc, (z+1) kc),
// written to C + z c_split.  One 128 x 128 fp32 accumulator tile per CTA
// in tensor memory (128 lanes x 128 columns), K in stages of 64: both
// operand tiles (128 rows x 64 bf16)
// staged by cp.async in the canonical K-major layout without swizzle (core
// matrices of 8 rows x 16 bytes; 16-byte K chunks 128 bytes apart, 8-row
// groups 1024 bytes apart), a ring of four stages (the whole K of a
// 256-wide layer in flight at once).  One thread issues four tcgen05.mma
// (M 128, N 128, K 16) per stage and commits them to the stage's mbarrier,
// which frees the stage for the load of the tile four steps on; the epilogue
// reads the accumulator with tcgen05.ld (warp w: rows 32w..32w+31).  Every
// mbarrier wait is bounded: on expiry the CTA raises `status` and goes on.
constexpr int TC_BM = 128, TC_BN = 128, TC_BK = kGemmBK, TC_THREADS = 128;
constexpr int TC_TILE = TC_BM * TC_BK * 2;  // bytes of one operand tile
constexpr int TC_STAGES = 4;
constexpr int TC_SMEM = 2 * TC_STAGES * TC_TILE;  // A and B per stage
constexpr uint32_t TC_LBO = 128, TC_SBO = 1024;
// instruction descriptor of kind::f16: fp32 accumulator (bits 4-5 = 1),
// A and B bf16 (bits 7-9, 10-12 = 1), both K-major (bits 15, 16 = 0),
// N >> 3 in bits 17-22, M >> 4 in bits 24-28
constexpr uint32_t TC_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TC_BN >> 3) << 17) |
                              ((uint32_t)(TC_BM >> 4) << 24);

// shared-memory matrix descriptor: start address >> 4 (bits 0-13), leading
// byte offset >> 4 (16-29), stride byte offset >> 4 (32-45), version 1
// (bits 46-47), no swizzle (bits 61-63 = 0)
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr) {
    return static_cast<uint64_t>((saddr >> 4) & 0x3FFFu) | (static_cast<uint64_t>((TC_LBO >> 4) & 0x3FFFu) << 16) |
           (static_cast<uint64_t>((TC_SBO >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
__device__ __forceinline__ uint32_t tc_off(int r, int kc) {
    return static_cast<uint32_t>((r >> 3) * TC_SBO + kc * TC_LBO + (r & 7) * 16);
}
__device__ __forceinline__ void mbar_init(uint64_t* b, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* b, unsigned parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait for the phase of the given parity; false if it did not complete
__device__ __forceinline__ bool mbar_wait(uint64_t* b, unsigned parity) {
    for (int i = 0; i < (1 << 22); i++)
        if (mbar_try_wait(b, parity)) return true;
    return false;
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }

// rows row0.. x k k0..k0+63 of a k-contiguous operand into a canonical tile.
// A warp stages 8 rows x 4 chunks per pass (lane: row lane & 7, chunk
// lane >> 3): each row's 64 bytes are read contiguously, and the 8 rows of
// one chunk fill one 128-byte core matrix (no bank conflict); 4 warps x 8
// passes cover 16 row groups x 2 chunk halves.
template <bool VEC>
__device__ __forceinline__ void tc_load(uint8_t* tile, const __nv_bfloat16* __restrict__ G, int64_t ld, int row0,
                                        int nrows, int k0, int ke) {
    const __nv_bfloat16 zero = __float2bfloat16(0.f);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int pass = 0; pass < 8; pass++) {
        const int unit = pass * 4 + warp;  // (row group, chunk half)
        const int r = (unit >> 1) * 8 + (lane & 7), kq = (unit & 1) * 4 + (lane >> 3);
        const int gr = row0 + r;
        const int gk = k0 + kq * 8;
        uint8_t* dst = tile + tc_off(r, kq);
        if (VEC && gr < nrows && gk + 8 <= ke) {
            cp_async16(smem_u32(dst), G + gr * ld + gk, 16);
        } else if (VEC && (gr >= nrows || gk >= ke)) {
            cp_async16(smem_u32(dst), G, 0);
        } else {
            __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(dst);
            for (int e = 0; e < 8; e++) d[e] = (gr < nrows && gk + e < ke) ? G[gr * ld + gk + e] : zero;
        }
    }
}

template <bool AV, bool BV>
__global__ void __launch_bounds__(TC_THREADS) gemm_tc_kernel(int M, int N, int K, int kc,
                                                           const __nv_bfloat16* __restrict__ A, int64_t lda,
                                                           const __nv_bfloat16* __restrict__ B, int64_t ldb,
                                                           float* __restrict__ C, int64_t ldc, int64_t c_split,
                                                           int* __restrict__ status) {
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    __shared__ uint64_t bars[TC_STAGES];
    __shared__ uint32_t tmem_slot;
    uint8_t* sA0 = tc_smem;
    uint8_t* sB0 = tc_smem + TC_STAGES * TC_TILE;
    const int m0 = blockIdx.y * TC_BM, n0 = blockIdx.x * TC_BN;
    const int kb = blockIdx.z * kc, ke = min(K, kb + kc);
    C += blockIdx.z * c_split;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                     "r"(TC_BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < TC_STAGES; i++) mbar_init(&bars[i], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int nk = ke > kb ? (ke - kb + TC_BK - 1) / TC_BK : 0;
    bool ok = true;
    // prologue: tiles 0 .. TC_STAGES-2, one commit group each
    for (int j = 0; j < TC_STAGES - 1; j++) {
        if (j < nk) {
            tc_load<AV>(sA0 + j * TC_TILE, A, lda, m0, M, kb + j * TC_BK, ke);
            tc_load<BV>(sB0 + j * TC_TILE, B, ldb, n0, N, kb + j * TC_BK, ke);
        }
        cp_async_commit();
    }
    static_assert(TC_STAGES == 4, "cp_async_wait_ring waits for TC_STAGES - 1 groups");
    for (int it = 0; it < nk; it++) {
        const int s = it % TC_STAGES;
        const int nx = it + TC_STAGES - 1;  // the tile loaded now, into the stage iteration it-1 used
        if (nx < nk) {
            const int sx = nx % TC_STAGES;
            if (it >= 1 && !mbar_wait(&bars[sx], ((it - 1) / TC_STAGES) & 1)) ok = false;
            tc_load<AV>(sA0 + sx * TC_TILE, A, lda, m0, M, kb + nx * TC_BK, ke);
            tc_load<BV>(sB0 + sx * TC_TILE, B, ldb, n0, N, kb + nx * TC_BK, ke);
        }
        cp_async_commit();
        cp_async_wait_ring();
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");  // staged bytes visible to the tensor cores
        __syncthreads();
        if (threadIdx.x == 0) {
            tc_fence_after();
            const uint32_t a0 = smem_u32(sA0 + s * TC_TILE), b0 = smem_u32(sB0 + s * TC_TILE);
#pragma unroll
            for (int k = 0; k < TC_BK / 16; k++) {
                const uint64_t ad = tc_desc(a0 + k * 2 * TC_LBO), bd = tc_desc(b0 + k * 2 * TC_LBO);
                const uint32_t acc = (it > 0 || k > 0) ? 1u : 0u;
                asm volatile(
                    "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                    " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n}\n" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(TC_IDESC), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
                    : "memory");
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                             smem_u32(&bars[s]))
                         : "memory");
        }
    }
    if (nk > 0 && !mbar_wait(&bars[(nk - 1) % TC_STAGES], ((nk - 1) / TC_STAGES) & 1)) ok = false;
    tc_fence_after();
    const int64_t row = m0 + warp * 32 + lane;
#pragma unroll 1
    for (int c0 = 0; c0 < TC_BN; c0 += 16) {
        uint32_t v[16];
        if (nk > 0) {
            const uint32_t taddr = tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(c0);
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                "[%16];\n"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15])
                : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        } else {
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] = 0u;
        }
        if (row < M) {
            float* dst = C + row * ldc + n0 + c0;
            if (n0 + c0 + 16 <= N && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
                for (int j = 0; j < 16; j += 4)
                    *reinterpret_cast<float4*>(dst + j) = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                                                      __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
            } else {
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (n0 + c0 + j < N) dst[j] = __uint_as_float(v[j]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TC_BN) : "memory");
    }
    if (!ok) atomicOr(status, 1);
}

// out[c][r] = in[r][c] (bf16, rows of ldin -> rows of ldout), 32 x 32 tiles
__global__ void transpose_bf16_kernel(int R, int Cc, const __nv_bfloat16* __restrict__ in, int64_t ldin,
                                      __nv_bfloat16* __restrict__ out, int64_t ldout) {
    __shared__ unsigned short tile[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int y = threadIdx.y; y < 32; y += 8) {
        const int r = r0 + y, c = c0 + threadIdx.x;
        if (r < R && c < Cc) tile[y][threadIdx.x] = __bfloat16_as_ushort(in[r * ldin + c]);
    }
    __syncthreads();
    for (int y = threadIdx.y; y < 32; y += 8) {
        const int c = c0 + y, r = r0 + threadIdx.x;
        if (r < R && c < Cc) out[c * ldout + r] = __ushort_as_bfloat16(tile[threadIdx.x][y]);
    }
}

__global__ void splitk_reduce_kernel(int64_t n, int S, const float* __restrict__ part, float* __restrict__ out) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float s = 0.f;
    for (int z = 0; z < S; z++) s += part[z * n + i];
    out[i] = s;
}

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float x) {
    const float cdf = 0.5f * (1.f + erff(x * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
    return cdf + x * pdf;
}

// ---- the GEMM with TMA staging
// Per stage and operand one box of 64 k x rows (128 bytes x 128 rows for A,
// x 64 rows for B) loaded with the 128-byte swizzle: row r lands at r * 128
// bytes with its 16-byte chunks permuted by (r mod 8), which is the
// canonical K-major SWIZZLE_128B layout the MMA descriptor names (8-row
// groups 1024 bytes apart; the k-th 16-deep slice of the stage starts 32 k
// bytes into the rows).  Stage buffers are 1024-byte aligned.  Thread 0
// issues the loads (mbarrier expect_tx / complete_tx per stage), waits for
// each stage, issues its four MMAs and commits them to the stage's "empty"
// mbarrier before refilling it.  Out-of-range rows and k are zero-filled by
// the TMA unit.  EPI 0: C (fp32) as gemm_tc_kernel writes it;
// EPI 1: z = C + bias per column, then Z = z, H = bf16(act(z)), Hf = act(z)
// (each output optional, rows of N); EPI 2: see GemmEpilogue.
// tile: TM_BN = 64 columns per CTA (256 CTAs for a 8192 x 256 layer, two
// resident per SM: one's epilogue overlaps the other's loads); k-chunk
// stride of the A stage 128 rows x 16 bytes, of the B stage 64 x 16 bytes
constexpr int TM_BN = 64;
constexpr uint32_t TM_SBO = 1024;
constexpr int TM_TILE_B = TM_BN * TC_BK * 2;
// + 1024: the dynamic shared memory base is rounded up to 1024 bytes
constexpr int TM_SMEM = TC_STAGES * (TC_TILE + TM_TILE_B) + 1024;
constexpr uint32_t TM_IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TM_BN >> 3) << 17) |
                              ((uint32_t)(TC_BM >> 4) << 24);
// shared-memory matrix descriptor of a K-major SWIZZLE_128B operand: start
// address >> 4 (bits 0-13), leading byte offset 16 (unused for swizzled
// K-major layouts; bits 16-29), stride byte offset 1024 >> 4 (bits 32-45),
// version 1 (bits 46-47), base offset 0 (1024-aligned buffers), layout type
// 2 = SWIZZLE_128B (bits 61-63)
__device__ __forceinline__ uint64_t tm_desc(uint32_t saddr) {
    return static_cast<uint64_t>((saddr >> 4) & 0x3FFFu) | (1ull << 16) |
           (static_cast<uint64_t>((TM_SBO >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::
            "r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// the tile in shared memory -> global memory through the tensor map (rows
// and columns outside the tensor are not written); one bulk group per CTA
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, uint32_t src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];\n" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(src), "r"(x), "r"(y)
                 : "memory");
}

struct GemmEpilogue {
    const float* bias = nullptr;
    float* Z = nullptr;
    __nv_bfloat16* H = nullptr;
    float* Hf = nullptr;
    int act = 0;
    // training: the transpose of H (EPI 1, with tstore) or of dZ (EPI 2), N
    // rows of ldt (a multiple of 8, >= M; 16-byte aligned)
    __nv_bfloat16* HT = nullptr;
    int64_t ldt = 0;
    // EPI 2: dZ = acc * GELU'(Zin) -> H (rows of N, N % 8 == 0), HT, and the
    // column sums of every 128-row tile, row by row, -> colpart[tile][N]
    const float* Zin = nullptr;
    float* colpart = nullptr;
};
// transposed tile in shared memory: 64 columns of 128 rows, pitch 136
constexpr int TM_TPITCH = 136;

// 16 warps: warp w reads TMEM lanes 32 (w % 4) .. (its rows) and the
// columns 16 (w / 4) .. +16 of the tile.
constexpr int TM_THREADS = 512;
template <int EPI>
__global__ void __launch_bounds__(TM_THREADS, 2) gemm_tma_kernel(const __grid_constant__ CUtensorMap tmA,
                                                            const __grid_constant__ CUtensorMap tmB, int M, int N,
                                                            int K, int kc, float* __restrict__ C, int64_t ldc,
                                                            int64_t c_split, GemmEpilogue ep, int* __restrict__ status,
                                                            const __grid_constant__ CUtensorMap tmZ,
                                                            const __grid_constant__ CUtensorMap tmH, int tstore) {
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    __shared__ uint64_t full[TC_STAGES], empty[TC_STAGES], done;
    __shared__ uint32_t tmem_slot;
    static_assert(3 * (TC_BM * 128) + TM_BN * TM_TPITCH * 2 <= TC_STAGES * (TC_TILE + TM_TILE_B) &&
                      TC_BM * (TM_BN + 1) * 4 <= 3 * (TC_BM * 128),
                  "the epilogue's tiles fit into the stage buffers");
    // 1024-byte aligned stage buffers (the swizzle pattern repeats every
    // 1024 bytes and the descriptors assume it starts at the buffer)
    uint8_t* base = tc_smem + ((1024u - (smem_u32(tc_smem) & 1023u)) & 1023u);
    uint8_t* sA0 = base;
    uint8_t* sB0 = base + TC_STAGES * TC_TILE;
    const int m0 = blockIdx.y * TC_BM, n0 = blockIdx.x * TM_BN;
    const int kb = blockIdx.z * kc, ke = min(K, kb + kc);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_slot)),
                     "r"(TM_BN)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (threadIdx.x == 0) {
        for (int i = 0; i < TC_STAGES; i++) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const int nk = ke > kb ? (ke - kb + TC_BK - 1) / TC_BK : 0;
    bool ok = true;
    if (threadIdx.x == 0 && nk > 0) {
        auto load = [&](int j) {
            const int st = j % TC_STAGES;
            mbar_expect_tx(&full[st], static_cast<uint32_t>(TC_TILE + TM_TILE_B));
            const uint32_t a = smem_u32(sA0 + st * TC_TILE), b = smem_u32(sB0 + st * TM_TILE_B);
            const int k0 = kb + j * TC_BK;
            tma_load_2d(a, &tmA, k0, m0, &full[st]);
            tma_load_2d(b, &tmB, k0, n0, &full[st]);
        };
        for (int j = 0; j < TC_STAGES && j < nk; j++) load(j);
        for (int it = 0; it < nk; it++) {
            const int st = it % TC_STAGES;
            const unsigned ph = (it / TC_STAGES) & 1;
            if (!mbar_wait(&full[st], ph)) ok = false;
            tc_fence_after();
            const uint32_t a0 = smem_u32(sA0 + st * TC_TILE), b0 = smem_u32(sB0 + st * TM_TILE_B);
#pragma unroll
            for (int k = 0; k < TC_BK / 16; k++) {
                const uint64_t ad = tm_desc(a0 + k * 32);
                const uint64_t bd = tm_desc(b0 + k * 32);
                const uint32_t acc = (it > 0 || k > 0) ? 1u : 0u;
                asm volatile(
                    "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
                    " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n}\n" ::"r"(tmem),
                    "l"(ad), "l"(bd), "r"(TM_IDESC), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u)
                    : "memory");
            }
            // The last commit goes to a barrier of its own.  The warps that wait
            // for the accumulator have not followed the stage's phases: on
            // empty[st] a second use (K > 256) is the parity that an unused
            // barrier already passes.
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                             smem_u32(it + 1 < nk ? &empty[st] : &done))
                         : "memory");
            if (it + TC_STAGES < nk) {
                // the stage is free once its MMAs have read it
                if (!mbar_wait(&empty[st], ph)) ok = false;
                load(it + TC_STAGES);
            }
        }
    }
    __syncwarp();
    if (nk > 0 && !mbar_wait(&done, 0)) ok = false;
    tc_fence_after();
    const int wl = warp & 3, wc = warp >> 2;
    const int64_t row = m0 + wl * 32 + lane;
    {
        const int c0 = wc * 16;
        uint32_t v[16];
        if (nk > 0) {
            const uint32_t taddr = tmem + (static_cast<uint32_t>(wl * 32) << 16) + static_cast<uint32_t>(c0);
            asm volatile(
                "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, "
                "[%16];\n"
                : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                  "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                  "=r"(v[15])
                : "r"(taddr));
            asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
        } else {
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] = 0u;
        }
        const int col0 = n0 + c0;
        if (EPI == 1 && tstore) {
            // Z and H of the tile into shared memory in the 128-byte-swizzled
            // layout of the output tensor maps (16-byte chunk c of tile row r
            // at r * 128 + ((c ^ (r & 7)) << 4), so the 8 rows of one store
            // phase fall on 8 different bank groups): Z as two boxes of 32
            // columns, H as one of 64; thread 0 stores them with the TMA
            // below.  The stage buffers are free: the last commit covered
            // every MMA, and every load had landed before its MMA.
            float bv[16];
            const float* bp = ep.bias + col0;
            if (col0 + 16 <= N && (reinterpret_cast<uintptr_t>(bp) & 15) == 0) {
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    const float4 q = __ldg(reinterpret_cast<const float4*>(bp + j));
                    bv[j] = q.x;
                    bv[j + 1] = q.y;
                    bv[j + 2] = q.z;
                    bv[j + 3] = q.w;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 16; j++) bv[j] = col0 + j < N ? bp[j] : 0.f;
            }
            float z[16], h[16];
#pragma unroll
            for (int j = 0; j < 16; j++) {
                z[j] = __uint_as_float(v[j]) + bv[j];
                h[j] = ep.act ? gelu(z[j]) : z[j];
            }
            const int r = wl * 32 + lane;
            const uint32_t sw = static_cast<uint32_t>(r & 7);
            uint8_t* zrow = base + (wc >> 1) * (TC_BM * 128) + r * 128;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t ch = static_cast<uint32_t>(4 * (wc & 1) + q);
                *reinterpret_cast<float4*>(zrow + ((ch ^ sw) << 4)) =
                    make_float4(z[4 * q], z[4 * q + 1], z[4 * q + 2], z[4 * q + 3]);
            }
            uint8_t* hrow = base + 2 * (TC_BM * 128) + r * 128;
#pragma unroll
            for (int q = 0; q < 2; q++) {
                __align__(16) __nv_bfloat16 hb[8];
#pragma unroll
                for (int j = 0; j < 8; j++) hb[j] = __float2bfloat16(h[8 * q + j]);
                const uint32_t ch = static_cast<uint32_t>(2 * wc + q);
                *reinterpret_cast<uint4*>(hrow + ((ch ^ sw) << 4)) = *reinterpret_cast<const uint4*>(hb);
            }
            // the generic-proxy writes, visible to the bulk copies
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
            if (ep.HT) {
                __nv_bfloat16* tt = reinterpret_cast<__nv_bfloat16*>(base + 3 * (TC_BM * 128));
#pragma unroll
                for (int j = 0; j < 16; j++) tt[(c0 + j) * TM_TPITCH + r] = __float2bfloat16(h[j]);
            }
        } else if (EPI == 2) {
            const int r = wl * 32 + lane;
            float* sd = reinterpret_cast<float*>(base);
            __nv_bfloat16* tt = reinterpret_cast<__nv_bfloat16*>(base + 3 * (TC_BM * 128));
            float z[16];
            const float* zp = ep.Zin + row * N + col0;
            if (row < M && col0 + 16 <= N) {
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    const float4 q = __ldg(reinterpret_cast<const float4*>(zp + j));
                    z[j] = q.x;
                    z[j + 1] = q.y;
                    z[j + 2] = q.z;
                    z[j + 3] = q.w;
                }
            } else {
#pragma unroll
                for (int j = 0; j < 16; j++) z[j] = row < M && col0 + j < N ? zp[j] : 0.f;
            }
            __align__(16) __nv_bfloat16 hb[16];
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const float dz = __uint_as_float(v[j]) * gelu_grad(z[j]);
                sd[r * (TM_BN + 1) + c0 + j] = dz;
                hb[j] = __float2bfloat16(dz);
                tt[(c0 + j) * TM_TPITCH + r] = hb[j];
            }
            if (row < M) {
                __nv_bfloat16* hp = ep.H + row * N + col0;
#pragma unroll
                for (int q = 0; q < 2; q++)
                    if (col0 + 8 * q + 8 <= N) *reinterpret_cast<uint4*>(hp + 8 * q) = *reinterpret_cast<uint4*>(hb + 8 * q);
            }
        } else if (row >= M) {
        } else if (EPI == 0) {
            float* dst = C + blockIdx.z * c_split + row * ldc + col0;
            if (col0 + 16 <= N && (reinterpret_cast<uintptr_t>(dst) & 15) == 0) {
#pragma unroll
                for (int j = 0; j < 16; j += 4)
                    *reinterpret_cast<float4*>(dst + j) = make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]),
                                                                      __uint_as_float(v[j + 2]), __uint_as_float(v[j + 3]));
            } else {
#pragma unroll
                for (int j = 0; j < 16; j++)
                    if (col0 + j < N) dst[j] = __uint_as_float(v[j]);
            }
        } else {
            float z[16], h[16];
#pragma unroll
            for (int j = 0; j < 16; j++) {
                z[j] = col0 + j < N ? __uint_as_float(v[j]) + ep.bias[col0 + j] : 0.f;
                h[j] = ep.act ? gelu(z[j]) : z[j];
            }
            const int64_t o = row * N + col0;
            const bool full16 = col0 + 16 <= N && (N & 7) == 0;
            if (ep.Z) {
                if (full16 && (N & 3) == 0) {
#pragma unroll
                    for (int j = 0; j < 16; j += 4)
                        *reinterpret_cast<float4*>(ep.Z + o + j) = make_float4(z[j], z[j + 1], z[j + 2], z[j + 3]);
                } else {
                    for (int j = 0; j < 16; j++)
                        if (col0 + j < N) ep.Z[o + j] = z[j];
                }
            }
            if (ep.Hf) {
                for (int j = 0; j < 16; j++)
                    if (col0 + j < N) ep.Hf[o + j] = h[j];
            }
            if (ep.H) {
                if (full16) {
                    __align__(16) __nv_bfloat16 hb[16];
#pragma unroll
                    for (int j = 0; j < 16; j++) hb[j] = __float2bfloat16(h[j]);
                    *reinterpret_cast<uint4*>(ep.H + o) = *reinterpret_cast<const uint4*>(hb);
                    *reinterpret_cast<uint4*>(ep.H + o + 8) = *reinterpret_cast<const uint4*>(hb + 8);
                } else {
                    for (int j = 0; j < 16; j++)
                        if (col0 + j < N) ep.H[o + j] = __float2bfloat16(h[j]);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TM_BN) : "memory");
    }
    if ((EPI == 1 && tstore && ep.HT) || EPI == 2) {
        // the transposed tile, 16 bytes (8 rows) a thread and pass
        const __nv_bfloat16* tt = reinterpret_cast<const __nv_bfloat16*>(base + 3 * (TC_BM * 128));
        for (int i = threadIdx.x; i < TM_BN * (TC_BM / 8); i += TM_THREADS) {
            const int c = i >> 4, r = (i & 15) * 8;
            if (n0 + c < N && m0 + r < ep.ldt)
                *reinterpret_cast<uint4*>(ep.HT + static_cast<int64_t>(n0 + c) * ep.ldt + m0 + r) =
                    *reinterpret_cast<const uint4*>(tt + c * TM_TPITCH + r);
        }
    }
    if (EPI == 2 && threadIdx.x < TM_BN && n0 + static_cast<int>(threadIdx.x) < N) {
        const float* sd = reinterpret_cast<const float*>(base) + threadIdx.x;
        const int nr = min(TC_BM, M - m0);
        float sum = 0.f;
#pragma unroll 8
        for (int r = 0; r < nr; r++) sum += sd[r * (TM_BN + 1)];
        ep.colpart[static_cast<int64_t>(blockIdx.y) * N + n0 + threadIdx.x] = sum;
    }
    if (EPI == 1 && tstore && threadIdx.x == 0) {
        // x = n0 and n0 + 32: multiples of 32 columns, 128-byte aligned
        tma_store_2d(&tmZ, smem_u32(base), n0, m0);
        if (n0 + 32 < N) tma_store_2d(&tmZ, smem_u32(base + TC_BM * 128), n0 + 32, m0);
        tma_store_2d(&tmH, smem_u32(base + 2 * TC_BM * 128), n0, m0);
        asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
        // the shared memory stays allocated until the copies are complete
        asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");
    }
    if (!ok) atomicOr(status, 1);
}

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
    return z ^ (z >> 31);
}

// One row of the network input from raw input row x (n_in floats) by kRowThreads
// threads (t = 0..): x, then per frequency f < nf sin(2^f pi s), cos(2^f pi s)
// for s = x[n_in-2] and for s = x[n_in-1], then zeros up to ld.  ht (may be
// null): the same values down column r of rows of ldt.
constexpr int kRowThreads = 16;
__device__ __forceinline__ void write_features(const float* __restrict__ x, int n_in, int nf, int ld, int t,
                                               __nv_bfloat16* __restrict__ out, __nv_bfloat16* __restrict__ ht,
                                               int64_t ldt) {
    const int in_w = n_in + 4 * nf;
    auto put = [&](int j, float v) {
        const __nv_bfloat16 b = __float2bfloat16(v);
        out[j] = b;
        if (ht && j < in_w) ht[j * ldt] = b;
    };
    for (int j = t; j < n_in; j += kRowThreads) put(j, x[j]);
    for (int i = t; i < 2 * nf; i += kRowThreads) {
        const int c = i >= nf ? 1 : 0, f = i - c * nf;
        const float w = ldexpf(3.14159265358979f, f);  // doubled f times: exact
        float sn, cs;
        sincosf(w * x[n_in - 2 + c], &sn, &cs);
        put(n_in + 2 * i, sn);
        put(n_in + 2 * i + 1, cs);
    }
    for (int j = in_w + t; j < ld; j += kRowThreads) put(j, 0.f);
}

__global__ void __launch_bounds__(128) features_kernel(int64_t M, int n_in, int nf, int ld,
                                                       const float* __restrict__ x, __nv_bfloat16* __restrict__ h) {
    const int64_t r = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / kRowThreads;
    if (r >= M) return;
    write_features(x + r * n_in, n_in, nf, ld, threadIdx.x % kRowThreads, h + r * ld, nullptr, 0);
}

// What changes from one training step to the next; the steps of a call read
// entry *at of an array, so that one captured graph serves every step.
// loss_kernel moves *at on once the batch is drawn; grad_adam_kernel, later in
// the step, reads the entry before it.
struct StepArgs {
    uint64_t key;
    float lr, c1, c2;
    int pad;
};

// ht (may be null): the transposed inputs, rows of ldt.  One thread per row
// took 11.4 us for 8192 rows (64 blocks, 12 sincosf in a row), 5.7 here.
__global__ void __launch_bounds__(128) gather_kernel(int M, int64_t n_rows, int n_in, int nf, int ld, int n_out,
                                                     const float* __restrict__ X, const float* __restrict__ T,
                                                     const StepArgs* __restrict__ args,
                                                     const int* __restrict__ at, __nv_bfloat16* __restrict__ h,
                                                     float* __restrict__ tb, __nv_bfloat16* __restrict__ ht,
                                                     int64_t ldt) {
    const int r = (blockIdx.x * blockDim.x + threadIdx.x) / kRowThreads, t = threadIdx.x % kRowThreads;
    if (r >= M) return;
    const uint64_t key = args[*at].key;
    const int64_t src = static_cast<int64_t>(mix64(key + static_cast<uint64_t>(r) * 0x9E3779B97F4A7C15ULL) %
                                             static_cast<uint64_t>(n_rows));
    write_features(X + src * n_in, n_in, nf, ld, t, h + static_cast<int64_t>(r) * ld, ht ? ht + r : nullptr, ldt);
    for (int j = t; j < n_out; j += kRowThreads) tb[static_cast<int64_t>(r) * n_out + j] = T[src * n_out + j];
}

__global__ void bias_act_kernel(int M, int N, const float* __restrict__ C, const float* __restrict__ bias,
                                float* __restrict__ Z, __nv_bfloat16* __restrict__ H, float* __restrict__ Hf, int act) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= static_cast<int64_t>(M) * N) return;
    const float z = C[i] + bias[i % N];
    if (Z) Z[i] = z;
    const float h = act ? gelu(z) : z;
    if (H) H[i] = __float2bfloat16(h);
    if (Hf) Hf[i] = h;
}

__global__ void act_bwd_kernel(int64_t n, const float* __restrict__ dH, const float* __restrict__ Z,
                               float* __restrict__ dZ, __nv_bfloat16* __restrict__ dZb, int act) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float d = act ? dH[i] * gelu_grad(Z[i]) : dH[i];
    dZ[i] = d;
    dZb[i] = __float2bfloat16(d);
}

// column sums of an M x N matrix: per chunk of kColRows rows, then the
// chunks in order
constexpr int kColRows = 128;
__global__ void col_sum_partial_kernel(int M, int N, const float* __restrict__ X, float* __restrict__ part) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= N) return;
    const int r0 = blockIdx.y * kColRows, r1 = min(M, r0 + kColRows);
    float s = 0.f;
    for (int r = r0; r < r1; r++) s += X[static_cast<int64_t>(r) * N + c];
    part[static_cast<int64_t>(blockIdx.y) * N + c] = s;
}
__global__ void col_sum_final_kernel(int chunks, int N, const float* __restrict__ part, float* __restrict__ out) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= N) return;
    float s = 0.f;
    for (int k = 0; k < chunks; k++) s += part[static_cast<int64_t>(k) * N + c];
    out[c] = s;
}

__global__ void mse_kernel(int M, int N, const float* __restrict__ Y, const float* __restrict__ T,
                           float* __restrict__ dY, float* __restrict__ row_err) {
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= M) return;
    const float scale = 2.f / (static_cast<float>(M) * N);
    float e = 0.f;
    for (int c = 0; c < N; c++) {
        const float d = Y[static_cast<int64_t>(r) * N + c] - T[static_cast<int64_t>(r) * N + c];
        e += d * d;
        dY[static_cast<int64_t>(r) * N + c] = scale * d;
    }
    row_err[r] = e;
}

// one block of 256 threads: strided partial sums, then a fixed tree; into
// out[0], or with `at` (see StepArgs) into out[*at], which it moves on
__global__ void loss_kernel(int M, int N, const float* __restrict__ row_err, float* __restrict__ out,
                            int* __restrict__ at) {
    __shared__ double s[256];
    double a = 0.0;
    for (int r = threadIdx.x; r < M; r += 256) a += row_err[r];
    s[threadIdx.x] = a;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const float l = static_cast<float>(s[0] / (static_cast<double>(M) * N));
        if (at) out[(*at)++] = l;
        else *out = l;
    }
}

// One layer as grad_adam_kernel reads it.
struct LayerGrad {
    int64_t w_off, b_off, part_off;  // part_off: its S x (dout * din) weight partials
    int din, dout, ld_in, ld_t;      // row strides of the padded W (layer 0) and of W^T
    int64_t col_off;                 // its chunks x dout column sums
    __nv_bfloat16* wpad;             // layer 0: W with rows of ld_in (or null)
    __nv_bfloat16* wt;               // W^T, din rows of ld_t (null for layer 0)
};

__global__ void adam_kernel(int64_t n, float* __restrict__ w, const float* __restrict__ gr, float* __restrict__ m,
                            float* __restrict__ v, float lr, float b1, float b2, float eps, float c1, float c2,
                            __nv_bfloat16* __restrict__ wb, LayerGrad first) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float g = gr[i];
    const float mi = b1 * m[i] + (1.f - b1) * g;
    const float vi = b2 * v[i] + (1.f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    const __nv_bfloat16 h = __float2bfloat16(wi);
    wb[i] = h;
    // the first layer's padded copy (its weights come first)
    if (i < static_cast<int64_t>(first.din) * first.dout) {
        const int k = static_cast<int>(i), o = k / first.din;
        first.wpad[static_cast<int64_t>(o) * first.ld_in + (k - o * first.din)] = h;
    }
}

// The last layer's dZ = dY of kColRows rows per block: bf16 rows of ld (zeros
// beyond N) and their transpose, column sums of the block row by row, squared
// error per row.  N <= kMseCols.
constexpr int kMseCols = 32;
__global__ void __launch_bounds__(kColRows) mse_grad_kernel(int M, int N, int ld, const float* __restrict__ Y,
                                                            const float* __restrict__ T,
                                                            __nv_bfloat16* __restrict__ dz,
                                                            __nv_bfloat16* __restrict__ dzt, int64_t ldt,
                                                            float* __restrict__ colpart, float* __restrict__ row_err) {
    __shared__ float sd[kColRows][kMseCols + 1];
    const int r = blockIdx.x * kColRows + threadIdx.x;
    const float scale = 2.f / (static_cast<float>(M) * N);
    if (r < M) {
        float e = 0.f;
        for (int c = 0; c < N; c++) {
            const float d = Y[static_cast<int64_t>(r) * N + c] - T[static_cast<int64_t>(r) * N + c];
            e += d * d;
            const float g = scale * d;
            sd[threadIdx.x][c] = g;
            const __nv_bfloat16 h = __float2bfloat16(g);
            dz[static_cast<int64_t>(r) * ld + c] = h;
            dzt[c * ldt + r] = h;
        }
        for (int c = N; c < ld; c++) dz[static_cast<int64_t>(r) * ld + c] = __float2bfloat16(0.f);
        row_err[r] = e;
    }
    __syncthreads();
    if (threadIdx.x < N) {
        const int nr = min(kColRows, M - static_cast<int>(blockIdx.x) * kColRows);
        float sum = 0.f;
#pragma unroll 8
        for (int i = 0; i < nr; i++) sum += sd[i][threadIdx.x];
        colpart[static_cast<int64_t>(blockIdx.x) * N + threadIdx.x] = sum;
    }
}

// The gradients of layer blockIdx.y (weights: the S split partial sums in
// order; bias: the chunks' column sums in order) into g, then, given args, the
// Adam step and the bf16 copies.
__global__ void __launch_bounds__(256) grad_adam_kernel(const LayerGrad* __restrict__ layers, int S, int chunks,
                                                        const float* __restrict__ part,
                                                        const float* __restrict__ colpart, float* __restrict__ g,
                                                        const StepArgs* __restrict__ args,
                                                        const int* __restrict__ at, float* __restrict__ w,
                                                        float* __restrict__ m, float* __restrict__ v, float b1, float b2,
                                                        float eps, __nv_bfloat16* __restrict__ wb,
                                                        const int* __restrict__ status, float* __restrict__ loss) {
    const LayerGrad L = layers[blockIdx.y];
    const int64_t wn = static_cast<int64_t>(L.din) * L.dout;
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    // the GEMM status word behind the loss just written, so that one copy
    // brings both (every GEMM of the step is done by now)
    if (i == 0 && blockIdx.y == 0) reinterpret_cast<int*>(loss)[at ? *at : 1] = *status;
    if (i >= wn + L.dout) return;
    const bool weight = i < wn;
    const float* p = weight ? part + L.part_off + i : colpart + L.col_off + (i - wn);
    const int64_t step = weight ? wn : L.dout;
    const int n = weight ? S : chunks;
    float gr = 0.f;
    int z = 0;
    for (; z + 16 <= n; z += 16) {  // sixteen loads in flight, added in order
        float e[16];
#pragma unroll
        for (int q = 0; q < 16; q++) e[q] = __ldcs(p + (z + q) * step);
#pragma unroll
        for (int q = 0; q < 16; q++) gr += e[q];
    }
    for (; z < n; z++) gr += p[z * step];
    const int64_t k = weight ? L.w_off + i : L.b_off + (i - wn);
    g[k] = gr;
    if (!args) return;
    const StepArgs a = args[*at - 1];
    const float lr = a.lr, c1 = a.c1, c2 = a.c2;
    const float mi = b1 * m[k] + (1.f - b1) * gr;
    const float vi = b2 * v[k] + (1.f - b2) * gr * gr;
    m[k] = mi;
    v[k] = vi;
    const float wi = w[k] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[k] = wi;
    const __nv_bfloat16 h = __float2bfloat16(wi);
    wb[k] = h;
    if (weight) {
        const int o = static_cast<int>(i / L.din), q = static_cast<int>(i - static_cast<int64_t>(o) * L.din);
        if (L.wpad) L.wpad[static_cast<int64_t>(o) * L.ld_in + q] = h;
        if (L.wt) L.wt[static_cast<int64_t>(q) * L.ld_t + o] = h;
    }
}
// the padded W of layer 0 and the W^T of the others from the bf16 weights
__global__ void weight_copies_kernel(const LayerGrad* __restrict__ layers, const __nv_bfloat16* __restrict__ wb) {
    const LayerGrad L = layers[blockIdx.y];
    const int64_t wn = static_cast<int64_t>(L.din) * L.dout;
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= wn) return;
    const int o = static_cast<int>(i / L.din), q = static_cast<int>(i - static_cast<int64_t>(o) * L.din);
    if (L.wpad) L.wpad[static_cast<int64_t>(o) * L.ld_in + q] = wb[L.w_off + i];
    if (L.wt) L.wt[static_cast<int64_t>(q) * L.ld_t + o] = wb[L.w_off + i];
}

__global__ void to_bf16_kernel(int64_t n, const float* __restrict__ x, __nv_bfloat16* __restrict__ y) {
    const int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __float2bfloat16(x[i]);
}

inline unsigned blocks(int64_t n, int t) { return static_cast<unsigned>((n + t - 1) / t); }

struct Buf {
    void* p = nullptr;
    size_t bytes = 0;
    Buf() = default;
    Buf(const Buf&) = delete;
    Buf& operator=(const Buf&) = delete;
    Buf(Buf&& o) noexcept : p(o.p), bytes(o.bytes) { o.p = nullptr; }
    ~Buf() {
        if (p) cudaFree(p);
    }
    bool alloc(size_t n) {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = n;
        return cudaMalloc(&p, n ? n : 16) == cudaSuccess;
    }
    template <typename T>
    T* as() const {
        return static_cast<T*>(p);
    }
};

inline bool vec_ok(const void* p, int64_t ld) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0 && ld % 8 == 0; }

// status word of the tensor-core GEMM (bit 0: an mbarrier wait expired)
__device__ int g_gemm_status = 0;

template <bool AV, bool BV>
void launch_tc(dim3 grid, int M, int N, int K, int kc, const __nv_bfloat16* A, int64_t lda, const __nv_bfloat16* B,
               int64_t ldb, float* C, int64_t ldc, int64_t c_split, cudaStream_t s) {
    // the shared-memory opt-in is a per-device attribute of the kernel
    static bool attr[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr[dev]) {
        cudaFuncSetAttribute(gemm_tc_kernel<AV, BV>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM);
        if (dev >= 0 && dev < 64) attr[dev] = true;
    }
    int* st = nullptr;
    cudaGetSymbolAddress(reinterpret_cast<void**>(&st), g_gemm_status);
    gemm_tc_kernel<AV, BV><<<grid, TC_THREADS, TC_SMEM, s>>>(M, N, K, kc, A, lda, B, ldb, C, ldc, c_split, st);
}

// cuTensorMapEncodeTiled, looked up in the driver once (no link against the
// driver library); null where the driver does not offer it
using TensorMapEncode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                     const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                     CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
TensorMapEncode tensor_map_encoder() {
    static TensorMapEncode fn = nullptr;
    static bool looked = false;
    if (!looked) {
        looked = true;
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<TensorMapEncode>(f);
        else
            cudaGetLastError();
    }
    return fn;
}

// The tensor map of a k-contiguous bf16 operand of `rows` rows of `ld`
// elements, K of them used: boxes of 64 k (128 bytes) x box_rows rows with
// the 128-byte swizzle, zero fill outside.
bool operand_map(CUtensorMap* map, const __nv_bfloat16* X, int64_t ld, int rows, int K, int box_rows) {
    const TensorMapEncode enc = tensor_map_encoder();
    if (!enc || rows <= 0 || K <= 0) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(ld) * 2};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(TC_BK), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(X), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The tensor map of a row-major output [rows][N] (fp32 or bf16) for the
// TMA stores of the fused epilogue: boxes of 128 bytes of a row (32 fp32 or
// 64 bf16) x 128 rows, 128-byte swizzle.
bool output_map(CUtensorMap* map, void* X, bool f32, int rows, int N) {
    const TensorMapEncode enc = tensor_map_encoder();
    if (!enc || rows <= 0 || N <= 0) return false;
    const int es = f32 ? 4 : 2;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(N), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(N) * es};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(128 / es), static_cast<cuuint32_t>(TC_BM)};
    const cuuint32_t estr[2] = {1, 1};
    return enc(map, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, X, dims, strides, box,
               estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// address of the GEMM status word on the current device (looked up once)
int* gemm_status_ptr() {
    static int* addr[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64) dev = 0;
    if (!addr[dev]) cudaGetSymbolAddress(reinterpret_cast<void**>(&addr[dev]), g_gemm_status);
    return addr[dev];
}

// The TMA GEMM; false (nothing launched) where an operand cannot be
// described by a tensor map (rows not 16-byte aligned) or the driver offers
// no encoder: the caller then uses gemm_tc_kernel.
template <int EPI>
bool launch_tma(dim3 grid, int M, int N, int K, int kc, const __nv_bfloat16* A, int64_t lda, const __nv_bfloat16* B,
                int64_t ldb, float* C, int64_t ldc, int64_t c_split, const GemmEpilogue& ep, cudaStream_t s) {
    if (!vec_ok(A, lda) || !vec_ok(B, ldb)) return false;
    CUtensorMap ma, mb;
    if (!operand_map(&ma, A, lda, M, K, TC_BM) || !operand_map(&mb, B, ldb, N, K, TM_BN)) return false;
    grid.x = blocks(N, TM_BN);
    static bool attr[64] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 0 || dev >= 64 || !attr[dev]) {
        cudaFuncSetAttribute(gemm_tma_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, TM_SMEM);
        if (dev >= 0 && dev < 64) attr[dev] = true;
    }
    // the fused epilogue of a hidden layer (Z and H, no fp32 activation)
    // leaves the tile through shared memory and the TMA where both outputs
    // can be described by tensor maps (16-byte aligned rows)
    CUtensorMap mz{}, mh{};
    const bool tstore = EPI == 1 && ep.Z && ep.H && !ep.Hf && N % 8 == 0 &&
                        (reinterpret_cast<uintptr_t>(ep.Z) & 15) == 0 && (reinterpret_cast<uintptr_t>(ep.H) & 15) == 0 &&
                        output_map(&mz, ep.Z, true, M, N) && output_map(&mh, ep.H, false, M, N);
    gemm_tma_kernel<EPI><<<grid, TM_THREADS, TM_SMEM, s>>>(ma, mb, M, N, K, kc, C, ldc, c_split, ep,
                                                           gemm_status_ptr(), mz, mh, tstore ? 1 : 0);
    return true;
}

// C = A . B^T with A [M][lda], B [N][ldb] (k contiguous); see gemm_tc_kernel
void gemm(int M, int N, int K, const __nv_bfloat16* A, int64_t lda, const __nv_bfloat16* B, int64_t ldb, float* C,
          int64_t ldc, cudaStream_t s, int splits = 1, int64_t c_split = 0) {
    if (M <= 0 || N <= 0) return;
    const int kc = tc_split_len(K, splits);
    dim3 grid(blocks(N, TC_BN), blocks(M, TC_BM), split_count(K, kc));
    if (launch_tma<0>(grid, M, N, K, kc, A, lda, B, ldb, C, ldc, c_split, GemmEpilogue{}, s)) return;
    const bool av = vec_ok(A, lda), bv = vec_ok(B, ldb);
    if (av && bv)
        launch_tc<true, true>(grid, M, N, K, kc, A, lda, B, ldb, C, ldc, c_split, s);
    else if (av)
        launch_tc<true, false>(grid, M, N, K, kc, A, lda, B, ldb, C, ldc, c_split, s);
    else if (bv)
        launch_tc<false, true>(grid, M, N, K, kc, A, lda, B, ldb, C, ldc, c_split, s);
    else
        launch_tc<false, false>(grid, M, N, K, kc, A, lda, B, ldb, C, ldc, c_split, s);
}

// enqueues the read of the GEMM status word before the call's own
// synchronisation
void gemm_status_fetch(int* to, cudaStream_t s) {
    cudaMemcpyAsync(to, gemm_status_ptr(), sizeof(int), cudaMemcpyDeviceToHost, s);
}
// reads and clears the GEMM status word (after a synchronisation)
bool gemm_status_ok() {
    int v = 0;
    cudaMemcpyFromSymbol(&v, g_gemm_status, sizeof(int));
    if (v) {
        const int zero = 0;
        cudaMemcpyToSymbol(g_gemm_status, &zero, sizeof(int));
    }
    return v == 0;
}

inline int64_t pad8(int64_t n) { return (n + 7) / 8 * 8; }

void transpose(int R, int Cc, const __nv_bfloat16* in, int64_t ldin, __nv_bfloat16* out, int64_t ldout,
               cudaStream_t s) {
    if (R <= 0 || Cc <= 0) return;
    transpose_bf16_kernel<<<dim3(blocks(Cc, 32), blocks(R, 32)), dim3(32, 8), 0, s>>>(R, Cc, in, ldin, out, ldout);
}

}  // namespace

struct gelios_mlp {
    int device = 0;
    cudaStream_t stream = nullptr;
    int n_in = 0, nf = 0, width = 0, depth = 0, n_out = 0, max_batch = 0;
    int in_w = 0;  // width of the first layer's input (raw inputs + 4 nf features)
    std::vector<int> din, dout;
    std::vector<int64_t> w_off, b_off;
    int64_t n_params = 0;
    int step = 0;
    Buf w32, g32, m, v, wb;
    std::vector<Buf> h;  // bf16 inputs of every layer [max_batch][din]
    std::vector<Buf> z;  // fp32 pre-activations of every hidden layer
    Buf c, y, dzb, tb, rowerr, loss, xin;
    int ld0 = 0;      // row stride of the first layer's input and of wpad (in_w rounded up to 8: TMA rows)
    Buf wpad;         // bf16 W of the first layer, rows of ld0
    // what a gradient needs, one allocation at its first use (ensure_training)
    bool fused = false, training_known = false;
    Buf train_mem;
    // fused: per layer H^T and dZ^T, W^T, gradient partials
    __nv_bfloat16 *f_ht = nullptr, *f_dzt = nullptr, *f_dzb2 = nullptr;
    float *f_part = nullptr, *f_col = nullptr;
    // separate kernels: dH and dZ of a layer, partials, transposes W_l^T, dZ^T, H_l^T
    float *dh = nullptr, *dz = nullptr, *part = nullptr, *colpart = nullptr;
    __nv_bfloat16 *wt = nullptr, *dzt = nullptr, *ht = nullptr;
    Buf f_layers;
    std::vector<LayerGrad> layers_host;
    cudaStream_t side = nullptr;
    cudaEvent_t ev_dz = nullptr, ev_side = nullptr;
    // steps of a training call: their StepArgs, losses and the step counter,
    // kept from call to call (they grow with the longest call)
    Buf args, hist, at;
    int64_t steps_cap = 0;
    cudaGraphExec_t graph = nullptr;  // one fused step of graph_batch rows
    int graph_batch = 0;
    void drop_graph() {
        if (graph) cudaGraphExecDestroy(graph);
        graph = nullptr;
    }
    // gelios_mlp_predict: rows of a chunk; once it is worth it (staging_worth)
    // one pinned allocation: a copy of the GEMM status word, then two chunks'
    // inputs and outputs
    int64_t chunk_rows = 0, predictions = 0, io_bytes = 0;
    int* stage = nullptr;
    bool stage_failed = false;
    float *px[2] = {nullptr, nullptr}, *py[2] = {nullptr, nullptr};
    cudaEvent_t ev_chunk[2] = {nullptr, nullptr};
    Buf X, T;  // training set (fp32 rows)
    int64_t n_rows = 0;
    ~gelios_mlp() {
        if (side) cudaStreamDestroy(side);
        if (stream) cudaStreamDestroy(stream);
        if (ev_dz) cudaEventDestroy(ev_dz);
        if (ev_side) cudaEventDestroy(ev_side);
        if (stage) cudaFreeHost(stage);
        drop_graph();
        for (int k = 0; k < 2; k++)
            if (ev_chunk[k]) cudaEventDestroy(ev_chunk[k]);
    }
    int layers() const { return depth + 1; }
    // H_l^T (din[l] rows) and dZ_l^T (dout[l] rows), max_batch rounded up to 8 apart
    __nv_bfloat16* ht_of(int l) const {
        return f_ht + (l == 0 ? 0 : pad8(max_batch) * (in_w + static_cast<int64_t>(l - 1) * width));
    }
    __nv_bfloat16* dzt_of(int l) const { return f_dzt + pad8(max_batch) * width * l; }
};

namespace {
int fail(const char* what) {
    gelios::set_error(what);
    return GELIOS_E_ARG;
}
int cuda_fail(cudaError_t e) {
    gelios::set_error(std::string("CUDA: ") + cudaGetErrorString(e));
    return GELIOS_E_CUDA;
}
#define MLP_TRY(x)                                   \
    do {                                             \
        cudaError_t e_ = (x);                        \
        if (e_ != cudaSuccess) return cuda_fail(e_); \
    } while (0)

// forward pass of M rows whose network inputs are in h[0]; output in y.
// train: the hidden layers' H^T as well (f_ht, rows of pad8(M)).
void forward(gelios_mlp* n, int M, bool train = false) {
    cudaStream_t s = n->stream;
    const __nv_bfloat16* wb = n->wb.as<__nv_bfloat16>();
    for (int l = 0; l < n->layers(); l++) {
        const int di = n->din[l], dO = n->dout[l];
        const bool last = l == n->layers() - 1;
        GemmEpilogue ep;
        ep.bias = n->w32.as<float>() + n->b_off[l];
        ep.Z = last ? nullptr : n->z[l].as<float>();
        ep.H = last ? nullptr : n->h[l + 1].as<__nv_bfloat16>();
        ep.Hf = last ? n->y.as<float>() : nullptr;
        ep.act = last ? 0 : 1;
        if (train && !last) {
            ep.ldt = pad8(M);
            ep.HT = n->ht_of(l + 1);
        }
        // bias and activation applied as the accumulator leaves tensor memory
        // (TMA path), or by bias_act_kernel after the GEMM
        const __nv_bfloat16* A = n->h[l].as<__nv_bfloat16>();
        const __nv_bfloat16* W = l == 0 ? n->wpad.as<__nv_bfloat16>() : wb + n->w_off[l];
        const int ld = l == 0 ? n->ld0 : di;
        dim3 grid(blocks(dO, TC_BN), blocks(M, TC_BM), 1);
        // (a hidden layer whose rows the TMA cannot store: gemm_tc_kernel and the
        // coalesced bias_act_kernel: a training step of 8192 rows of 100 304 us, 294 so)
        if (M > 0 && (last || dO % 8 == 0) &&
            launch_tma<1>(grid, M, dO, di, tc_split_len(di, 1), A, ld, W, ld, nullptr, 0, 0, ep, s))
            continue;
        gemm(M, dO, di, A, ld, W, ld, n->c.as<float>(), dO, s);
        const int64_t e = static_cast<int64_t>(M) * dO;
        bias_act_kernel<<<blocks(e, 256), 256, 0, s>>>(M, dO, n->c.as<float>(), ep.bias, ep.Z, ep.H, ep.Hf, ep.act);
    }
}

// The backward pass of the fused training step: loss of the batch into
// loss[0]; the gradients' partial sums into f_part and f_col, which
// grad_adam_kernel then adds up.  The data GEMMs run down the layers on the
// main stream, each layer's weight GEMM and the loss beside them on the side
// stream.  Per 8192-row step of the 31 -> 5 x 256 -> 5 network, as ~45
// launches of separate transposes, activations, sums and reductions the
// whole step took 480 us, 189 here;
// as a captured graph (train_graph) 156 (117 of 4096 rows, 100 of 128; the
// slope between calls of 200 and 600 steps).
bool backward_fused(gelios_mlp* n, int M, float* loss, int* at) {
    cudaStream_t s = n->stream, s2 = n->side;
    const int L = n->layers();
    const int64_t Mp = pad8(M);
    const int S = splits_of(M), kc = tc_split_len(M, split_target(M)), chunks = (M + kColRows - 1) / kColRows;
    const int ldo = static_cast<int>(pad8(n->n_out));
    __nv_bfloat16* dz[2] = {n->dzb.as<__nv_bfloat16>(), n->f_dzb2};
    float* col = n->f_col;
    mse_grad_kernel<<<chunks, kColRows, 0, s>>>(M, n->n_out, ldo, n->y.as<float>(), n->tb.as<float>(), dz[0],
                                                n->dzt_of(L - 1), Mp, col + n->layers_host[L - 1].col_off,
                                                n->rowerr.as<float>());
    for (int l = L - 1; l >= 0; l--) {
        const int di = n->din[l], dO = n->dout[l];
        cudaEventRecord(n->ev_dz, s);
        cudaStreamWaitEvent(s2, n->ev_dz, 0);
        if (l == L - 1) loss_kernel<<<1, 256, 0, s2>>>(M, n->n_out, n->rowerr.as<float>(), loss, at);
        // dW[dO][di] = dZ^T . H_l, split over the rows of the batch
        bool ok = launch_tma<0>(dim3(1, blocks(dO, TC_BM), S), dO, di, M, kc, n->dzt_of(l), Mp, n->ht_of(l), Mp,
                                n->f_part + n->layers_host[l].part_off, di, static_cast<int64_t>(dO) * di,
                                GemmEpilogue{}, s2);
        if (!ok) return false;  // an operand without a tensor map (not with the strides gelios_mlp_create chose)
        if (l == 0) break;
        // dZ_{l-1} = (dZ . W_l) * GELU'(Z_{l-1})
        const int b = (L - 1 - l) & 1;
        GemmEpilogue ep;
        ep.Zin = n->z[l - 1].as<float>();
        ep.H = dz[b ^ 1];
        ep.HT = n->dzt_of(l - 1);
        ep.ldt = Mp;
        ep.colpart = col + n->layers_host[l - 1].col_off;
        const int ldz = l == L - 1 ? ldo : dO;
        ok = launch_tma<2>(dim3(1, blocks(M, TC_BM), 1), M, di, dO, tc_split_len(dO, 1), dz[b], ldz,
                           n->layers_host[l].wt, n->layers_host[l].ld_t, nullptr, 0, 0, ep, s);
        if (!ok) return false;
    }
    return cudaEventRecord(n->ev_side, s2) == cudaSuccess && cudaStreamWaitEvent(s, n->ev_side, 0) == cudaSuccess;
}
// the gradients into g32 and, given args, the Adam step (see grad_adam_kernel)
constexpr float kAdamB1 = 0.9f, kAdamB2 = 0.999f, kAdamEps = 1e-8f;
void reduce_fused(gelios_mlp* n, int M, const StepArgs* args, const int* at, float* loss) {
    int64_t most = 0;
    for (int l = 0; l < n->layers(); l++)
        most = std::max(most, static_cast<int64_t>(n->din[l] + 1) * n->dout[l]);
    grad_adam_kernel<<<dim3(blocks(most, 256), n->layers()), 256, 0, n->stream>>>(
        n->f_layers.as<LayerGrad>(), splits_of(M), (M + kColRows - 1) / kColRows, n->f_part,
        n->f_col, n->g32.as<float>(), args, at, n->w32.as<float>(), n->m.as<float>(), n->v.as<float>(),
        kAdamB1, kAdamB2, kAdamEps, n->wb.as<__nv_bfloat16>(), gemm_status_ptr(), loss);
}
void draw_batch(gelios_mlp* n, int batch) {
    gather_kernel<<<blocks(static_cast<int64_t>(batch) * kRowThreads, 128), 128, 0, n->stream>>>(
        batch, n->n_rows, n->n_in, n->nf, n->ld0, n->n_out, n->X.as<float>(), n->T.as<float>(),
        n->args.as<StepArgs>(), n->at.as<int>(), n->h[0].as<__nv_bfloat16>(), n->tb.as<float>(),
        n->fused ? n->ht_of(0) : nullptr, pad8(batch));
}
// One fused training step on the network's streams.
bool enqueue_train_step(gelios_mlp* n, int batch) {
    draw_batch(n, batch);
    forward(n, batch, true);
    if (!backward_fused(n, batch, n->hist.as<float>(), n->at.as<int>())) return false;
    reduce_fused(n, batch, n->args.as<StepArgs>(), n->at.as<int>(), n->hist.as<float>());
    return cudaGetLastError() == cudaSuccess;
}
// The same as a graph, captured once per batch size and training set; null
// where it cannot be captured (the step is then enqueued directly).
cudaGraphExec_t train_graph(gelios_mlp* n, int batch) {
    if (n->graph && n->graph_batch == batch) return n->graph;
    n->drop_graph();
    capture_graph(n->stream, &n->graph, [&]() { return enqueue_train_step(n, batch); });
    n->graph_batch = batch;
    return n->graph;
}

// loss of the batch (targets in tb) into loss[0]; gradients into g32
void backward(gelios_mlp* n, int M, float* loss, int* at) {
    cudaStream_t s = n->stream;
    const int L = n->layers();
    const int64_t eo = static_cast<int64_t>(M) * n->n_out;
    mse_kernel<<<blocks(M, 256), 256, 0, s>>>(M, n->n_out, n->y.as<float>(), n->tb.as<float>(), n->dh,
                                              n->rowerr.as<float>());
    loss_kernel<<<1, 256, 0, s>>>(M, n->n_out, n->rowerr.as<float>(), loss, at);
    act_bwd_kernel<<<blocks(eo, 256), 256, 0, s>>>(eo, n->dh, nullptr, n->dz,
                                                   n->dzb.as<__nv_bfloat16>(), 0);
    const __nv_bfloat16* wb = n->wb.as<__nv_bfloat16>();
    float* g = n->g32.as<float>();
    const int splits = split_target(M), S = splits_of(M);
    const int64_t Mp = pad8(M);
    __nv_bfloat16* dzt = n->dzt;
    __nv_bfloat16* ht = n->ht;
    for (int l = L - 1; l >= 0; l--) {
        const int di = n->din[l], dO = n->dout[l];
        // dW[dO][di] = dZ^T . H_l (both transposed so k = batch row is
        // contiguous), split over the rows of the batch
        const int64_t wn = static_cast<int64_t>(dO) * di;
        transpose(M, dO, n->dzb.as<__nv_bfloat16>(), dO, dzt, Mp, s);
        transpose(M, di, n->h[l].as<__nv_bfloat16>(), l == 0 ? n->ld0 : di, ht, Mp, s);
        gemm(dO, di, M, dzt, Mp, ht, Mp, n->part, di, s, splits, wn);
        splitk_reduce_kernel<<<blocks(wn, 256), 256, 0, s>>>(wn, S, n->part, g + n->w_off[l]);
        // db = column sums of dZ
        const int chunks = (M + kColRows - 1) / kColRows;
        col_sum_partial_kernel<<<dim3(blocks(dO, 128), chunks), 128, 0, s>>>(M, dO, n->dz,
                                                                             n->colpart);
        col_sum_final_kernel<<<blocks(dO, 128), 128, 0, s>>>(chunks, dO, n->colpart, g + n->b_off[l]);
        if (l == 0) break;
        // dH_l[M][di] = dZ . W_l, then dZ_{l-1} = dH_l * GELU'(Z_{l-1})
        transpose(dO, di, wb + n->w_off[l], di, n->wt, pad8(dO), s);
        gemm(M, di, dO, n->dzb.as<__nv_bfloat16>(), dO, n->wt, pad8(dO), n->dh, di,
             s);
        const int64_t e = static_cast<int64_t>(M) * di;
        act_bwd_kernel<<<blocks(e, 256), 256, 0, s>>>(e, n->dh, n->z[l - 1].as<float>(),
                                                      n->dz, n->dzb.as<__nv_bfloat16>(), 1);
    }
}

// The W^T copies (and layer 0's padded W) of the current bf16 weights.
void copy_weights(gelios_mlp* n) {
    int64_t most = 0;
    for (int l = 0; l < n->layers(); l++) most = std::max(most, static_cast<int64_t>(n->din[l]) * n->dout[l]);
    weight_copies_kernel<<<dim3(blocks(most, 256), n->layers()), 256, 0, n->stream>>>(n->f_layers.as<LayerGrad>(),
                                                                                      n->wb.as<__nv_bfloat16>());
}

// Decides, at the first use of a gradient, whether the fused training step
// takes the network (16-byte rows for the TMA: a width that is a multiple of
// 8; the output columns in mse_grad_kernel's tile; partial sums of at most
// 256 MB) and allocates what it needs: per layer H^T, dZ^T, W^T, the partial
// and column sums.  Otherwise, and without room for them, the separate
// kernels run, with their own workspaces.
int ensure_training(gelios_mlp* n) {
    if (n->training_known) return GELIOS_OK;
    const int depth = n->depth, width = n->width;
    const size_t MB = static_cast<size_t>(n->max_batch), Mp = static_cast<size_t>(pad8(n->max_batch));
    const size_t widest = static_cast<size_t>(std::max({n->in_w, width, n->n_out}));
    const int64_t chunks = (n->max_batch + kColRows - 1) / kColRows;
    int64_t part = 0, col = 0, wt = 0;
    for (int l = 0; l <= depth; l++) {
        LayerGrad& g = n->layers_host[l];
        g.part_off = part;
        g.col_off = col;
        part += static_cast<int64_t>(reserved_splits(n->max_batch)) * g.din * g.dout;
        col += chunks * g.dout;
        if (l > 0) wt += static_cast<int64_t>(g.din) * g.ld_t;
    }
    CUtensorMap tz, th;
    if (width % 8 == 0 && n->n_out <= kMseCols && part <= (int64_t(64) << 20) &&
        output_map(&tz, n->z[0].p, true, n->max_batch, width) &&
        output_map(&th, n->h[1].p, false, n->max_batch, width)) {
        Carve c;
        const size_t o_ht = c.take(Mp * (n->in_w + static_cast<size_t>(depth) * width) * 2);
        const size_t o_dzt = c.take(Mp * width * (static_cast<size_t>(depth) + 1) * 2 + Mp * kMseCols * 2);
        const size_t o_wt = c.take(static_cast<size_t>(wt) * 2), o_part = c.take(static_cast<size_t>(part) * 4);
        const size_t o_col = c.take(static_cast<size_t>(col) * 4), o_dz = c.take(MB * pad8(widest) * 2);
        if (n->train_mem.alloc(c.bytes)) {
            char* p = n->train_mem.as<char>();
            n->f_ht = reinterpret_cast<__nv_bfloat16*>(p + o_ht);
            n->f_dzt = reinterpret_cast<__nv_bfloat16*>(p + o_dzt);
            n->f_dzb2 = reinterpret_cast<__nv_bfloat16*>(p + o_dz);
            n->f_part = reinterpret_cast<float*>(p + o_part);
            n->f_col = reinterpret_cast<float*>(p + o_col);
            __nv_bfloat16* w = reinterpret_cast<__nv_bfloat16*>(p + o_wt);
            for (int l = 1; l <= depth; l++) {
                LayerGrad& g = n->layers_host[l];
                g.wt = w;
                w += static_cast<int64_t>(g.din) * g.ld_t;
            }
            MLP_TRY(cudaStreamCreateWithFlags(&n->side, cudaStreamNonBlocking));
            MLP_TRY(cudaEventCreateWithFlags(&n->ev_dz, cudaEventDisableTiming));
            MLP_TRY(cudaEventCreateWithFlags(&n->ev_side, cudaEventDisableTiming));
            MLP_TRY(cudaMemsetAsync(p + o_wt, 0, static_cast<size_t>(wt) * 2, n->stream));
            MLP_TRY(cudaMemcpyAsync(n->f_layers.p, n->layers_host.data(), sizeof(LayerGrad) * n->layers_host.size(),
                                    cudaMemcpyHostToDevice, n->stream));
            copy_weights(n);
            MLP_TRY(cudaGetLastError());
            n->fused = n->training_known = true;
            return GELIOS_OK;
        }
        cudaGetLastError();
    }
    Carve c;
    const size_t o_dh = c.take(MB * widest * 4), o_dz = c.take(MB * widest * 4);
    const size_t o_part = c.take(static_cast<size_t>(kMaxSplit) * widest * widest * 4);
    const size_t o_col = c.take(static_cast<size_t>(chunks) * widest * 4), o_wt = c.take(widest * pad8(widest) * 2);
    const size_t o_dzt = c.take(widest * Mp * 2), o_ht = c.take(widest * Mp * 2);
    if (!n->train_mem.alloc(c.bytes)) return cuda_fail(cudaErrorMemoryAllocation);
    char* p = n->train_mem.as<char>();
    n->dh = reinterpret_cast<float*>(p + o_dh);
    n->dz = reinterpret_cast<float*>(p + o_dz);
    n->part = reinterpret_cast<float*>(p + o_part);
    n->colpart = reinterpret_cast<float*>(p + o_col);
    n->wt = reinterpret_cast<__nv_bfloat16*>(p + o_wt);
    n->dzt = reinterpret_cast<__nv_bfloat16*>(p + o_dzt);
    n->ht = reinterpret_cast<__nv_bfloat16*>(p + o_ht);
    n->training_known = true;
    return GELIOS_OK;
}

// The pinned staging of gelios_mlp_predict; without it the copies go through
// the driver's.
void ensure_staging(gelios_mlp* n) {
    const int64_t xf = pad8(n->chunk_rows * n->n_in), yf = pad8(n->chunk_rows * n->n_out);
    const int64_t bytes = (16 + 2 * (xf + yf)) * 4;
    if (n->stage || n->stage_failed || !staging_worth(n->predictions, n->io_bytes, bytes)) return;
    void* p = nullptr;
    n->stage_failed = cudaMallocHost(&p, static_cast<size_t>(bytes)) != cudaSuccess;
    for (cudaEvent_t& e : n->ev_chunk)
        n->stage_failed = n->stage_failed || cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess;
    if (n->stage_failed) {
        cudaGetLastError();
        if (p) cudaFreeHost(p);
        return;
    }
    n->stage = static_cast<int*>(p);
    for (int k = 0; k < 2; k++) {
        n->px[k] = static_cast<float*>(p) + 16 + k * (xf + yf);
        n->py[k] = n->px[k] + xf;
    }
}
}  // namespace

extern "C" int gelios_mlp_create(gelios_mlp** out, int device, int n_in, int n_fourier, int width, int depth,
                                 int n_out, int max_batch) {
    if (!out) return fail("gelios_mlp_create: null output");
    *out = nullptr;
    if (n_in < 2 || n_in > 256 || n_fourier < 0 || n_fourier > 16 || width < 1 || width > 4096 || depth < 1 ||
        depth > 64 || n_out < 1 || n_out > 4096 || max_batch < 1 || max_batch > (1 << 20))
        return fail("gelios_mlp_create: sizes out of range");
    auto n = std::make_unique<gelios_mlp>();
    n->device = device;
    n->n_in = n_in;
    n->nf = n_fourier;
    n->width = width;
    n->depth = depth;
    n->n_out = n_out;
    n->max_batch = max_batch;
    n->in_w = n_in + 4 * n_fourier;
    n->ld0 = static_cast<int>(pad8(n->in_w));
    MLP_TRY(cudaSetDevice(device));
    MLP_TRY(cudaStreamCreateWithFlags(&n->stream, cudaStreamNonBlocking));
    int64_t off = 0;
    int widest = n->in_w > width ? n->in_w : width;
    if (n_out > widest) widest = n_out;
    for (int l = 0; l <= depth; l++) {
        const int di = l == 0 ? n->in_w : width, dO = l == depth ? n_out : width;
        n->din.push_back(di);
        n->dout.push_back(dO);
        n->w_off.push_back(off);
        off += static_cast<int64_t>(di) * dO;
        n->b_off.push_back(off);
        off += dO;
    }
    n->n_params = off;
    const size_t P = static_cast<size_t>(off);
    const size_t MB = static_cast<size_t>(max_batch), W = static_cast<size_t>(widest);
    bool ok = n->w32.alloc(P * 4) && n->g32.alloc(P * 4) && n->m.alloc(P * 4) && n->v.alloc(P * 4) &&
              n->wb.alloc(P * 2);
    n->h.resize(depth + 1);
    n->z.resize(depth);
    for (int l = 0; l <= depth; l++) ok = ok && n->h[l].alloc(MB * (l == 0 ? n->ld0 : n->din[l]) * 2);
    ok = ok && n->wpad.alloc(static_cast<size_t>(n->dout[0]) * n->ld0 * 2);
    for (int l = 0; l < depth; l++) ok = ok && n->z[l].alloc(MB * width * 4);
    ok = ok && n->c.alloc(MB * W * 4) && n->y.alloc(MB * n_out * 4) && n->dzb.alloc(MB * pad8(widest) * 2) &&
         n->tb.alloc(MB * n_out * 4) && n->rowerr.alloc(MB * 4) && n->loss.alloc(16) && n->xin.alloc(MB * n_in * 4);
    if (!ok) return cuda_fail(cudaErrorMemoryAllocation);
    n->chunk_rows = stage_rows(max_batch, n_in, n_out);
    MLP_TRY(cudaMemsetAsync(n->wpad.p, 0, n->wpad.bytes, n->stream));
    for (int l = 0; l <= depth; l++) {
        LayerGrad g{};
        g.w_off = n->w_off[l];
        g.b_off = n->b_off[l];
        g.din = n->din[l];
        g.dout = n->dout[l];
        g.ld_in = n->ld0;
        g.ld_t = static_cast<int>(pad8(g.dout));
        if (l == 0) g.wpad = n->wpad.as<__nv_bfloat16>();
        n->layers_host.push_back(g);
    }
    if (!n->f_layers.alloc(sizeof(LayerGrad) * n->layers_host.size())) return cuda_fail(cudaErrorMemoryAllocation);
    MLP_TRY(cudaMemcpyAsync(n->f_layers.p, n->layers_host.data(), sizeof(LayerGrad) * n->layers_host.size(),
                            cudaMemcpyHostToDevice, n->stream));
    MLP_TRY(cudaMemsetAsync(n->w32.p, 0, P * 4, n->stream));
    MLP_TRY(cudaMemsetAsync(n->wb.p, 0, P * 2, n->stream));
    MLP_TRY(cudaMemsetAsync(n->m.p, 0, P * 4, n->stream));
    MLP_TRY(cudaMemsetAsync(n->v.p, 0, P * 4, n->stream));
    MLP_TRY(cudaStreamSynchronize(n->stream));
    *out = n.release();
    return GELIOS_OK;
}

extern "C" void gelios_mlp_destroy(gelios_mlp* n) {
    if (!n) return;
    cudaSetDevice(n->device);
    cudaStreamSynchronize(n->stream);
    delete n;
}

extern "C" int64_t gelios_mlp_param_count(const gelios_mlp* n) { return n ? n->n_params : -1; }

extern "C" int gelios_mlp_set_params(gelios_mlp* n, const float* host, int64_t count) {
    if (!n || !host || count != n->n_params) return fail("gelios_mlp_set_params: wrong parameter count");
    MLP_TRY(cudaSetDevice(n->device));
    const size_t P = static_cast<size_t>(n->n_params);
    MLP_TRY(cudaMemcpyAsync(n->w32.p, host, P * 4, cudaMemcpyHostToDevice, n->stream));
    to_bf16_kernel<<<blocks(n->n_params, 256), 256, 0, n->stream>>>(n->n_params, n->w32.as<float>(),
                                                                    n->wb.as<__nv_bfloat16>());
    copy_weights(n);
    MLP_TRY(cudaMemsetAsync(n->m.p, 0, P * 4, n->stream));
    MLP_TRY(cudaMemsetAsync(n->v.p, 0, P * 4, n->stream));
    MLP_TRY(cudaGetLastError());
    MLP_TRY(cudaStreamSynchronize(n->stream));
    n->step = 0;
    return GELIOS_OK;
}

extern "C" int gelios_mlp_get_params(const gelios_mlp* n, float* host, int64_t count) {
    if (!n || !host || count != n->n_params) return fail("gelios_mlp_get_params: wrong parameter count");
    MLP_TRY(cudaSetDevice(n->device));
    MLP_TRY(cudaMemcpyAsync(host, n->w32.p, static_cast<size_t>(count) * 4, cudaMemcpyDeviceToHost, n->stream));
    MLP_TRY(cudaStreamSynchronize(n->stream));
    return GELIOS_OK;
}

extern "C" int gelios_mlp_loss_grad(gelios_mlp* n, const float* x, const float* t, int M, double* loss, float* grad) {
    if (!n || !x || !t || M < 1 || M > n->max_batch) return fail("gelios_mlp_loss_grad: bad arguments");
    MLP_TRY(cudaSetDevice(n->device));
    if (const int rc = ensure_training(n)) return rc;
    cudaStream_t s = n->stream;
    MLP_TRY(cudaMemcpyAsync(n->xin.p, x, static_cast<size_t>(M) * n->n_in * 4, cudaMemcpyHostToDevice, s));
    MLP_TRY(cudaMemcpyAsync(n->tb.p, t, static_cast<size_t>(M) * n->n_out * 4, cudaMemcpyHostToDevice, s));
    features_kernel<<<blocks(static_cast<int64_t>(M) * kRowThreads, 128), 128, 0, s>>>(M, n->n_in, n->nf, n->ld0, n->xin.as<float>(),
                                                   n->h[0].as<__nv_bfloat16>());
    forward(n, M, n->fused);
    if (n->fused) {
        transpose(M, n->in_w, n->h[0].as<__nv_bfloat16>(), n->ld0, n->ht_of(0), pad8(M), s);
        if (!backward_fused(n, M, n->loss.as<float>(), nullptr)) return cuda_fail(cudaErrorInvalidValue);
        reduce_fused(n, M, nullptr, nullptr, n->loss.as<float>());
    } else {
        backward(n, M, n->loss.as<float>(), nullptr);
    }
    MLP_TRY(cudaGetLastError());
    struct {
        float loss;
        int bad;
    } got{};
    MLP_TRY(cudaMemcpyAsync(&got, n->loss.p, n->fused ? 8 : 4, cudaMemcpyDeviceToHost, s));
    if (grad)
        MLP_TRY(cudaMemcpyAsync(grad, n->g32.p, static_cast<size_t>(n->n_params) * 4, cudaMemcpyDeviceToHost, s));
    if (!n->fused) gemm_status_fetch(&got.bad, s);
    MLP_TRY(cudaStreamSynchronize(s));
    if (got.bad && !gemm_status_ok()) return cuda_fail(cudaErrorLaunchTimeout);
    if (loss) *loss = got.loss;
    return GELIOS_OK;
}

extern "C" int gelios_mlp_set_data(gelios_mlp* n, const float* x, const float* t, int64_t n_rows) {
    if (!n || !x || !t || n_rows < 1) return fail("gelios_mlp_set_data: bad arguments");
    MLP_TRY(cudaSetDevice(n->device));
    n->drop_graph();  // it holds the training set's addresses and size
    if (const int rc = ensure_training(n)) return rc;
    n->n_rows = 0;
    if (!n->X.alloc(static_cast<size_t>(n_rows) * n->n_in * 4) ||
        !n->T.alloc(static_cast<size_t>(n_rows) * n->n_out * 4))
        return cuda_fail(cudaErrorMemoryAllocation);
    MLP_TRY(cudaMemcpyAsync(n->X.p, x, static_cast<size_t>(n_rows) * n->n_in * 4, cudaMemcpyHostToDevice, n->stream));
    MLP_TRY(cudaMemcpyAsync(n->T.p, t, static_cast<size_t>(n_rows) * n->n_out * 4, cudaMemcpyHostToDevice, n->stream));
    MLP_TRY(cudaStreamSynchronize(n->stream));
    n->n_rows = n_rows;
    return GELIOS_OK;
}

extern "C" int gelios_mlp_train(gelios_mlp* n, int iters, int batch, float lr_max, float lr_min, int warmup,
                                uint64_t seed, float* loss_hist) {
    if (!n || iters < 0 || batch < 1 || batch > n->max_batch || !(lr_max >= 0.f) || !(lr_min >= 0.f) || warmup < 0)
        return fail("gelios_mlp_train: bad arguments");
    if (n->n_rows < 1) return fail("gelios_mlp_train: no training set (gelios_mlp_set_data)");
    MLP_TRY(cudaSetDevice(n->device));
    cudaStream_t s = n->stream;
    if (iters > n->steps_cap) {
        const int64_t cap = std::max<int64_t>(iters, 256);
        n->drop_graph();
        n->steps_cap = 0;
        if (!n->args.alloc(static_cast<size_t>(cap) * sizeof(StepArgs)) ||
            !n->hist.alloc(static_cast<size_t>(cap + 1) * 4) || (!n->at.p && !n->at.alloc(sizeof(int))))
            return cuda_fail(cudaErrorMemoryAllocation);
        n->steps_cap = cap;
    }
    const float b1 = kAdamB1, b2 = kAdamB2;
    std::vector<StepArgs> args(static_cast<size_t>(iters));
    for (int it = 0; it < iters; it++) {
        StepArgs& a = args[it];
        a.key = seed * 0xD1B54A32D192ED03ULL + static_cast<uint64_t>(n->step) * 0x8CB92BA72F3D8DD7ULL;
        if (it < warmup) {
            a.lr = lr_max * static_cast<float>(it + 1) / static_cast<float>(warmup);
        } else {
            const double q = iters > warmup ? static_cast<double>(it - warmup) / (iters - warmup) : 1.0;
            a.lr = static_cast<float>(lr_min + 0.5 * (lr_max - lr_min) * (1.0 + std::cos(3.14159265358979 * q)));
        }
        n->step++;
        a.c1 = static_cast<float>(1.0 - std::pow(static_cast<double>(b1), n->step));
        a.c2 = static_cast<float>(1.0 - std::pow(static_cast<double>(b2), n->step));
        a.pad = 0;
    }
    if (iters > 0) {
        MLP_TRY(cudaMemcpyAsync(n->args.p, args.data(), sizeof(StepArgs) * args.size(), cudaMemcpyHostToDevice, s));
        MLP_TRY(cudaMemsetAsync(n->at.p, 0, sizeof(int), s));
    }
    cudaGraphExec_t graph = n->fused && iters > 1 ? train_graph(n, batch) : nullptr;
    for (int it = 0; it < iters; it++) {
        if (graph) {
            MLP_TRY(cudaGraphLaunch(graph, s));
        } else if (n->fused) {
            if (!enqueue_train_step(n, batch)) return cuda_fail(cudaErrorInvalidValue);
        } else {
            draw_batch(n, batch);
            forward(n, batch);
            backward(n, batch, n->hist.as<float>(), n->at.as<int>());
            const StepArgs& a = args[it];
            adam_kernel<<<blocks(n->n_params, 256), 256, 0, s>>>(n->n_params, n->w32.as<float>(), n->g32.as<float>(),
                                                                 n->m.as<float>(), n->v.as<float>(), a.lr, b1, b2,
                                                                 kAdamEps, a.c1, a.c2, n->wb.as<__nv_bfloat16>(),
                                                                 n->layers_host[0]);
        }
        MLP_TRY(cudaGetLastError());
    }
    // the losses, and behind them the GEMM status word (grad_adam_kernel)
    int bad = 0;
    if (n->fused && iters > 0) {
        std::vector<float> got(static_cast<size_t>(iters) + 1);
        MLP_TRY(cudaMemcpyAsync(got.data(), n->hist.p, got.size() * 4, cudaMemcpyDeviceToHost, s));
        MLP_TRY(cudaStreamSynchronize(s));
        if (loss_hist) std::memcpy(loss_hist, got.data(), static_cast<size_t>(iters) * 4);
        std::memcpy(&bad, &got[iters], 4);
    } else {
        if (loss_hist && iters > 0)
            MLP_TRY(cudaMemcpyAsync(loss_hist, n->hist.p, static_cast<size_t>(iters) * 4, cudaMemcpyDeviceToHost, s));
        gemm_status_fetch(&bad, s);
        MLP_TRY(cudaStreamSynchronize(s));
    }
    if (bad && !gemm_status_ok()) return cuda_fail(cudaErrorLaunchTimeout);
    return GELIOS_OK;
}

extern "C" int gelios_mlp_predict(gelios_mlp* n, const float* x, int64_t M, float* y) {
    if (!n || !x || !y || M < 0) return fail("gelios_mlp_predict: bad arguments");
    MLP_TRY(cudaSetDevice(n->device));
    cudaStream_t s = n->stream;
    // The chunks pass through pinned staging, two at a time, once that is worth
    // it: a copy from or to pageable memory of this size goes through the
    // driver's own, in turn.
    n->predictions++;
    n->io_bytes += M * (n->n_in + n->n_out) * 4;
    ensure_staging(n);
    const bool staged = n->stage != nullptr;
    const int64_t mb = n->chunk_rows;
    auto rows = [&](int64_t k) { return std::min(mb, M - k * mb); };
    auto collect = [&](int64_t k) {
        const cudaError_t e = cudaEventSynchronize(n->ev_chunk[k & 1]);
        if (e == cudaSuccess)
            std::memcpy(y + k * mb * n->n_out, n->py[k & 1], static_cast<size_t>(rows(k)) * n->n_out * 4);
        return e;
    };
    const int64_t chunks = (M + mb - 1) / mb;
    for (int64_t k = 0; k < chunks; k++) {
        const int b = static_cast<int>(k & 1), m = static_cast<int>(rows(k));
        const size_t xb = static_cast<size_t>(m) * n->n_in * 4;
        const float* xs = x + k * mb * n->n_in;
        if (staged) {
            if (k >= 2) MLP_TRY(collect(k - 2));
            std::memcpy(n->px[b], xs, xb);
            xs = n->px[b];
        }
        MLP_TRY(cudaMemcpyAsync(n->xin.p, xs, xb, cudaMemcpyHostToDevice, s));
        features_kernel<<<blocks(static_cast<int64_t>(m) * kRowThreads, 128), 128, 0, s>>>(
            m, n->n_in, n->nf, n->ld0, n->xin.as<float>(), n->h[0].as<__nv_bfloat16>());
        forward(n, m);
        MLP_TRY(cudaGetLastError());
        MLP_TRY(cudaMemcpyAsync(staged ? n->py[b] : y + k * mb * n->n_out, n->y.p,
                                static_cast<size_t>(m) * n->n_out * 4, cudaMemcpyDeviceToHost, s));
        if (staged) {
            if (k + 1 == chunks) gemm_status_fetch(n->stage, s);
            MLP_TRY(cudaEventRecord(n->ev_chunk[b], s));
        }
    }
    int bad = 0;
    if (staged) {
        for (int64_t k = std::max<int64_t>(0, chunks - 2); k < chunks; k++) MLP_TRY(collect(k));
        bad = chunks > 0 ? *n->stage : 0;
    } else {
        gemm_status_fetch(&bad, s);
        MLP_TRY(cudaStreamSynchronize(s));
    }
    if (bad && !gemm_status_ok()) return cuda_fail(cudaErrorLaunchTimeout);
    return GELIOS_OK;
}

extern "C" int gelios_mlp_gemm_bf16(int M, int N, int K, const void* A, int64_t lda, const void* B, int64_t ldb,
                                    float* C, int64_t ldc, void* stream) {
    if (M < 0 || N < 0 || K < 0 || !A || !B || !C || lda < K || ldb < K || ldc < N)
        return fail("gelios_mlp_gemm_bf16: bad arguments");
    gemm(M, N, K, static_cast<const __nv_bfloat16*>(A), lda, static_cast<const __nv_bfloat16*>(B), ldb, C, ldc,
         static_cast<cudaStream_t>(stream));
    MLP_TRY(cudaGetLastError());
    MLP_TRY(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
    if (!gemm_status_ok()) return cuda_fail(cudaErrorLaunchTimeout);
    return GELIOS_OK;
}

extern "C" int gelios_mlp_time_layer(int M, int N, int K, int reps, int tma, double* ms) {
    if (M <= 0 || N <= 0 || K <= 0 || reps < 1 || !ms) return fail("gelios_mlp_time_layer: bad arguments");
    const int64_t lda = pad8(K);
    Buf A, B, bias, Z, H, Cf;
    if (!A.alloc(static_cast<size_t>(M) * lda * 2) || !B.alloc(static_cast<size_t>(N) * lda * 2) ||
        !Cf.alloc(tma ? 16 : static_cast<size_t>(M) * N * 4) ||
        !bias.alloc(static_cast<size_t>(N) * 4) || !Z.alloc(static_cast<size_t>(M) * N * 4) ||
        !H.alloc(static_cast<size_t>(M) * N * 2))
        return cuda_fail(cudaErrorMemoryAllocation);
    cudaStream_t s = nullptr;
    MLP_TRY(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
    std::unique_ptr<CUstream_st, void (*)(cudaStream_t)> guard(s, [](cudaStream_t x) { cudaStreamDestroy(x); });
    // seeded operands (a fixed hash of the index, scaled like a trained layer)
    {
        std::vector<__nv_bfloat16> ha(static_cast<size_t>(M) * lda), hb(static_cast<size_t>(N) * lda);
        std::vector<float> hbias(N);
        auto val = [](uint64_t i) {
            uint64_t z = i * 0x9E3779B97F4A7C15ULL;
            z = (z ^ (z >> 31)) * 0xBF58476D1CE4E5B9ULL;
            return static_cast<float>((z >> 40) & 0xFFFF) / 65536.f - 0.5f;
        };
        for (size_t i = 0; i < ha.size(); i++) ha[i] = __float2bfloat16(val(i));
        for (size_t i = 0; i < hb.size(); i++) hb[i] = __float2bfloat16(0.1f * val(i + ha.size()));
        for (int i = 0; i < N; i++) hbias[i] = 0.01f * val(i + 7);
        MLP_TRY(cudaMemcpyAsync(A.p, ha.data(), ha.size() * 2, cudaMemcpyHostToDevice, s));
        MLP_TRY(cudaMemcpyAsync(B.p, hb.data(), hb.size() * 2, cudaMemcpyHostToDevice, s));
        MLP_TRY(cudaMemcpyAsync(bias.p, hbias.data(), hbias.size() * 4, cudaMemcpyHostToDevice, s));
    }
    GemmEpilogue ep;
    ep.bias = bias.as<float>();
    ep.Z = Z.as<float>();
    ep.H = H.as<__nv_bfloat16>();
    ep.act = 1;
    const dim3 grid(blocks(N, TC_BN), blocks(M, TC_BM), 1);
    const int kc = tc_split_len(K, 1);
    auto layer = [&]() {
        if (tma)
            return launch_tma<1>(grid, M, N, K, kc, A.as<__nv_bfloat16>(), lda, B.as<__nv_bfloat16>(), lda, nullptr, 0,
                                 0, ep, s);
        // the cp.async-staged GEMM, then the bias + activation kernel
        const dim3 g2(blocks(N, TC_BN), blocks(M, TC_BM), 1);
        launch_tc<true, true>(g2, M, N, K, kc, A.as<__nv_bfloat16>(), lda, B.as<__nv_bfloat16>(), lda, Cf.as<float>(),
                              N, 0, s);
        const int64_t e = static_cast<int64_t>(M) * N;
        bias_act_kernel<<<blocks(e, 256), 256, 0, s>>>(M, N, Cf.as<float>(), ep.bias, ep.Z, ep.H, nullptr, 1);
        return true;
    };
    if (!layer()) return fail("gelios_mlp_time_layer: no tensor-map encoder in this driver");
    // the reps launches captured in one CUDA graph, so that the device time
    // per layer is not the host's launch rate
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    MLP_TRY(cudaStreamBeginCapture(s, cudaStreamCaptureModeRelaxed));
    for (int r = 0; r < reps; r++) layer();
    MLP_TRY(cudaStreamEndCapture(s, &graph));
    std::unique_ptr<CUgraph_st, void (*)(cudaGraph_t)> gguard(graph, [](cudaGraph_t g) { cudaGraphDestroy(g); });
    MLP_TRY(cudaGraphInstantiate(&exec, graph, 0));
    std::unique_ptr<CUgraphExec_st, void (*)(cudaGraphExec_t)> xguard(exec,
                                                                      [](cudaGraphExec_t x) { cudaGraphExecDestroy(x); });
    MLP_TRY(cudaGraphLaunch(exec, s));
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    MLP_TRY(cudaEventCreate(&e0));
    MLP_TRY(cudaEventCreate(&e1));
    MLP_TRY(cudaEventRecord(e0, s));
    MLP_TRY(cudaGraphLaunch(exec, s));
    MLP_TRY(cudaEventRecord(e1, s));
    MLP_TRY(cudaEventSynchronize(e1));
    float t = 0.f;
    MLP_TRY(cudaEventElapsedTime(&t, e0, e1));
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    MLP_TRY(cudaGetLastError());
    if (!gemm_status_ok()) return cuda_fail(cudaErrorLaunchTimeout);
    *ms = static_cast<double>(t) / reps;
    return GELIOS_OK;
}
