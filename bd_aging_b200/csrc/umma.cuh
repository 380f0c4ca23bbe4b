// umma.cuh -- BF16 GEMMs on the sm_100a tensor cores (tcgen05 / UMMA) for the
// surrogate network's weight gradients: C[M][N] = sum_k A[M][k] B[N][k] (both
// operands K-major, BF16; FP32 accumulation in tensor memory), written
// transposed as FP32 split-K partials.  The PTX helpers here are shared with
// the fused forward / input-gradient kernel (mlp_chain.cuh).
//
// One launch takes a table of GEMMs (every layer's weight gradient), a CTA
// (16 warps) a 128 x bn tile of one of them over a K range of at most 256:
//   * one lane of warp 0 issues every TMA load of the range at once (64-wide K chunks,
//     128-byte swizzle, one mbarrier per chunk, no multicast);
//   * one lane of warp 1 issues tcgen05.mma (M=128, N=bn, K=16) per 16-wide
//     slice as each chunk lands, then tcgen05.commit to the "done" barrier;
//   * all warps read accumulator rows with tcgen05.ld (warp w: lanes
//     32 (w % 4) .. + 31, every fourth group of 32 columns) and store them.
// What bounds it: a CTA's loads (up to 192 KB), its few MMAs and its stores
// (up to 128 KB) follow one another, so the layers run side by side: the five
// GEMMs of the 256-wide network at a batch of 4096 are 144 CTAs, one wave of
// the 148 SMs, with bn = all of N (a 128 x 64 tile reads A four times).
// All five take 11.0 us (as launches of 128 x 64 tiles, 5 x 6.5 us).
// Every mbarrier wait is bounded: on expiry the CTA records an error flag,
// waits (bounded) for its own copies, frees its tensor memory and returns.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>

namespace bd {
namespace umma {

constexpr int kBM = 128, kBN = 64, kBK = 64;  // kBK bf16 = one 128-byte swizzle row
constexpr int kMaxChunks = 4;                  // K range per CTA <= 256
constexpr int kThreads = 512;                  // 16 warps: warp w reads TMEM lanes 32 (w % 4)
constexpr int kMaxBN = 256;                    // widest tile (rows of B per CTA)
constexpr int kStageA = kBM * kBK * 2;         // 16 KB per A tile
constexpr int gemm_stage_b(int bn) { return bn * kBK * 2; }
constexpr int gemm_smem(int bn) { return kMaxChunks * (kStageA + gemm_stage_b(bn)) + 1024 /* align */ + 256 /* barriers */; }
static_assert(gemm_smem(kMaxBN) <= 227 * 1024, "shared memory of one CTA");
constexpr long kSpinLimit = 1L << 20;
constexpr int kMaxJobs = 9;                    // GEMMs of one launch (layers of the network)

struct GemmJob {
    CUtensorMap a, b;     // A [M][K], box 64 x 128; B [N][K], box 64 x bn
    // split-K partials stored transposed, [splits][N][M]: the epilogue thread
    // owns one row m, so consecutive lanes touch consecutive addresses
    float *out_f32;
    int M, N, K;          // logical sizes (rows of A, rows of B, reduction)
    int k_split;          // K range per CTA (multiple of 64, <= 256)
    int bn;               // tile width: a multiple of 64, <= kMaxBN
    int first;            // first block of the job (tiles m fastest, then n, then the K ranges)
};
struct GemmTable {
    GemmJob job[kMaxJobs];
    int n_jobs;
    long long *count;     // counter the launch adds 1 to, or nullptr
    unsigned *err;
};

// ----------------------------------------------------------------- PTX
__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// bounded wait: false (and the error flag set) when the barrier never flips
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, unsigned *err, unsigned code) {
    for (long i = 0; i < kSpinLimit; i++)
        if (mbar_try_wait(bar, parity)) return true;
    atomicOr(err, code);
    return false;
}
// One lane of a converged warp.  The loads, MMAs and commits below take it as
// a predicate inside warp-uniform code instead of standing in a branch of lane
// 0: their operands then live in uniform registers (in the branch an MMA took
// about 125 cycles to issue, and a load about 350).
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t e;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(e));
    return e;
}
__device__ __forceinline__ void tma_load_2d(uint32_t lead, uint32_t dst, const CUtensorMap *map, uint32_t bar, int x,
                                            int y) {
    asm volatile(
        "{\n\t.reg .pred e;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n\t}" ::
            "r"(dst),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 bytes apart (SBO), leading offset 1 (unused for swizzled K-major),
// descriptor version 1 (bits 46-47), layout type 2 = SWIZZLE_128B (bits 61-63)
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t addr) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// instruction descriptor, kind::f16, M = 128 and n columns: D f32 (bits 4-5 =
// 1), A and B bf16 (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17,
// M >> 4 at bit 24
__device__ __forceinline__ uint32_t umma_idesc(int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
}
__device__ __forceinline__ void umma_bf16(uint32_t lead, uint32_t tmem_d, uint64_t adesc, uint64_t bdesc,
                                          uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, e;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 e, %5, 0;\n\t"
        "@e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t lead, uint64_t *bar) {
    asm volatile(
        "{\n\t.reg .pred e;\n\t"
        "setp.ne.b32 e, %1, 0;\n\t"
        "@e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)),
        "r"(lead)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float *v) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
        "%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float *v) {
    tmem_ld16(taddr, v);
    tmem_ld16(taddr + 16, v + 16);
}

// ----------------------------------------------------------------- math
__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678f)); }
// gelu(z) and its derivative, which share erf
__device__ __forceinline__ void gelu_both(float z, float *h, float *d) {
    const float e = 1.0f + erff(z * 0.70710678f);
    *h = 0.5f * z * e;
    *d = 0.5f * e + z * 0.39894228f * expf(-0.5f * z * z);
}

// ----------------------------------------------------------------- kernel
__global__ void __launch_bounds__(kThreads, 1) k_umma_gemm(const __grid_constant__ GemmTable t) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem =
        reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    int ji = 0;
    while (ji + 1 < t.n_jobs && (int)blockIdx.x >= t.job[ji + 1].first) ji++;
    const GemmJob &g = t.job[ji];
    const int stage_b = gemm_stage_b(g.bn);
    unsigned char *sA = smem;                          // [kMaxChunks][kStageA]
    unsigned char *sB = smem + kMaxChunks * kStageA;   // [kMaxChunks][stage_b]
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kMaxChunks * (kStageA + stage_b));
    uint64_t *done = full + kMaxChunks;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int mt = (g.M + kBM - 1) / kBM, nt = (g.N + g.bn - 1) / g.bn;
    int tile = (int)blockIdx.x - g.first;
    const int m0 = tile % mt * kBM;
    tile /= mt;
    const int n0 = tile % nt * g.bn, split = tile / nt;
    const int kb = split * g.k_split;
    const int nk = max(0, min(kMaxChunks, (min(g.k_split, g.K - kb) + kBK - 1) / kBK));
    const uint32_t tmem_cols = g.bn <= 64 ? 64u : g.bn <= 128 ? 128u : 256u;

    if (threadIdx.x == 0) {
        if (blockIdx.x == 0 && t.count) *t.count += 1;
        for (int c = 0; c < kMaxChunks; c++) mbar_init(&full[c], 1);
        mbar_init(done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        for (int c = 0; c < nk; c++) mbar_expect_tx(&full[c], (uint32_t)(kStageA + stage_b));
    }
    if (warp == 0) {
        __syncwarp();
        const uint32_t lead = elect_one();
        for (int c = 0; c < nk; c++) {
            tma_load_2d(lead, smem_u32(sA + c * kStageA), &g.a, smem_u32(&full[c]), kb + c * kBK, m0);
            tma_load_2d(lead, smem_u32(sB + c * stage_b), &g.b, smem_u32(&full[c]), kb + c * kBK, n0);
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (warp == 1) {
        bool ok = true;
        const uint32_t idesc = umma_idesc(g.bn), lead = elect_one();
        for (int c = 0; c < nk; c++) {
            ok = __all_sync(0xffffffffu, mbar_wait(&full[c], 0, t.err, 1u));
            if (!ok) break;
            tc_fence_after();
            const uint64_t ad = smem_desc_sw128(smem_u32(sA + c * kStageA));
            const uint64_t bd = smem_desc_sw128(smem_u32(sB + c * stage_b));
#pragma unroll
            for (int kk = 0; kk < kBK / 16; kk++)  // 16 bf16 = 32 bytes = 2 descriptor units
                umma_bf16(lead, tmem, ad + 2 * kk, bd + 2 * kk, idesc, (c | kk) ? 1u : 0u);
        }
        // after a load that did not come, this CTA's other copies before its memory goes away
        if (!ok)
            for (int c = 0; c < nk; c++) mbar_wait(&full[c], 0, t.err, 4u);
        umma_commit(lead, done);  // arrives once every issued MMA has completed
    }
    __syncwarp();
    const bool have = mbar_wait(done, 0, t.err, 2u) && nk > 0;
    tc_fence_after();

    const int quad = warp & 3;
    const int m = m0 + quad * 32 + lane;
    if (have) {
#pragma unroll 1
        for (int cc = warp >> 2; cc * 32 < g.bn; cc += kThreads / kBM) {
            float v[32];
            tmem_ld32(tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(cc * 32), v);
            const int nb = n0 + cc * 32;
            // lane = row m: outputs indexed [n][m] are coalesced across lanes
            float *out = g.out_f32 + ((size_t)split * g.N + nb) * g.M + m;
#pragma unroll
            for (int j = 0; j < 32; j++)
                if (m < g.M && nb + j < g.N) out[(size_t)j * g.M] = v[j];
        }
    } else if (threadIdx.x == 0) {
        // bounded wait for this CTA's own copies before its memory goes away
        for (int c = 0; c < nk; c++) mbar_wait(&full[c], 0, t.err, 4u);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols));
    }
}

}  // namespace umma
}  // namespace bd
