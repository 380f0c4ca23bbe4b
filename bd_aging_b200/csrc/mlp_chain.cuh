// mlp_chain.cuh -- the surrogate's forward pass and its input-gradient chain
// in one kernel, on the sm_100a tensor cores (tcgen05, BF16 in, FP32 in
// tensor memory).
//
// Rows of the batch never mix in these GEMMs, so one CTA takes 32 rows
// through every layer without leaving the chip:
//   forward   Z_l^T = W_l H_{l-1}^T + b_l, H_l = gelu(Z_l)        (l = 0 .. L-1)
//   backward  dZ_{l-1}^T = (W_l^T dZ_l^T) * gelu'(Z_{l-1})^T      (l = L-1 .. 1)
// The features are the M of each MMA (one or two tiles of 128), the 32 rows
// its N: the whole [32][K] operand of activations or gradients is this CTA's
// own, so nothing crosses CTAs.  It sits in shared memory in the
// 128-byte-swizzled K-major layout the MMA descriptor reads.  The weights W_l
// (forward) or W_l^T (backward) stream through a ring of stages of 128 x 64 by
// TMA (no multicast), ahead of the MMAs and under the epilogues.  The
// accumulator is 128 lanes (features) by 32 columns (rows) of tensor memory a
// tile.  The input rows are drawn (or taken in order) and rounded to BF16 by
// the kernel itself, straight into the first operand; the targets are read
// where the loss gradient needs them.  The epilogue of each GEMM writes the
// next GEMM's operand (the other of two buffers) and, in training, the
// transposed copies the weight-gradient GEMMs read (H_l^T, dZ_l^T, both
// [N][M]: a thread owns one feature, so its rows are 16-byte stores) to global
// memory.  gelu'(Z) is computed beside gelu(Z), where erf is shared, and kept
// in FP32 in tensor memory (512 columns: 64 for the running accumulator, 64 a
// hidden layer).  The eighth hidden layer of a network of depth 8 has no
// columns left and keeps its gelu' in global memory.  The weight-gradient
// GEMMs reduce over the batch and stay a separate launch.
//
// What bounds it: per GEMM one chain of MMAs (about 80 cycles each: a tile's
// 4 KB of weights are read for only 32 rows), tensor-memory read, epilogue
// (hidden layers: erf and exp, about 70 instructions an element) and the next
// operand.  So the two tiles overlap: half of the warps take tile 0 while the
// MMAs of tile 1 run, and the next GEMM starts on the half of its operand that
// is ready.  At 4096 rows, 5-256x4-34, a training pass takes 31.8 us
// (40.9 before the overlap; 91.7, and 9 more to gather the rows, as clusters of
// four CTAs that shared 128 rows and exchanged 48 KB a GEMM and CTA; whole
// training step 47 us, 124 before).
//
// Warps: 16 for the epilogues, one that issues the MMAs, one that loads.
// Every mbarrier wait is bounded: on expiry the error flag is recorded, the
// remaining MMAs, loads and epilogues are skipped while every barrier is still
// passed, and the loading warp waits (bounded) for its own copies, which nobody
// else does where the MMA warp gave up (always, in its own time: a word that
// told it to, read after the block's last barrier, took 1.2 us of a step).
#pragma once
#include "umma.cuh"

namespace bd {
namespace umma {

constexpr int kChainRows = 32;              // batch rows of a CTA (N of its MMAs)
constexpr int kChainEpi = 512;              // epilogue threads: warp w reads TMEM lanes 32 (w % 4)
constexpr int kChainGroups = kChainEpi / 128;  // warps that share a quadrant of lanes
constexpr int kChainThreads = kChainEpi + 64;  // ... the MMA warp, the loading warp
constexpr int kChainMaxLayers = 9;
constexpr int kChainMaxDim = 256;           // K and N of every GEMM
constexpr int kChainMaxTiles = kChainMaxDim / kBM;
constexpr int kChainCols = kChainMaxTiles * kChainRows;       // TMEM columns of one accumulator
constexpr int kChainTmemLayers = 512 / kChainCols - 1;        // hidden layers whose gelu' stays in tensor memory
constexpr int kChainB = kChainRows * kChainMaxDim * 2;        // operand: 4 chunks of [32][64] BF16
constexpr int kChainStage = kBM * kBK * 2;                    // weights: 64 columns of a tile's 128 rows
constexpr int kChainStages = 12;
constexpr int kChainSmem = 2 * kChainB + kChainStages * kChainStage + 1024 /* align */ + 256 /* barriers, TMEM slot */;
static_assert(kChainSmem + 512 /* static */ <= 227 * 1024, "shared memory of one CTA");
constexpr int kChainWarps = kChainEpi / 32;                   // epilogue warps

struct ChainLayer {
    int K, N;                   // padded sizes of W_l [N][K]: multiples of 64, at most 256
    const float *bias;          // [N]
    float *dg;                  // training, hidden layer >= kChainTmemLayers: gelu'(Z_l) [N][M]
    __nv_bfloat16 *ht;          // training, hidden layer: H_l^T [N][M] (the next layer's input, transposed)
    __nv_bfloat16 *dzt;         // training: dZ_l^T [N][M]; the output layer's rows past n_out stay zero
};

struct ChainArgs {
    int L;                      // weight layers
    int M;                      // rows; training: a multiple of 32
    int backward;               // 1: training (loss gradient and the input-gradient chain)
    ChainLayer lay[kChainMaxLayers];
    // inputs [n_data][n_in]: row r of the batch is row r of the data, or in
    // training steps (step != nullptr) the row chain_draw gives; rows past
    // n_data read as zeros
    const float *x;
    int n_data, n_in;
    const long long *step;
    unsigned long long seed;
    __nv_bfloat16 *x0t;         // training: X0^T [K_0][M]; its rows past n_in stay zero
    const float *target;        // training: targets [n_data][n_out]
    const float *tweight;       // [N_out] loss weight per output
    int n_out;                  // live outputs
    float *y;                   // inference: outputs [M][n_out]
    float grad_scale;           // d loss / d y = grad_scale * w (y - t)
    float *loss_part;           // [M / 32]: sum w (y - t)^2 per CTA
    unsigned *err;
};

struct ChainMaps {
    CUtensorMap w[kChainMaxLayers];         // W_l [N_l][K_l], box 64 x 128
    CUtensorMap wt[kChainMaxLayers];        // W_l^T [K_l][N_l], box 64 x 128
};

// counter-based sample index (splitmix64 of seed, step, row)
__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
    x += 0x9E3779B97F4A7C15ULL;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ULL;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBULL;
    return x ^ (x >> 31);
}
__device__ __forceinline__ int chain_draw(unsigned long long seed, long long step, int row, int n_data) {
    return (int)(mix64(seed ^ mix64((unsigned long long)step * 1315423911ULL + (unsigned long long)row)) %
                 (unsigned long long)n_data);
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float *v) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const float *v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
                 "r"(__float_as_uint(v[0])), "r"(__float_as_uint(v[1])), "r"(__float_as_uint(v[2])),
                 "r"(__float_as_uint(v[3])), "r"(__float_as_uint(v[4])), "r"(__float_as_uint(v[5])),
                 "r"(__float_as_uint(v[6])), "r"(__float_as_uint(v[7]))
                 : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Byte offset in the operand of row r, column k: chunk k / 64 of [32][64]
// (4 KB), row r at 128 bytes, its 16-byte unit (k % 64) / 8 at position
// unit ^ (r % 8) -- the 128-byte swizzle of a 1024-byte-aligned buffer.
__device__ __forceinline__ uint32_t chain_b_offset(int r, int k) {
    return (uint32_t)((k >> 6) * (kChainRows * 128) + r * 128 + ((((k & 63) >> 3) ^ (r & 7)) << 4) + (k & 7) * 2);
}
__device__ __forceinline__ uint4 chain_pack8(const float *v) {
    __nv_bfloat162 p0 = __floats2bfloat162_rn(v[0], v[1]), p1 = __floats2bfloat162_rn(v[2], v[3]);
    __nv_bfloat162 p2 = __floats2bfloat162_rn(v[4], v[5]), p3 = __floats2bfloat162_rn(v[6], v[7]);
    uint4 q;
    q.x = *reinterpret_cast<uint32_t *>(&p0);
    q.y = *reinterpret_cast<uint32_t *>(&p1);
    q.z = *reinterpret_cast<uint32_t *>(&p2);
    q.w = *reinterpret_cast<uint32_t *>(&p3);
    return q;
}
// rows r0 .. r0 + 7 (r0 a multiple of 8) of column k of the operand
__device__ __forceinline__ void chain_put8(unsigned char *sB, int r0, int k, const uint4 &q) {
    unsigned char *b = sB + (k >> 6) * (kChainRows * 128) + r0 * 128 + (k & 7) * 2;
    const int unit = (k & 63) >> 3;
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int i = 0; i < 8; i++)
        *reinterpret_cast<unsigned short *>(b + i * 128 + ((unit ^ i) << 4)) =
            (unsigned short)((i & 1) ? w[i >> 1] >> 16 : w[i >> 1] & 0xffffu);
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
// An epilogue warp's columns of the next operand to the MMAs, and the
// accumulator read: the barrier of that half of the features completes with
// kChainWarps arrivals.
__device__ __forceinline__ void chain_publish(uint64_t *bar, uint32_t count, int lane) {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(bar, count);
}

// GEMM gi of the chain: forward layer gi for gi < L, then backward layer
// 2L - 1 - gi (L - 1 down to 1).  Weights [N][K]: forward W_l, backward W_l^T
// (reduction over the layer's outputs).
struct ChainStep {
    bool fwd;
    int l, K, N;
};
__device__ __forceinline__ ChainStep chain_step(const ChainArgs &g, int gi) {
    ChainStep c;
    c.fwd = gi < g.L;
    c.l = c.fwd ? gi : 2 * g.L - 1 - gi;
    c.K = c.fwd ? g.lay[c.l].K : g.lay[c.l].N;
    c.N = c.fwd ? g.lay[c.l].N : g.lay[c.l].K;
    return c;
}
__device__ __forceinline__ int chain_tiles(const ChainStep &c) { return (c.N + kBM - 1) / kBM; }

__global__ void __launch_bounds__(kChainThreads, 1)
    k_mlp_chain(const __grid_constant__ ChainMaps maps, const __grid_constant__ ChainArgs g) {
    extern __shared__ unsigned char smem_raw[];
    unsigned char *smem =
        reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    unsigned char *sB0 = smem;                // operands [2][K / 64][32][64] BF16, swizzled
    unsigned char *sW = smem + 2 * kChainB;   // ring of weight stages [128][64] BF16, swizzled
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + 2 * kChainB + kChainStages * kChainStage);  // stage loaded
    uint64_t *empty = full + kChainStages;    // stage read by its MMAs
    uint64_t *bar_d = empty + kChainStages;   // [2]: MMAs of tile 0, 1 of the current GEMM completed
    uint64_t *bar_e = bar_d + 2;              // [2]: columns 0 .. 127, 128 .. 255 of the next operand written
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bar_e + 2);
    __shared__ float red[kChainWarps];
    __shared__ int s_src[kChainRows];         // data row of each row, -1: none

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * kChainRows;
    const bool train = g.backward != 0;
    const int nG = g.L + (train ? g.L - 1 : 0);
    // tensor memory: the running accumulator, then (training) one region for
    // each hidden layer: its accumulator, replaced by gelu'
    const int n_keep = train ? min(g.L - 1, kChainTmemLayers) : 0;
    const uint32_t tmem_cols = n_keep == 0 ? 64u : n_keep == 1 ? 128u : n_keep <= 3 ? 256u : 512u;

    if (tid == 0) {
        for (int i = 0; i < 2 * kChainStages + 2; i++) mbar_init(&full[i], 1);
        mbar_init(&bar_e[0], kChainWarps);
        mbar_init(&bar_e[1], kChainWarps);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    if (warp == 2) {
        const int row = m0 + lane;
        const int src = g.step ? chain_draw(g.seed, *g.step, row, g.n_data) : row;
        s_src[lane] = src < g.n_data ? src : -1;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    float loss = 0.f;
    if (warp == kChainWarps + 1) {  // the loading warp
        const uint32_t lead = elect_one();
        int idx = 0;
        bool ok = true;
#pragma unroll 1
        for (int gi = 0; gi < nG && ok; gi++) {
            const ChainStep c = chain_step(g, gi);
            const CUtensorMap *map = c.fwd ? &maps.w[c.l] : &maps.wt[c.l];
            const int nt = chain_tiles(c);
#pragma unroll 1
            for (int tk = 0; tk < nt * (c.K / kBK); tk++, idx++) {  // tile by tile, 64 columns each
                const int t = tk / (c.K / kBK), k = tk % (c.K / kBK);
                const int s = idx % kChainStages, use = idx / kChainStages;
                ok = use == 0 ||
                     __all_sync(0xffffffffu, mbar_wait(&empty[s], (uint32_t)((use - 1) & 1), g.err, 1u));
                if (!ok) break;
                if (lead) mbar_expect_tx(&full[s], (uint32_t)kChainStage);
                __syncwarp();
                tma_load_2d(lead, smem_u32(sW + s * kChainStage), map, smem_u32(&full[s]), k * kBK, t * kBM);
            }
        }
        // the CTA's copies, before its memory goes away
        for (int i = max(0, idx - kChainStages); i < idx; i++)
            mbar_wait(&full[i % kChainStages], (uint32_t)((i / kChainStages) & 1), g.err, 4u);
    } else if (warp == kChainWarps) {  // the MMA warp
        const uint32_t lead = elect_one(), idesc = umma_idesc(kChainRows);
        int idx = 0;
        uint32_t used1 = 0;  // operands so far with a second half
        bool ok = true;
#pragma unroll 1
        for (int gi = 0; gi < nG; gi++) {
            const ChainStep c = chain_step(g, gi);
            const int nt = chain_tiles(c);
            const uint32_t acc = tmem + (c.fwd && c.l < n_keep ? (uint32_t)(kChainCols * (c.l + 1)) : 0u);
            const unsigned char *sB = sB0 + (gi & 1) * kChainB;
#pragma unroll 1
            for (int t = 0; t < nt; t++) {
#pragma unroll 1
                for (int k = 0; k < c.K / kBK; k++, idx++) {
                    // tile 0 takes each half of the operand as its epilogue warps publish
                    // it: they have also read the accumulator that this tile (half 0) and
                    // the next (half 1) overwrite
                    if (t == 0 && (k & 1) == 0 && ok) {
                        const uint32_t use = (k >> 1) ? used1++ : (uint32_t)gi;
                        ok = __all_sync(0xffffffffu, mbar_wait(&bar_e[k >> 1], use & 1u, g.err, 3u));
                    }
                    const int s = idx % kChainStages;
                    ok = ok && __all_sync(0xffffffffu, mbar_wait(&full[s], (uint32_t)((idx / kChainStages) & 1), g.err, 2u));
                    if (!ok) continue;
                    tc_fence_after();
                    const uint64_t bd = smem_desc_sw128(smem_u32(sB + k * (kChainRows * 128)));
                    const uint64_t ad = smem_desc_sw128(smem_u32(sW + s * kChainStage));
#pragma unroll
                    for (int kk = 0; kk < kBK / 16; kk++)  // 16 BF16 = 32 bytes = 2 descriptor units
                        umma_bf16(lead, acc + (uint32_t)(t * kChainRows), ad + 2 * kk, bd + 2 * kk, idesc,
                                  (k | kk) ? 1u : 0u);
                    umma_commit(lead, &empty[s]);
                }
                // arrives when every MMA issued so far has completed, also when none was issued
                umma_commit(lead, &bar_d[t]);
            }
        }
    } else {  // the epilogue warps
        const int quad = warp & 3, group = warp >> 2;
        const uint32_t quad_row = (uint32_t)(quad * 32) << 16;
        {   // X0, a thread four columns of a row; X0^T
            const int r = tid >> 4, k0 = (tid & 15) * 4, src = s_src[r];
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) v[j] = (src >= 0 && k0 + j < g.n_in) ? g.x[(size_t)src * g.n_in + k0 + j] : 0.f;
            __align__(8) __nv_bfloat162 p[2] = {__floats2bfloat162_rn(v[0], v[1]), __floats2bfloat162_rn(v[2], v[3])};
            *reinterpret_cast<uint2 *>(sB0 + chain_b_offset(r, k0)) = *reinterpret_cast<uint2 *>(p);
            if (train)
#pragma unroll
                for (int j = 0; j < 4; j++)
                    if (k0 + j < g.n_in) g.x0t[(size_t)(k0 + j) * g.M + m0 + r] = __float2bfloat16_rn(v[j]);
            chain_publish(&bar_e[0], 1, lane);
        }
        uint32_t used1 = 0;  // GEMMs so far with a second tile
#pragma unroll 1
        for (int gi = 0; gi < nG; gi++) {
            const ChainStep c = chain_step(g, gi);
            const int nt = chain_tiles(c);
            const bool out_layer = c.fwd && c.l == g.L - 1;
            const bool next = gi + 1 < nG;  // a GEMM follows that reads the operand written here
            const uint32_t acc = tmem + (c.fwd && c.l < n_keep ? (uint32_t)(kChainCols * (c.l + 1)) : 0u);
            const uint32_t keep = tmem + (uint32_t)(kChainCols * c.l);  // backward: gelu' of layer l - 1
            // warp (quad, group): features 32 quad .. + 31 of a tile (lane =
            // feature); the nt tiles' units of 8 rows, nt neighbouring units a group
            const int tile = group * nt / kChainGroups, n = tile * kBM + quad * 32 + lane;
            const bool live = tile * kBM + quad * 32 < c.N;
            // inputs that do not depend on the MMAs load under them
            const float bias = c.fwd && live ? g.lay[c.l].bias[n] : 0.f;
            float tgt[8], tw = 0.f;
            if (out_layer && train) {  // N = 128: one tile, one unit a group
                if (n < g.n_out) tw = g.tweight[n];
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const int src = s_src[group * 8 + j];
                    tgt[j] = (src >= 0 && n < g.n_out) ? g.target[(size_t)src * g.n_out + n] : 0.f;
                }
            }
            const bool ok = mbar_wait(&bar_d[tile], (tile ? used1 : (uint32_t)gi) & 1u, g.err, 2u);
            if (nt == 2) used1++;
            tc_fence_after();
            if (ok && live) {
#pragma unroll 1
                for (int i = 0; i < nt; i++) {
                    const int u = group * nt + i, r0 = (u & 3) * 8;
                    const uint32_t col = quad_row + (uint32_t)(tile * kChainRows + r0);
                    const size_t at = (size_t)n * g.M + m0 + r0;  // in the [N][M] arrays
                    float v[8];
                    tmem_ld8(acc + col, v);
                    uint4 q;
                    if (c.fwd && !out_layer) {  // hidden layer: bias, GELU and its derivative
                        const ChainLayer &Ly = g.lay[c.l];
                        if (train) {
                            float d[8];
#pragma unroll
                            for (int j = 0; j < 8; j++) gelu_both(v[j] + bias, &v[j], &d[j]);
                            if (c.l < n_keep) {
                                tmem_st8(acc + col, d);
                            } else {
#pragma unroll
                                for (int j = 0; j < 8; j++) Ly.dg[at + j] = d[j];
                            }
                            q = chain_pack8(v);
                            *reinterpret_cast<uint4 *>(Ly.ht + at) = q;
                        } else {
#pragma unroll
                            for (int j = 0; j < 8; j++) v[j] = gelu(v[j] + bias);
                            q = chain_pack8(v);
                        }
                    } else if (c.fwd) {  // output layer: y, or in training the loss gradient
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            const float y = v[j] + bias;
                            float gr = 0.f;
                            if (train) {
                                if (n < g.n_out) {
                                    const float e = y - tgt[j];
                                    loss += tw * e * e;
                                    gr = g.grad_scale * tw * e;
                                }
                            } else if (n < g.n_out && m0 + r0 + j < g.M) {
                                g.y[(size_t)(m0 + r0 + j) * g.n_out + n] = y;
                            }
                            v[j] = gr;
                        }
                        q = chain_pack8(v);
                        if (train && n < g.n_out) *reinterpret_cast<uint4 *>(g.lay[c.l].dzt + at) = q;
                    } else {  // backward: dZ_{l-1} = (dZ_l W_l) * gelu'(Z_{l-1})
                        const ChainLayer &Lp = g.lay[c.l - 1];
                        float d[8];
                        if (c.l - 1 < n_keep) {
                            tmem_ld8(keep + col, d);
                        } else {
#pragma unroll
                            for (int j = 0; j < 8; j++) d[j] = Lp.dg[at + j];
                        }
#pragma unroll
                        for (int j = 0; j < 8; j++) v[j] *= d[j];
                        q = chain_pack8(v);
                        *reinterpret_cast<uint4 *>(Lp.dzt + at) = q;
                    }
                    if (next) chain_put8(sB0 + ((gi + 1) & 1) * kChainB, r0, n, q);
                }
            }
            // two tiles: half of the warps stand for each half of the features
            if (next) chain_publish(&bar_e[tile], (uint32_t)nt, lane);
        }
        if (train) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, off);
            if (lane == 0) red[warp] = loss;
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (train && tid == 0) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < kChainWarps; w++) t += red[w];
        g.loss_part[blockIdx.x] = t;
    }
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tmem_cols));
    }
}

}  // namespace umma
}  // namespace bd
