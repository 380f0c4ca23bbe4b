// surrogate.cu -- the learned surrogate: an MLP n_in -> width (GELU) x depth
// -> n_out trained and evaluated by hand-written tcgen05 BF16 GEMMs with FP32
// accumulation, Adam in FP32 on FP32 master weights.
//
// Per layer l (K_l inputs, N_l outputs, batch B) every GEMM has both
// operands K-major; the transposed copies it needs are written by the
// epilogue or the optimizer that produces them:
//   forward   Z_l  = H_{l-1} W_l^T + b_l        A = H_{l-1} [B][K_l], B = W_l  [N_l][K_l]
//   input     dH_{l-1} = dZ_l W_l               A = dZ_l    [B][N_l], B = W_l^T [K_l][N_l]
//   weights   dW_l = dZ_l^T H_{l-1}             A = dZ_l^T  [N_l][B], B = H_{l-1}^T [K_l][B]
// A training step is three launches: the fused kernel (mlp_chain.cuh) draws
// the minibatch and runs every forward and input-gradient GEMM, keeping each
// 32-row block's activations and gradients on chip and writing H_l^T and
// dZ_l^T; one launch runs every weight-gradient GEMM (umma.cuh); one launch
// sums the bias gradients and applies Adam.  dW is split over the batch (256
// rows per CTA) into FP32 partials that the Adam kernel adds in a fixed
// order, so a training step is deterministic.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>

#include "mlp_chain.cuh"
#include "runtime.cuh"
#include "umma.cuh"

namespace bd {
namespace {

using umma::GemmJob;
using umma::GemmTable;
using umma::kBK;
using umma::kBM;
using umma::kBN;

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static bool tried = false;
    if (!tried) {
        tried = true;
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(p);
    }
    return fn;
}

// 2-D BF16 row-major matrix [rows][cols] as a TMA map with a box of 64
// columns (128 bytes, 128-byte swizzle) by box_rows rows (kBM for A
// operands, the tile width for B operands); out-of-range rows and columns read as zero.
int make_tmap(CUtensorMap *map, const void *ptr, int rows, int cols, int box_rows) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return BD_ERR_CUDA;
    if ((reinterpret_cast<uintptr_t>(ptr) & 15) || (cols % 8)) return BD_ERR_ARG;
    cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    cuuint32_t box[2] = {(cuuint32_t)kBK, (cuuint32_t)box_rows};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? BD_OK : BD_ERR_ARG;
}

// dynamic shared memory above 48 KB for the GEMM and the fused kernel;
// called outside stream capture (create, direct GEMM)
int set_gemm_attrs() {
    BD_CUDA_TRY(cudaFuncSetAttribute(umma::k_umma_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     umma::gemm_smem(umma::kMaxBN)));
    BD_CUDA_TRY(cudaFuncSetAttribute(umma::k_mlp_chain, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     umma::kChainSmem));
    return BD_OK;
}

// the table's GEMMs side by side; fills in each job's first block
int launch_gemms(GemmTable &t, cudaStream_t st) {
    int blocks = 0, bn = 0;
    for (int i = 0; i < t.n_jobs; i++) {
        GemmJob &g = t.job[i];
        if (g.k_split % kBK || g.k_split > umma::kMaxChunks * kBK || g.k_split < kBK) return BD_ERR_ARG;
        if (g.bn % kBN || g.bn < kBN || g.bn > umma::kMaxBN) return BD_ERR_ARG;
        const long long n = (long long)div_up(g.M, kBM) * div_up(g.N, g.bn) * div_up(g.K, g.k_split);
        if (n > 0x7fffffffLL - blocks) return BD_ERR_ARG;
        g.first = blocks;
        blocks += (int)n;
        bn = std::max(bn, g.bn);
    }
    umma::k_umma_gemm<<<blocks, umma::kThreads, umma::gemm_smem(bn), st>>>(t);
    BD_LAUNCH_CHECK();
    return BD_OK;
}

// ---------------------------------------------------------------- kernels
__global__ void k_sum_splits(const float *part, int splits, size_t n, float *out) {
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float s = 0.f;
    for (int k = 0; k < splits; k++) s += part[(size_t)k * n + i];
    out[i] = s;
}

// Bias gradients: row n of layer l's dZ_l^T summed over the batch by one warp,
// in the fixed order of eight strided slices (16-byte loads), each a shuffle
// tree, added in turn.  The slices are independent chains, which keeps enough
// loads in flight for one warp.
struct BiasGradArgs {
    const __nv_bfloat16 *dzt[umma::kChainMaxLayers];  // [N_l][B]
    float *db[umma::kChainMaxLayers];                 // [N_l]
    int first[umma::kChainMaxLayers + 1];             // first row of each layer
    int L, B;                                         // B a multiple of 8
};
constexpr int kBiasSlices = 8;
__device__ __forceinline__ float bias_row_sum(const __nv_bfloat16 *row, int B, int lane) {
    const uint4 *src = reinterpret_cast<const uint4 *>(row);
    float sum[kBiasSlices];
#pragma unroll
    for (int w = 0; w < kBiasSlices; w++) sum[w] = 0.f;
    for (int i0 = 0; i0 < B / 8; i0 += 32 * kBiasSlices) {
        uint4 v[kBiasSlices];
#pragma unroll
        for (int w = 0; w < kBiasSlices; w++) {
            const int i = i0 + w * 32 + lane;
            v[w] = i < B / 8 ? src[i] : make_uint4(0u, 0u, 0u, 0u);
        }
#pragma unroll
        for (int w = 0; w < kBiasSlices; w++) {
            const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&v[w]);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float2 f = __bfloat1622float2(h[j]);
                sum[w] += f.x;
                sum[w] += f.y;
            }
        }
    }
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kBiasSlices; w++) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sum[w] += __shfl_down_sync(0xffffffffu, sum[w], off);
        t += sum[w];
    }
    return t;  // of lane 0
}
__device__ __forceinline__ int layer_of_row(const int *first, int L, int row) {
    int l = 0;
    while (l + 1 < L && row >= first[l + 1]) l++;
    return l;
}
constexpr int kBiasRows = 8;  // rows (warps) per block
__global__ void k_bias_grads(const __grid_constant__ BiasGradArgs a) {
    const int row = blockIdx.x * kBiasRows + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= a.first[a.L]) return;
    const int l = layer_of_row(a.first, a.L, row), n = row - a.first[l];
    const float g = bias_row_sum(a.dzt[l] + (size_t)n * a.B, a.B, lane);
    if (lane == 0) a.db[l][n] = g;
}

struct AdamArgs {
    float lr, b1, b2, eps;
    const long long *step;  // number of this update (1 for the first)
};
// Every layer's weights and biases in one launch.  The first blocks take tiles
// of 16 k by 64 n of the weights of layer 0, 1, ...: the gradient is the sum of
// the split partials, stored [splits][K][N] by the weight-gradient GEMM, and
// the FP32 master weights and moments are kept in that order too, so a thread's
// four n are one 16-byte access each.  It writes the BF16 copies W^T [K][N]
// directly and W [N][K] through shared memory in 32-byte runs (written lane by
// lane, each 2-byte store touched a sector of its own).  The other blocks sum
// eight bias gradients each, a warp a row, and update the biases.
// What bounds it: the partials, 14.7 MB at the 256-wide network and a batch of
// 4096, which the GEMM has just left in L2.
// 9.1 us at that size (before: 13, and 5 and 2.5 for the bias sums' and the
// step counter's own launches).
constexpr int kAdamK = 16, kAdamN = 64;
struct AdamTable {
    float *w[umma::kChainMaxLayers], *wm[umma::kChainMaxLayers], *wv[umma::kChainMaxLayers];
    const float *part[umma::kChainMaxLayers];
    __nv_bfloat16 *wb[umma::kChainMaxLayers], *wbt[umma::kChainMaxLayers];
    float *b[umma::kChainMaxLayers], *bm[umma::kChainMaxLayers], *bv[umma::kChainMaxLayers];
    int N[umma::kChainMaxLayers], K[umma::kChainMaxLayers];
    int n_live[umma::kChainMaxLayers], k_live[umma::kChainMaxLayers];
    int first_w[umma::kChainMaxLayers + 1];  // first weight tile of each layer
    int L, splits;
    BiasGradArgs bias;                       // db unused
};
__device__ __forceinline__ float adam_update(const AdamArgs &a, const float *corr, float w, float g, float &m, float &v) {
    m = a.b1 * m + (1.f - a.b1) * g;
    v = a.b2 * v + (1.f - a.b2) * g * g;
    const float mh = m / corr[0], vh = v / corr[1];
    return w - a.lr * mh / (sqrtf(vh) + a.eps);
}
__global__ void __launch_bounds__(256) k_adam_all(const __grid_constant__ AdamTable t, AdamArgs a) {
    __shared__ float corr[2];
    __shared__ __nv_bfloat16 tile[kAdamK][kAdamN + 2];
    if (threadIdx.x < 2) corr[threadIdx.x] = 1.f - powf(threadIdx.x ? a.b2 : a.b1, (float)*a.step);
    const int tiles = t.first_w[t.L];
    if ((int)blockIdx.x < tiles) {
        const int l = layer_of_row(t.first_w, t.L, blockIdx.x);
        const int N = t.N[l], K = t.K[l], ti = blockIdx.x - t.first_w[l];
        const int k0 = ti / (N / kAdamN) * kAdamK, n0 = ti % (N / kAdamN) * kAdamN;
        const int kk = threadIdx.x >> 4, nn = (threadIdx.x & 15) * 4, k = k0 + kk, n = n0 + nn;
        const size_t i = (size_t)k * N + n;
        const float *part = t.part[l] + i;
        float g[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 8
        for (int s = 0; s < t.splits; s++) {
            const float4 p = *reinterpret_cast<const float4 *>(part + (size_t)s * N * K);
            g[0] += p.x;
            g[1] += p.y;
            g[2] += p.z;
            g[3] += p.w;
        }
        __align__(16) float w[4], m[4], v[4];
        *reinterpret_cast<float4 *>(w) = *reinterpret_cast<const float4 *>(t.w[l] + i);
        *reinterpret_cast<float4 *>(m) = *reinterpret_cast<const float4 *>(t.wm[l] + i);
        *reinterpret_cast<float4 *>(v) = *reinterpret_cast<const float4 *>(t.wv[l] + i);
        __syncthreads();
        if (k < t.k_live[l]) {
#pragma unroll
            for (int j = 0; j < 4; j++)
                if (n + j < t.n_live[l]) w[j] = adam_update(a, corr, w[j], g[j], m[j], v[j]);
            *reinterpret_cast<float4 *>(t.w[l] + i) = *reinterpret_cast<float4 *>(w);
            *reinterpret_cast<float4 *>(t.wm[l] + i) = *reinterpret_cast<float4 *>(m);
            *reinterpret_cast<float4 *>(t.wv[l] + i) = *reinterpret_cast<float4 *>(v);
        }
        __align__(8) __nv_bfloat162 q[2] = {__floats2bfloat162_rn(w[0], w[1]), __floats2bfloat162_rn(w[2], w[3])};
        *reinterpret_cast<uint2 *>(t.wbt[l] + i) = *reinterpret_cast<uint2 *>(q);
        *reinterpret_cast<__nv_bfloat162 *>(&tile[kk][nn]) = q[0];
        *reinterpret_cast<__nv_bfloat162 *>(&tile[kk][nn + 2]) = q[1];
        __syncthreads();
        const int tn = threadIdx.x >> 2, tk = (threadIdx.x & 3) * 4;
        __nv_bfloat16 o[4];
#pragma unroll
        for (int j = 0; j < 4; j++) o[j] = tile[tk + j][tn];
        __align__(8) __nv_bfloat162 oq[2] = {__nv_bfloat162(o[0], o[1]), __nv_bfloat162(o[2], o[3])};
        *reinterpret_cast<uint2 *>(t.wb[l] + (size_t)(n0 + tn) * K + k0 + tk) = *reinterpret_cast<uint2 *>(oq);
        return;
    }
    __syncthreads();
    const int row = ((int)blockIdx.x - tiles) * kBiasRows + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (row >= t.bias.first[t.L]) return;
    const int l = layer_of_row(t.bias.first, t.L, row), n = row - t.bias.first[l];
    if (n >= t.n_live[l]) return;
    const float g = bias_row_sum(t.bias.dzt[l] + (size_t)n * t.bias.B, t.bias.B, lane);
    if (lane == 0) {
        float m = t.bm[l][n], v = t.bv[l][n];
        t.b[l][n] = adam_update(a, corr, t.b[l][n], g, m, v);
        t.bm[l][n] = m;
        t.bv[l][n] = v;
    }
}
// BF16 copies W [N][K] and W^T [K][N] of the FP32 master weights (kept [K][N])
__global__ void k_to_bf16(const float *w, int N, int K, __nv_bfloat16 *wb, __nv_bfloat16 *wbt) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;  // [k][n] order
    if (i >= (size_t)N * K) return;
    const int k = (int)(i / N), n = (int)(i % N);
    const __nv_bfloat16 b = __float2bfloat16_rn(w[i]);
    wb[(size_t)n * K + k] = b;
    wbt[i] = b;
}

// The flat host order (for each layer W [N_l][K_l] then b [N_l], live sizes)
// of the parameters, or of the gradients (sums of the split partials), written
// on the device, so that one copy of the live values replaces a padded copy
// and a host transpose a layer.  Element order [k][n]: reads coalesce.
struct FlatTable {
    const float *w[umma::kChainMaxLayers];   // [splits][K][N]
    const float *b[umma::kChainMaxLayers];
    int N[umma::kChainMaxLayers], K[umma::kChainMaxLayers];
    int n_live[umma::kChainMaxLayers], k_live[umma::kChainMaxLayers];
    int out[umma::kChainMaxLayers];          // first flat element of the layer
    int first[umma::kChainMaxLayers + 1];    // prefix of (K + 1) N: the weights, then the biases
    int L, splits;
};
__global__ void k_flatten(const __grid_constant__ FlatTable t, float *flat) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= t.first[t.L]) return;
    const int l = layer_of_row(t.first, t.L, e), i = e - t.first[l];
    const int N = t.N[l], K = t.K[l], k = i / N, n = i % N;
    if (n >= t.n_live[l]) return;
    float *out = flat + t.out[l];
    if (k == K) {
        out[(size_t)t.n_live[l] * t.k_live[l] + n] = t.b[l][n];
    } else if (k < t.k_live[l]) {
        float s = 0.f;
        for (int j = 0; j < t.splits; j++) s += t.w[l][(size_t)j * N * K + i];
        out[(size_t)n * t.k_live[l] + k] = s;
    }
}

}  // namespace
}  // namespace bd

using namespace bd;

// ---------------------------------------------------------------- state
struct bd_surrogate {
    int n_in = 0, n_out = 0, width = 0, depth = 0, batch = 0;
    int L = 0;                        // weight layers = depth + 1
    std::vector<int> Kp, Np;          // padded input / output sizes per layer
    std::vector<int> Kl, Nl;          // live sizes
    cudaStream_t stream = nullptr;
    // parameters (FP32 master weights [K][N] and Adam moments in that order, biases), BF16 copies
    std::vector<float *> w, b, wm, wv, bm, bv;
    std::vector<__nv_bfloat16 *> wb, wbt;
    // activations and gradients the weight-gradient GEMMs read
    std::vector<__nv_bfloat16 *> ht;      // ht[0] = X0^T; ht[l+1] = H_l^T, output of hidden layer l [N_l][B]
    std::vector<float *> dg;              // gelu'(Z_l) [N_l][B] of the hidden layers tensor memory has no room for
    std::vector<__nv_bfloat16 *> dzt;     // dZ_l^T, gradient w.r.t. z[l] [N_l][B]
    float *tw = nullptr;                  // loss weight per output
    float *part = nullptr;            // weight-gradient split partials [splits][K_l][N_l] per layer
    std::vector<float *> db;          // bias gradients
    float *flat = nullptr;            // parameters or gradients in the flat host order
    long long *step = nullptr;
    // loss partials, then the error flag, copied together to the pinned words
    float *loss_part = nullptr;
    unsigned *err = nullptr;
    float *host = nullptr;
    // inputs and outputs of predict and gradients on the device, kept (pred_rows rows)
    float *px = nullptr, *py = nullptr;
    int pred_rows = 0;
    float *data_x = nullptr, *data_y = nullptr;
    int n_data = 0;
    unsigned long long seed = 1;
    // TMA maps: the weight-gradient GEMMs' operands dZ_l^T and H_{l-1}^T, and
    // the fused kernel's W_l, W_l^T
    std::vector<CUtensorMap> tm_ht, tm_dzt, tm_w, tm_wt;
    float lr = 1e-3f;
    int loss_cells = 0;
    int ksplit = 256;
};

namespace {

void free_surrogate(bd_surrogate *s) {
    auto F = [](void *p) {
        if (p) cudaFree(p);
    };
    for (auto *p : s->w) F(p);
    for (auto *p : s->b) F(p);
    for (auto *p : s->wm) F(p);
    for (auto *p : s->wv) F(p);
    for (auto *p : s->bm) F(p);
    for (auto *p : s->bv) F(p);
    for (auto *p : s->wb) F(p);
    for (auto *p : s->wbt) F(p);
    for (auto *p : s->ht) F(p);
    for (auto *p : s->dg) F(p);
    for (auto *p : s->dzt) F(p);
    for (auto *p : s->db) F(p);
    F(s->tw); F(s->part); F(s->flat); F(s->step); F(s->loss_part); F(s->data_x); F(s->data_y); F(s->px); F(s->py);
    if (s->host) cudaFreeHost(s->host);
    if (s->stream) cudaStreamDestroy(s->stream);
    delete s;
}

// waits for the stream's work; the loss partials and the error flag come over
// in one copy to pinned memory
int sg_finish(bd_surrogate *s, double *loss_sum) {
    BD_CUDA_TRY(cudaMemcpyAsync(s->host, s->loss_part, (size_t)(s->loss_cells + 1) * 4, cudaMemcpyDeviceToHost,
                                s->stream));
    BD_CUDA_TRY(cudaStreamSynchronize(s->stream));
    if (loss_sum) {
        double sum = 0;
        for (int i = 0; i < s->loss_cells; i++) sum += s->host[i];
        *loss_sum = sum;
    }
    unsigned e;
    std::memcpy(&e, s->host + s->loss_cells, 4);
    return e ? BD_ERR_TIMEOUT : BD_OK;
}

// The fused kernel (a CTA per 32 rows): training (`train`)
// on the batch, from the training set (`draw`) or from rows in order, with the
// loss gradient and every dZ_l; or the outputs y of `rows` rows of x.
int chain_launch(bd_surrogate *s, bool train, bool draw, const float *x, const float *target, int rows, float *y) {
    umma::ChainMaps maps;
    std::memset(&maps, 0, sizeof(maps));
    umma::ChainArgs g;
    std::memset(&g, 0, sizeof(g));
    g.L = s->L;
    g.M = train ? s->batch : rows;
    g.backward = train ? 1 : 0;
    for (int l = 0; l < s->L; l++) {
        maps.w[l] = s->tm_w[l];
        maps.wt[l] = s->tm_wt[l];
        g.lay[l] = {s->Kp[l], s->Np[l], s->b[l], s->dg[l], l < s->L - 1 ? s->ht[l + 1] : nullptr, s->dzt[l]};
    }
    g.x = x;
    g.n_data = rows;
    g.n_in = s->n_in;
    g.step = draw ? s->step : nullptr;
    g.seed = s->seed;
    g.n_out = s->n_out;
    g.y = y;
    if (train) {
        g.x0t = s->ht[0];
        g.target = target;
        g.tweight = s->tw;
        g.grad_scale = 2.0f / ((float)s->batch * (float)s->n_out);
        g.loss_part = s->loss_part;
    }
    g.err = s->err;
    umma::k_mlp_chain<<<div_up(g.M, umma::kChainRows), umma::kChainThreads, umma::kChainSmem, s->stream>>>(maps, g);
    BD_LAUNCH_CHECK();
    return BD_OK;
}

size_t part_offset(const bd_surrogate *s, int l) {
    size_t off = 0;
    for (int i = 0; i < l; i++) off += (size_t)(s->batch / s->ksplit) * s->Np[i] * s->Kp[i];
    return off;
}

// weight gradients dW_l = dZ_l^T H_{l-1} of every layer, as split partials at
// part + part_offset(l); `count` also counts the training step
int weight_grads(bd_surrogate *s, bool count) {
    GemmTable t;
    std::memset(&t, 0, sizeof(t));
    t.n_jobs = s->L;
    t.count = count ? s->step : nullptr;
    t.err = s->err;
    for (int l = 0; l < s->L; l++) {
        GemmJob &g = t.job[l];
        g.a = s->tm_dzt[l];
        g.b = s->tm_ht[l];
        g.out_f32 = s->part + part_offset(s, l);
        g.M = s->Np[l];
        g.N = s->Kp[l];
        g.K = s->batch;
        g.k_split = s->ksplit;
        g.bn = s->Kp[l];
    }
    return launch_gemms(t, s->stream);
}

BiasGradArgs bias_args(const bd_surrogate *s) {
    BiasGradArgs a;
    std::memset(&a, 0, sizeof(a));
    a.L = s->L;
    a.B = s->batch;
    for (int l = 0; l < s->L; l++) {
        a.dzt[l] = s->dzt[l];
        a.db[l] = s->db[l];
        a.first[l + 1] = a.first[l] + s->Np[l];
    }
    return a;
}

int adam(bd_surrogate *s) {
    AdamArgs a{s->lr, 0.9f, 0.999f, 1e-8f, s->step};
    AdamTable t;
    std::memset(&t, 0, sizeof(t));
    t.L = s->L;
    t.splits = s->batch / s->ksplit;
    t.bias = bias_args(s);
    for (int l = 0; l < s->L; l++) {
        t.w[l] = s->w[l];
        t.wm[l] = s->wm[l];
        t.wv[l] = s->wv[l];
        t.part[l] = s->part + part_offset(s, l);
        t.wb[l] = s->wb[l];
        t.wbt[l] = s->wbt[l];
        t.b[l] = s->b[l];
        t.bm[l] = s->bm[l];
        t.bv[l] = s->bv[l];
        t.N[l] = s->Np[l];
        t.K[l] = s->Kp[l];
        t.n_live[l] = s->Nl[l];
        t.k_live[l] = s->Kl[l];
        t.first_w[l + 1] = t.first_w[l] + s->Np[l] / kAdamN * (s->Kp[l] / kAdamK);
    }
    k_adam_all<<<t.first_w[s->L] + div_up(t.bias.first[s->L], kBiasRows), 256, 0, s->stream>>>(t, a);
    BD_LAUNCH_CHECK();
    return BD_OK;
}

// the flat host order of the parameters or (gradients) of the last backward pass
int flatten(bd_surrogate *s, bool gradients, float *out) {
    FlatTable t;
    std::memset(&t, 0, sizeof(t));
    t.L = s->L;
    t.splits = gradients ? s->batch / s->ksplit : 1;
    int off = 0;
    for (int l = 0; l < s->L; l++) {
        t.w[l] = gradients ? s->part + part_offset(s, l) : s->w[l];
        t.b[l] = gradients ? s->db[l] : s->b[l];
        t.N[l] = s->Np[l];
        t.K[l] = s->Kp[l];
        t.n_live[l] = s->Nl[l];
        t.k_live[l] = s->Kl[l];
        t.out[l] = off;
        off += s->Nl[l] * (s->Kl[l] + 1);
        t.first[l + 1] = t.first[l] + s->Np[l] * (s->Kp[l] + 1);
    }
    k_flatten<<<div_up(t.first[s->L], 256), 256, 0, s->stream>>>(t, s->flat);
    BD_LAUNCH_CHECK();
    BD_CUDA_TRY(cudaMemcpyAsync(out, s->flat, (size_t)off * 4, cudaMemcpyDeviceToHost, s->stream));
    return BD_OK;
}

// device rows for predict and gradients; grows, freed with the object
int io_rows(bd_surrogate *s, int rows) {
    if (rows <= s->pred_rows) return BD_OK;
    if (s->px) cudaFree(s->px);
    if (s->py) cudaFree(s->py);
    s->px = s->py = nullptr;
    s->pred_rows = 0;
    BD_CUDA_TRY(cudaMalloc(&s->px, (size_t)rows * s->n_in * 4));
    BD_CUDA_TRY(cudaMalloc(&s->py, (size_t)rows * s->n_out * 4));
    s->pred_rows = rows;
    return BD_OK;
}
constexpr int kPredictRows = 32768;  // rows predict keeps on the device at a time

}  // namespace

extern "C" {

int bd_surrogate_create(int n_in, int n_out, int width, int depth, int batch, unsigned long long seed,
                        bd_surrogate **out) {
    if (!out || n_in < 1 || n_in > 64 || n_out < 1 || n_out > 128 || width < 64 || width > 256 || width % 64 ||
        depth < 1 || depth > 8 || batch < 256 || batch % 256)
        return BD_ERR_ARG;
    bd_surrogate *s = new (std::nothrow) bd_surrogate();
    if (!s) return BD_ERR_NOMEM;
    s->n_in = n_in;
    s->n_out = n_out;
    s->width = width;
    s->depth = depth;
    s->batch = batch;
    s->seed = seed;
    s->L = depth + 1;
    for (int l = 0; l < s->L; l++) {
        s->Kl.push_back(l == 0 ? n_in : width);
        s->Kp.push_back(l == 0 ? 64 : width);
        s->Nl.push_back(l == s->L - 1 ? n_out : width);
        s->Np.push_back(l == s->L - 1 ? 128 : width);
    }
    // the fused forward / input-gradient kernel covers every shape accepted here
    static_assert(8 + 1 <= umma::kChainMaxLayers && 256 % kBM == 0, "depth <= 8, batch a multiple of 256");
    if (set_gemm_attrs() != BD_OK || cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete s;
        return BD_ERR_CUDA;
    }
    bool ok = true;
    auto A = [&](void **p, size_t bytes) {
        if (ok && cudaMalloc(p, bytes) != cudaSuccess) ok = false;
        if (ok) cudaMemsetAsync(*p, 0, bytes, s->stream);
    };
    size_t part_total = 0;
    for (int l = 0; l < s->L; l++) {
        const size_t nk = (size_t)s->Np[l] * s->Kp[l];
        float *p;
        __nv_bfloat16 *q;
        A((void **)&p, nk * 4); s->w.push_back(p);
        A((void **)&p, nk * 4); s->wm.push_back(p);
        A((void **)&p, nk * 4); s->wv.push_back(p);
        A((void **)&p, s->Np[l] * 4); s->b.push_back(p);
        A((void **)&p, s->Np[l] * 4); s->bm.push_back(p);
        A((void **)&p, s->Np[l] * 4); s->bv.push_back(p);
        A((void **)&p, s->Np[l] * 4); s->db.push_back(p);
        A((void **)&q, nk * 2); s->wb.push_back(q);
        A((void **)&q, nk * 2); s->wbt.push_back(q);
        A((void **)&q, (size_t)batch * s->Kp[l] * 2); s->ht.push_back(q);
        p = nullptr;
        if (l >= umma::kChainTmemLayers && l < s->L - 1) A((void **)&p, (size_t)batch * s->Np[l] * 4);
        s->dg.push_back(p);
        A((void **)&q, (size_t)batch * s->Np[l] * 2); s->dzt.push_back(q);
        part_total += (size_t)(batch / s->ksplit) * nk;
    }
    A((void **)&s->tw, 128 * 4);
    A((void **)&s->part, part_total * 4);
    // loss partials: one per CTA of the fused kernel
    s->loss_cells = batch / umma::kChainRows;
    A((void **)&s->loss_part, (size_t)(s->loss_cells + 1) * 4);
    s->err = reinterpret_cast<unsigned *>(s->loss_part + s->loss_cells);
    A((void **)&s->step, sizeof(long long));
    size_t n_param = 0;
    for (int l = 0; l < s->L; l++) n_param += (size_t)s->Nl[l] * (s->Kl[l] + 1);
    A((void **)&s->flat, n_param * 4);
    if (ok && cudaMallocHost(&s->host, (size_t)(s->loss_cells + 1) * 4) != cudaSuccess) ok = false;
    if (!ok) {
        free_surrogate(s);
        return BD_ERR_NOMEM;
    }
    // He-style initialisation on the host (deterministic), biases zero
    unsigned long long st = seed * 6364136223846793005ULL + 1442695040888963407ULL;
    auto rnd = [&]() {
        st = st * 6364136223846793005ULL + 1442695040888963407ULL;
        return ((st >> 11) * (1.0 / 9007199254740992.0)) * 2.0 - 1.0;  // uniform(-1, 1)
    };
    for (int l = 0; l < s->L; l++) {
        std::vector<float> hw((size_t)s->Np[l] * s->Kp[l], 0.f);
        const double scale = std::sqrt(6.0 / (double)s->Kl[l]);
        for (int n = 0; n < s->Nl[l]; n++)
            for (int k = 0; k < s->Kl[l]; k++) hw[(size_t)k * s->Np[l] + n] = (float)(scale * rnd() * 0.5);
        cudaMemcpyAsync(s->w[l], hw.data(), hw.size() * 4, cudaMemcpyHostToDevice, s->stream);
        k_to_bf16<<<div_up((long)hw.size(), 256), 256, 0, s->stream>>>(s->w[l], s->Np[l], s->Kp[l], s->wb[l],
                                                                       s->wbt[l]);
    }
    std::vector<float> ones(128, 1.f);
    cudaMemcpyAsync(s->tw, ones.data(), 128 * 4, cudaMemcpyHostToDevice, s->stream);
    // tensor maps
    int rc = BD_OK;
    s->tm_ht.resize(s->L);
    s->tm_dzt.resize(s->L);
    s->tm_w.resize(s->L);
    s->tm_wt.resize(s->L);
    for (int l = 0; l < s->L && !rc; l++) {
        // weight gradient: A = dZ_l^T, B = H_{l-1}^T; fused kernel: W_l and W_l^T
        rc |= make_tmap(&s->tm_dzt[l], s->dzt[l], s->Np[l], batch, kBM);
        rc |= make_tmap(&s->tm_ht[l], s->ht[l], s->Kp[l], batch, s->Kp[l]);
        rc |= make_tmap(&s->tm_w[l], s->wb[l], s->Np[l], s->Kp[l], kBM);
        rc |= make_tmap(&s->tm_wt[l], s->wbt[l], s->Kp[l], s->Np[l], kBM);
    }
    if (rc || cudaStreamSynchronize(s->stream) != cudaSuccess) {
        free_surrogate(s);
        return rc ? rc : BD_ERR_CUDA;
    }
    *out = s;
    return BD_OK;
}

int bd_surrogate_destroy(bd_surrogate *s) {
    if (!s) return BD_ERR_ARG;
    cudaStreamSynchronize(s->stream);
    free_surrogate(s);
    return BD_OK;
}

int bd_surrogate_get_stream(const bd_surrogate *s, void **stream) {
    if (!s || !stream) return BD_ERR_ARG;
    *stream = (void *)s->stream;
    return BD_OK;
}

int bd_surrogate_param_count(const bd_surrogate *s, long long *count) {
    if (!s || !count) return BD_ERR_ARG;
    long long c = 0;
    for (int l = 0; l < s->L; l++) c += (long long)s->Nl[l] * s->Kl[l] + s->Nl[l];
    *count = c;
    return BD_OK;
}

// Parameters as a flat FP32 vector: for each layer W [N_l][K_l] then b [N_l].
int bd_surrogate_get_params(bd_surrogate *s, float *out) {
    if (!s || !out) return BD_ERR_ARG;
    const int rc = flatten(s, false, out);
    if (rc) return rc;
    BD_CUDA_TRY(cudaStreamSynchronize(s->stream));
    return BD_OK;
}

int bd_surrogate_set_params(bd_surrogate *s, const float *in) {
    if (!s || !in) return BD_ERR_ARG;
    size_t off = 0;
    for (int l = 0; l < s->L; l++) {
        std::vector<float> hw((size_t)s->Np[l] * s->Kp[l], 0.f), hb(s->Np[l], 0.f);
        for (int n = 0; n < s->Nl[l]; n++)
            for (int k = 0; k < s->Kl[l]; k++) hw[(size_t)k * s->Np[l] + n] = in[off++];  // master kept [K][N]
        for (int n = 0; n < s->Nl[l]; n++) hb[n] = in[off++];
        BD_CUDA_TRY(cudaMemcpyAsync(s->w[l], hw.data(), hw.size() * 4, cudaMemcpyHostToDevice, s->stream));
        BD_CUDA_TRY(cudaMemcpyAsync(s->b[l], hb.data(), hb.size() * 4, cudaMemcpyHostToDevice, s->stream));
        k_to_bf16<<<div_up((long)hw.size(), 256), 256, 0, s->stream>>>(s->w[l], s->Np[l], s->Kp[l], s->wb[l],
                                                                       s->wbt[l]);
        BD_LAUNCH_CHECK();
    }
    BD_CUDA_TRY(cudaStreamSynchronize(s->stream));
    return BD_OK;
}

// Loss weight per output (default 1).
int bd_surrogate_set_output_weights(bd_surrogate *s, const float *w) {
    if (!s || !w) return BD_ERR_ARG;
    std::vector<float> hw(128, 0.f);
    for (int i = 0; i < s->n_out; i++) hw[i] = w[i];
    BD_CUDA_TRY(cudaMemcpyAsync(s->tw, hw.data(), 128 * 4, cudaMemcpyHostToDevice, s->stream));
    BD_CUDA_TRY(cudaStreamSynchronize(s->stream));
    return BD_OK;
}

// Training set on the device: x [n][n_in], y [n][n_out] (host, FP32).
int bd_surrogate_set_data(bd_surrogate *s, const float *x, const float *y, int n) {
    if (!s || !x || !y || n < 1) return BD_ERR_ARG;
    if (s->data_x) cudaFree(s->data_x);
    if (s->data_y) cudaFree(s->data_y);
    s->data_x = s->data_y = nullptr;
    BD_CUDA_TRY(cudaMalloc(&s->data_x, (size_t)n * s->n_in * 4));
    BD_CUDA_TRY(cudaMalloc(&s->data_y, (size_t)n * s->n_out * 4));
    BD_CUDA_TRY(cudaMemcpyAsync(s->data_x, x, (size_t)n * s->n_in * 4, cudaMemcpyHostToDevice, s->stream));
    BD_CUDA_TRY(cudaMemcpyAsync(s->data_y, y, (size_t)n * s->n_out * 4, cudaMemcpyHostToDevice, s->stream));
    BD_CUDA_TRY(cudaStreamSynchronize(s->stream));
    s->n_data = n;
    return BD_OK;
}

// `steps` Adam steps on random minibatches (with replacement) of the
// training set, three launches each; mean loss of the last step.
int bd_surrogate_train(bd_surrogate *s, int steps, float lr, float *last_loss) {
    if (!s || steps < 0 || !(lr > 0.f)) return BD_ERR_ARG;
    if (!s->data_x) return BD_ERR_STATE;
    s->lr = lr;
    for (int i = 0; i < steps; i++) {
        int rc = chain_launch(s, true, true, s->data_x, s->data_y, s->n_data, nullptr);
        if (!rc) rc = weight_grads(s, true);
        if (!rc) rc = adam(s);
        if (rc) return rc;
    }
    double sum = 0;
    const int rc = sg_finish(s, &sum);
    if (last_loss) *last_loss = (float)(sum / ((double)s->batch * s->n_out));
    return rc;
}

}  // extern "C"

namespace {

// the work of bd_surrogate_gradients and bd_surrogate_predict, which wait for
// the stream also where it fails: copies from and to the caller's arrays may be
// in flight
int gradients_of(bd_surrogate *s, const float *x, const float *y, float *grad, double *sum) {
    const int B = s->batch;
    int rc = io_rows(s, B);
    if (rc) return rc;
    BD_CUDA_TRY(cudaMemcpyAsync(s->px, x, (size_t)B * s->n_in * 4, cudaMemcpyHostToDevice, s->stream));
    BD_CUDA_TRY(cudaMemcpyAsync(s->py, y, (size_t)B * s->n_out * 4, cudaMemcpyHostToDevice, s->stream));
    rc = chain_launch(s, true, false, s->px, s->py, B, nullptr);
    if (!rc) rc = weight_grads(s, false);
    if (rc) return rc;
    const BiasGradArgs a = bias_args(s);
    k_bias_grads<<<div_up(a.first[s->L], kBiasRows), kBiasRows * 32, 0, s->stream>>>(a);
    BD_LAUNCH_CHECK();
    rc = flatten(s, true, grad);
    return rc ? rc : sg_finish(s, sum);
}
int predict_rows(bd_surrogate *s, const float *x, int n, float *y) {
    int rc = io_rows(s, std::min(n, kPredictRows));
    for (int r0 = 0; r0 < n && !rc; r0 += kPredictRows) {
        const int cnt = std::min(kPredictRows, n - r0);
        BD_CUDA_TRY(cudaMemcpyAsync(s->px, x + (size_t)r0 * s->n_in, (size_t)cnt * s->n_in * 4, cudaMemcpyHostToDevice,
                                    s->stream));
        rc = chain_launch(s, false, false, s->px, nullptr, cnt, s->py);
        if (!rc)
            BD_CUDA_TRY(cudaMemcpyAsync(y + (size_t)r0 * s->n_out, s->py, (size_t)cnt * s->n_out * 4,
                                        cudaMemcpyDeviceToHost, s->stream));
    }
    return rc ? rc : sg_finish(s, nullptr);
}

}  // namespace

extern "C" {

// Gradients of the mean loss over one batch (x [batch][n_in], y
// [batch][n_out], host) without an update, flat like bd_surrogate_get_params;
// loss = (1 / (batch n_out)) sum w (y_pred - y)^2.
int bd_surrogate_gradients(bd_surrogate *s, const float *x, const float *y, float *grad, float *loss) {
    if (!s || !x || !y || !grad) return BD_ERR_ARG;
    double sum = 0;
    const int rc = gradients_of(s, x, y, grad, &sum);
    if (rc) cudaStreamSynchronize(s->stream);
    if (loss && (!rc || rc == BD_ERR_TIMEOUT)) *loss = (float)(sum / ((double)s->batch * s->n_out));
    return rc;
}

// Network outputs for n inputs (host x [n][n_in] -> y [n][n_out]).
int bd_surrogate_predict(bd_surrogate *s, const float *x, int n, float *y) {
    if (!s || !x || !y || n < 0) return BD_ERR_ARG;
    const int rc = predict_rows(s, x, n, y);
    if (rc) cudaStreamSynchronize(s->stream);
    return rc;
}

// Plain GEMM through the same kernel, for tests and measurement:
// C [M][N] (FP32) = A [M][K] B [N][K]^T with BF16 inputs given as raw bits.
int bd_umma_gemm_bf16(const unsigned short *a, const unsigned short *b, int M, int N, int K, float *c) {
    if (!a || !b || !c || M < 1 || N < 1 || K < 8 || K % 8) return BD_ERR_ARG;
    __nv_bfloat16 *da = nullptr, *db = nullptr;
    float *dc = nullptr, *part = nullptr;
    unsigned *err = nullptr;
    const int ks = 256, splits = div_up(K, ks);
    int rc = BD_OK;
    cudaStream_t st = nullptr;
    if (set_gemm_attrs() != BD_OK) return BD_ERR_CUDA;
    if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return BD_ERR_CUDA;
    if (cudaMalloc(&da, (size_t)M * K * 2) != cudaSuccess || cudaMalloc(&db, (size_t)N * K * 2) != cudaSuccess ||
        cudaMalloc(&part, (size_t)splits * M * N * 4) != cudaSuccess || cudaMalloc(&dc, (size_t)M * N * 4) != cudaSuccess ||
        cudaMalloc(&err, 4) != cudaSuccess)
        rc = BD_ERR_NOMEM;
    CUtensorMap ta, tb;
    if (!rc) {
        cudaMemcpyAsync(da, a, (size_t)M * K * 2, cudaMemcpyHostToDevice, st);
        cudaMemcpyAsync(db, b, (size_t)N * K * 2, cudaMemcpyHostToDevice, st);
        cudaMemsetAsync(err, 0, 4, st);
        rc = make_tmap(&ta, da, M, K, kBM);
        if (!rc) rc = make_tmap(&tb, db, N, K, kBN);
    }
    if (!rc) {
        GemmTable t;
        std::memset(&t, 0, sizeof(t));
        t.n_jobs = 1;
        t.err = err;
        GemmJob &g = t.job[0];
        g.a = ta;
        g.b = tb;
        g.M = M;
        g.N = N;
        g.K = K;
        g.k_split = ks;
        g.out_f32 = part;
        g.bn = kBN;
        rc = launch_gemms(t, st);
    }
    if (!rc) {
        k_sum_splits<<<div_up((long)M * N, 256), 256, 0, st>>>(part, splits, (size_t)M * N, dc);
        std::vector<float> ct((size_t)M * N);  // the kernel writes C transposed
        cudaMemcpyAsync(ct.data(), dc, (size_t)M * N * 4, cudaMemcpyDeviceToHost, st);
        unsigned e = 0;
        cudaMemcpyAsync(&e, err, 4, cudaMemcpyDeviceToHost, st);
        if (cudaStreamSynchronize(st) != cudaSuccess) rc = BD_ERR_CUDA;
        else if (e) rc = BD_ERR_TIMEOUT;
        for (int i = 0; i < M && !rc; i++)
            for (int j = 0; j < N; j++) c[(size_t)i * N + j] = ct[(size_t)j * M + i];
    }
    cudaFree(da);
    cudaFree(db);
    cudaFree(dc);
    cudaFree(part);
    cudaFree(err);
    cudaStreamDestroy(st);
    return rc;
}

}  // extern "C"
