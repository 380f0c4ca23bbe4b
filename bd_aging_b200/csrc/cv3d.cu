// cv3d.cu -- Contracting_Vector3D (Contracting_Vector3D.cuh:39-75) on the GPU.
//
// add_statistics (Contracting_Vector3D.cu:57-164): for every particle m, the
// per-bin sums h_b(m) of unit vectors d/|d| towards its neighbours closer than
// `range` (d = r_m - r_n, optional minimum image with floor() of the double
// sum, Contracting_Vector3D.cu:101-105), then per Cartesian component c the
// normal equations A^T A_c += h_c h_c^T and A^T b_c += h_c f_c.
//   k_cv_hits: 32 particles per block, a lane each; its warps share the
//     partners.  Up to kCvFused bins, with enough particles for them, the block
//     adds its rows' products H_c^T H_c and H_c^T f_c (FP64; the reference
//     accumulates in float) to the sums;
//   otherwise H[c][m][b] (float, like the reference's hit_vec) goes to
//     memory, k_cv_normal multiplies it, tiled over the bins and split over m
//     so that every SM has a block, and k_cv_reduce adds the splits in order.
// k_cv_hits is bound by issue: all but about 2% of the pairs are out of range.
// Partners are staged in shared memory and read as broadcasts, two per packed
// operation, with the minimum image rounded to the nearest integer and 1e-4 of
// slack on the squared range; a lane notes the partners that pass in a bit
// mask per 32 (no branch in that loop), and the reference's arithmetic decides
// on those, eight masks at a time.  Where that test could miss a pair (range
// beyond 0.49 side, a coordinate far outside the box) every pair is noted.  A
// lane adds to a row of its own (a copy per warp, summed at the end), so it
// needs no atomics; with H in memory it adds there.
// Measured, 4000 particles, 24 bins to 3.5: 38 us a configuration (84 + 259 for
// a warp per particle with a double-precision floor per component of every
// pair, and a product kernel of 12 blocks).
// calculate_vector (Contracting_Vector3D.cu:166-297): per component the SVD
// pseudo-inverse x = V diag(1/w) U^T b with 1/w dropped where
// |w / w_max| <= 1e-6, averaged over the three components.  The matrices are
// bins x bins, so the FP64 one-sided Jacobi SVD runs on the host.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "runtime.cuh"

namespace bd {

constexpr int kCvNeighsMax = 10000;  // Contracting_Vector3D.cuh:36

constexpr int kCvBlock = 32;   // particles per block
constexpr int kCvTile = 1024;  // partners staged at a time
constexpr int kCvMasks = 8;    // masks of 32 partners a lane notes before they are settled
// Products in k_cv_hits: us a call, in it / by k_cv_normal from H in memory, at
// 60 particles 30 / 32 with 24 bins, 38 / 32 with 40, 52 / 32 with 60; at 1000
// 26 / 33, 36 / 37, 50 / 42; at 4000 38 / 57, 50 (34 bins) / 71, 68 / 89.  A block's products
// take 3 bins^2 sums of 32 terms however few blocks there are, so that with
// more than 24 bins some 40 particles a bin have to be there; beyond 60 bins its
// 8 warps' rows don't fit (4 warps: 79 / 34 at 300 particles, 105 / 88 at 4000).
constexpr int kCvFused = 60;
inline bool cv_fused(int n, int bins) { return bins <= kCvFused && n >= 40 * (bins - 24); }
constexpr size_t kCvSmemMost = (size_t)227 * 1024 - 256;  // beside the static shared memory
struct CvHits {
    const float *rr, *xx;
    int n;
    float side, range;
    int bins;
    float *H;            // [3][n][bins] (zero), or null: the block adds to ata and atb
    double *ata, *atb;
    CallStatus *st;
};
// shared memory: tile [3][kCvTile] and masks [warps][kCvMasks][32] (later the
// rows in FP64, [32][3 bins | 1]), bin sums [warps][32][3 bins | 1] (an odd row
// length spreads the lanes over the banks)
static size_t cv_hits_smem(int bins, bool fused, int warps) {
    const size_t row = (3 * (size_t)bins) | 1, stage = sizeof(float) * (3 * kCvTile + (size_t)warps * kCvMasks * 32);
    return (fused ? std::max(stage, sizeof(double) * 32 * row) + sizeof(float) * warps * 32 * row : stage);
}
__global__ void __launch_bounds__(512) k_cv_hits(const CvHits a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int T = blockDim.x, W = T >> 5, lane = threadIdx.x & 31, wid = threadIdx.x >> 5, bins = a.bins, n = a.n;
    const int row = (3 * bins) | 1;
    float *tx = reinterpret_cast<float *>(smem), *ty = tx + kCvTile, *tz = ty + kCvTile;
    unsigned *masks = reinterpret_cast<unsigned *>(tz + kCvTile) + wid * kCvMasks * 32 + lane;  // mask k at [32 k]
    double *s_rows = reinterpret_cast<double *>(smem);
    float *s_hits = reinterpret_cast<float *>(
        smem + max(sizeof(float) * (3 * kCvTile + W * kCvMasks * 32), sizeof(double) * 32 * row));
    float *hw = s_hits + ((size_t)wid * 32 + lane) * row;
    __shared__ int s_neighs[kCvBlock];
    const int first = blockIdx.x * kCvBlock, m = first + lane;
    const bool live = m < n;
    if (!a.H)
        for (int b = threadIdx.x; b < W * 32 * row; b += T) s_hits[b] = 0.f;
    if (threadIdx.x < kCvBlock) s_neighs[threadIdx.x] = 0;
    const bool pbc = a.side > 0.f;
    const float side = a.side, side_inv = pbc ? __fdiv_rn(1.0f, a.side) : 0.f;
    const float range_sq = __fmul_rn(a.range, a.range), lim = range_sq * 1.0001f;
    const float bin_size_inv = __fdiv_rn(1.0f, __fdiv_rn(a.range, (float)bins));
    const float nan = __int_as_float(0x7fffffff);  // never within range
    auto far_out = [&](float v) { return pbc && !(v >= -0.2f * side && v <= 1.2f * side); };
    const float xm = live ? a.rr[3 * (size_t)m] : nan, ym = live ? a.rr[3 * (size_t)m + 1] : nan,
                zm = live ? a.rr[3 * (size_t)m + 2] : nan;
    const bool every = (pbc && a.range > 0.49f * side) || (live && (far_out(xm) || far_out(ym) || far_out(zm)));
    const f2 XM = f2_bcast(xm), YM = f2_bcast(ym), ZM = f2_bcast(zm);
    const f2 SINV = f2_bcast(side_inv), NSIDE = f2_bcast(-side), MAGIC = f2_bcast(kRintMagic);
    auto image = [&](f2 d) { return pbc ? f2_fma(f2_sub(f2_fma(d, SINV, MAGIC), MAGIC), NSIDE, d) : d; };
    // the minimum image of the reference, floor of a double sum; away from half
    // a box the floor is the nearest integer
    auto image_exact = [&](float d) {
        const float x = __fmul_rn(side_inv, d), k = rintf(x);
        const float f = fabsf(x - k) < 0.4999f ? k : (float)floor(__dadd_rn((double)x, 0.5));
        return __fsub_rn(d, __fmul_rn(side, f));
    };
    const int share = kCvTile / W, words = share / 32;  // a warp's partners and masks per tile
    int held = 0, from = 0, neighs = 0;                 // masks held, tile of the first
    auto settle = [&]() {  // the reference's test and sums of the noted partners
        unsigned mask = 0;
        int k = -1;
        for (;;) {
            while (mask == 0u && ++k < held) mask = masks[32 * k];
            if (mask == 0u) break;
            const int t = __ffs(mask) - 1;
            mask &= mask - 1u;
            const int partner = from + k / words * kCvTile + wid * share + k % words * 32 + t;
            if (partner == m) continue;
            const size_t j = 3 * (size_t)partner;
            float dx = __fsub_rn(xm, a.rr[j]), dy = __fsub_rn(ym, a.rr[j + 1]), dz = __fsub_rn(zm, a.rr[j + 2]);
            if (pbc) dx = image_exact(dx), dy = image_exact(dy), dz = image_exact(dz);
            const float d2 = dist2_rn(dx, dy, dz);
            if (!(d2 < range_sq)) continue;
            const float dist = __fsqrt_rn(d2);
            const int nb = min((int)__fmul_rn(bin_size_inv, dist), bins - 1);  // the reference indexes hit_vec[bins] here
            const float ux = __fdiv_rn(dx, dist), uy = __fdiv_rn(dy, dist), uz = __fdiv_rn(dz, dist);
            if (a.H) {
                float *h = a.H + (size_t)m * bins + nb;
                const size_t comp = (size_t)n * bins;
                atomicAdd(h, ux);
                atomicAdd(h + comp, uy);
                atomicAdd(h + 2 * comp, uz);
            } else {
                hw[nb] += ux;
                hw[bins + nb] += uy;
                hw[2 * bins + nb] += uz;
            }
            neighs++;
        }
        held = 0;
    };
    for (int t0 = 0; t0 < n; t0 += kCvTile) {
        const int tn = min(kCvTile, n - t0);
        bool wild = false;
        __syncthreads();
        for (int t = threadIdx.x; t < kCvTile; t += T) {
            float x = nan, y = nan, z = nan;  // padding
            if (t < tn) {
                const size_t j = 3 * (size_t)(t0 + t);
                x = a.rr[j], y = a.rr[j + 1], z = a.rr[j + 2];
                wild = wild || far_out(x) || far_out(y) || far_out(z);
            }
            tx[t] = x, ty[t] = y, tz[t] = z;
        }
        const bool all = (__syncthreads_or(wild) || every) && live;
        if (held == 0) from = t0;
        for (int w = 0; w < words; w++) {
            const int base = wid * share + 32 * w;
            unsigned mask = 0;
            if (base < tn) {
#pragma unroll
                for (int t = 0; t < 32; t += 4) {
                    const float4 x = *reinterpret_cast<const float4 *>(tx + base + t),
                                 y = *reinterpret_cast<const float4 *>(ty + base + t),
                                 z = *reinterpret_cast<const float4 *>(tz + base + t);
#pragma unroll
                    for (int u = 0; u < 4; u += 2) {
                        const f2 DX = image(f2_sub(XM, u ? f2_make(x.z, x.w) : f2_make(x.x, x.y)));
                        const f2 DY = image(f2_sub(YM, u ? f2_make(y.z, y.w) : f2_make(y.x, y.y)));
                        const f2 DZ = image(f2_sub(ZM, u ? f2_make(z.z, z.w) : f2_make(z.x, z.y)));
                        const f2 D2 = f2_fma(DZ, DZ, f2_fma(DY, DY, f2_mul(DX, DX)));
                        float d2a, d2b;
                        f2_split(D2, d2a, d2b);
                        if (d2a < lim) mask |= 1u << (t + u);
                        if (d2b < lim) mask |= 2u << (t + u);
                    }
                }
                if (all) mask = base + 32 <= tn ? 0xffffffffu : (1u << (tn - base)) - 1u;
            }
            masks[32 * (held + w)] = mask;
        }
        held += words;
        if (held + words > kCvMasks) settle();
    }
    settle();
    if (neighs) atomicAdd(&s_neighs[lane], neighs);
    __syncthreads();
    if (threadIdx.x < kCvBlock && s_neighs[threadIdx.x] >= kCvNeighsMax) set_status(a.st, kStatCellOverflow);
    if (a.H) return;
    // rows summed over the warps in order, in FP64 from there (a conversion per
    // row entry, not per product), then their products
    for (int t = threadIdx.x; t < 32 * row; t += T) {
        float v = s_hits[t];
        for (int w = 1; w < W; w++) v += s_hits[(size_t)w * 32 * row + t];
        s_rows[t] = (double)v;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < 3 * bins * bins; t += T) {
        const int c = t / (bins * bins), i = t / bins % bins, j = t % bins;
        const double *h = s_rows + c * bins;
        double v = 0.0;
#pragma unroll 8
        for (int k = 0; k < kCvBlock; k++) v += h[k * row + i] * h[k * row + j];
        if (v != 0.0) atomicAdd(&a.ata[t], v);
    }
    for (int t = threadIdx.x; t < 3 * bins; t += T) {
        double v = 0.0;
        for (int k = 0; k < min(kCvBlock, n - first); k++)
            v += s_rows[k * row + t] * (double)a.xx[3 * (size_t)(first + k) + t / bins];
        if (v != 0.0) atomicAdd(&a.atb[t], v);
    }
}

// A^T A_c[i][j] += sum_m H_c[m][i] H_c[m][j];  A^T b_c[i] += sum_m H_c[m][i] f_c[m]
// grid: (ceil(bins/16), ceil(bins/16), 3 splits), block 16x16, m tiled by 64;
// split k of component c takes the tiles k, k + splits, ... and writes its
// sums to part[k] ([3][bins][bins] then [3][bins]), or adds them to the result
// when there is one split.
constexpr int kCvRows = 64;
__global__ void k_cv_normal(const float *__restrict__ H, const float *__restrict__ xx, int n, int bins, int splits,
                            double *part, double *ata, double *atb) {
    __shared__ float hi[kCvRows][17], hj[kCvRows][17], fc[kCvRows];
    const int c = blockIdx.z % 3, split = blockIdx.z / 3;
    const int i = blockIdx.y * 16 + threadIdx.y, j = blockIdx.x * 16 + threadIdx.x;
    const float *Hc = H + (size_t)c * n * bins;
    double acc = 0.0, accb = 0.0;
    const int tid = threadIdx.y * 16 + threadIdx.x;
    for (int m0 = split * kCvRows; m0 < n; m0 += splits * kCvRows) {
        __syncthreads();
        for (int t = tid; t < kCvRows * 16; t += 256) {
            int mm = t / 16, kk = t % 16;
            int m = m0 + mm;
            int ii = blockIdx.y * 16 + kk, jj = blockIdx.x * 16 + kk;
            hi[mm][kk] = (m < n && ii < bins) ? Hc[(size_t)m * bins + ii] : 0.f;
            hj[mm][kk] = (m < n && jj < bins) ? Hc[(size_t)m * bins + jj] : 0.f;
        }
        if (tid < kCvRows) fc[tid] = (m0 + tid < n) ? xx[3 * (size_t)(m0 + tid) + c] : 0.f;
        __syncthreads();
#pragma unroll 8
        for (int mm = 0; mm < kCvRows; mm++) {
            acc += (double)hi[mm][threadIdx.y] * (double)hj[mm][threadIdx.x];
            if (blockIdx.x == 0 && threadIdx.x == 0) accb += (double)hi[mm][threadIdx.y] * (double)fc[mm];
        }
    }
    const size_t cells = 3 * (size_t)bins * bins, at = ((size_t)c * bins + i) * bins + j;
    double *pa = part + (size_t)split * (cells + 3 * (size_t)bins), *pb = pa + cells;
    const bool whole = splits == 1;
    if (i < bins && j < bins) {
        if (whole) ata[at] += acc;
        else pa[at] = acc;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0 && i < bins) {
        if (whole) atb[(size_t)c * bins + i] += accb;
        else pb[(size_t)c * bins + i] = accb;
    }
}
// result (A^T A then A^T b, contiguous) += the splits in order
__global__ void k_cv_reduce(const double *__restrict__ part, int splits, int count, double *out) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= count) return;
    double v = 0.0;
#pragma unroll 8
    for (int k = 0; k < splits; k++) v += part[(size_t)k * count + t];
    out[t] += v;
}

// One-sided Jacobi SVD of a symmetric bins x bins matrix in FP64 (host).  a
// and v hold their columns one after another (a rotation runs down two of
// them).  The squared column norms are recomputed every sweep and carried
// through its rotations (al - t ga, be + t ga), so a pair costs one product
// sum, in four chains.
static void jacobi_svd(int N, std::vector<double> &a, std::vector<double> &v, std::vector<double> &w) {
    v.assign((size_t)N * N, 0.0);
    for (int i = 0; i < N; i++) v[(size_t)i * N + i] = 1.0;
    auto dot = [N](const double *x, const double *y) {
        double s0 = 0, s1 = 0, s2 = 0, s3 = 0;
        int i = 0;
        for (; i + 3 < N; i += 4) {
            s0 += x[i] * y[i]; s1 += x[i + 1] * y[i + 1]; s2 += x[i + 2] * y[i + 2]; s3 += x[i + 3] * y[i + 3];
        }
        for (; i < N; i++) s0 += x[i] * y[i];
        return (s0 + s1) + (s2 + s3);
    };
    std::vector<double> norm(N);
    for (int sweep = 0; sweep < 100; sweep++) {
        double off = 0.0;
        for (int p = 0; p < N; p++) norm[p] = dot(&a[(size_t)p * N], &a[(size_t)p * N]);
        for (int p = 0; p + 1 < N; p++)
            for (int q = p + 1; q < N; q++) {
                double *ap = &a[(size_t)p * N], *aq = &a[(size_t)q * N];
                const double al = norm[p], be = norm[q];
                if (!(al > 0.0) || !(be > 0.0)) continue;
                const double ga = dot(ap, aq);
                if (ga == 0.0) continue;
                const double den = std::sqrt(al * be);
                if (den == 0.0) continue;
                const double co = std::fabs(ga) / den;
                off = std::max(off, co);
                if (co < 1e-15) continue;
                const double zeta = (be - al) / (2.0 * ga);
                const double t = (zeta >= 0 ? 1.0 : -1.0) / (std::fabs(zeta) + std::sqrt(1.0 + zeta * zeta));
                const double cs = 1.0 / std::sqrt(1.0 + t * t), sn = cs * t;
                double *vp = &v[(size_t)p * N], *vq = &v[(size_t)q * N];
                for (int i = 0; i < N; i++) {
                    const double x = ap[i], y = aq[i];
                    ap[i] = cs * x - sn * y;
                    aq[i] = sn * x + cs * y;
                }
                for (int i = 0; i < N; i++) {
                    const double x = vp[i], y = vq[i];
                    vp[i] = cs * x - sn * y;
                    vq[i] = sn * x + cs * y;
                }
                norm[p] = std::max(0.0, al - t * ga);
                norm[q] = be + t * ga;
            }
        if (off < 1e-15) break;
    }
    w.assign(N, 0.0);
    for (int j = 0; j < N; j++) {
        double s = 0;
        for (int i = 0; i < N; i++) s += a[(size_t)j * N + i] * a[(size_t)j * N + i];
        s = std::sqrt(s);
        w[j] = s;
        if (s > 0)
            for (int i = 0; i < N; i++) a[(size_t)j * N + i] /= s;
    }
}

}  // namespace bd

using namespace bd;

struct bd_cv3d {
    int bins = 0;
    float range = 0.f;
    int samples = 0;
    bool calculated = false;
    double *d_ata = nullptr, *d_atb = nullptr;  // one allocation: [3][bins][bins], [3][bins]
    void *d_work = nullptr;                     // partial normal equations, then H
    size_t work_cap = 0;
    std::vector<float> result;
};

extern "C" {

int bd_cv3d_create(int bins, float range, bd_cv3d **out) {
    if (!out || bins < 1 || bins > 1024 || !(range > 0)) return BD_ERR_ARG;
    bd_cv3d *cv = new bd_cv3d();
    cv->bins = bins;
    cv->range = range;
    cv->result.assign(bins, 0.f);
    const size_t sums = 3 * (size_t)bins * bins + 3 * (size_t)bins;
    if (int rc = allow_smem(k_cv_hits, kCvSmemMost)) {
        bd_cv3d_destroy(cv);
        return rc;
    }
    if (cudaMalloc(&cv->d_ata, sizeof(double) * sums) != cudaSuccess) {
        bd_cv3d_destroy(cv);
        return BD_ERR_NOMEM;
    }
    cv->d_atb = cv->d_ata + 3 * (size_t)bins * bins;
    cudaMemset(cv->d_ata, 0, sizeof(double) * sums);
    *out = cv;
    return BD_OK;
}

int bd_cv3d_add_statistics(bd_cv3d *cv, const float *rr, const float *xx, int n, float side, void *stream) {
    if (!cv || n <= 0 || !rr || !xx) return BD_ERR_ARG;  // DEBUG_ASSERT(nparticles > 0) in the reference
    cudaStream_t s = as_stream(stream);
    const int bins = cv->bins, tiles = div_up(bins, 16);
    const bool fused = cv_fused(n, bins);
    // splits over the particles until about two blocks per SM, each with a tile
    // of rows at least
    const int splits = std::max(1, std::min(div_up(n, kCvRows), 148 * 2 / (3 * tiles * tiles)));
    const size_t sums = 3 * (size_t)bins * bins + 3 * (size_t)bins;
    const size_t part = splits > 1 ? sizeof(double) * sums * splits : 0;
    const size_t need = fused ? 0 : part + sizeof(float) * 3 * (size_t)n * bins;
    if (need > cv->work_cap) {
        if (cv->d_work) cudaFree(cv->d_work);
        cv->d_work = nullptr;
        cv->work_cap = 0;
        if (cudaMalloc(&cv->d_work, need) != cudaSuccess) return BD_ERR_NOMEM;
        cv->work_cap = need;
    }
    double *d_part = static_cast<double *>(cv->d_work);
    float *d_H = fused ? nullptr : reinterpret_cast<float *>(static_cast<unsigned char *>(cv->d_work) + part);
    // 16 warps a block where their copies of the rows fit beside the static
    // shared memory (33 bins), else 8 (60 bins)
    const int warps = cv_hits_smem(bins, fused, 16) <= kCvSmemMost ? 16 : 8;
    const size_t sm = cv_hits_smem(bins, fused, warps);
    CallSlot w(s);
    if (!w.ok()) return BD_ERR_NOMEM;
    if (!fused) BD_CUDA_TRY(cudaMemsetAsync(d_H, 0, sizeof(float) * 3 * (size_t)n * bins, s));
    k_cv_hits<<<div_up(n, kCvBlock), warps * 32, sm, s>>>({rr, xx, n, side, cv->range, bins, d_H, cv->d_ata, cv->d_atb,
                                                           w.status});
    BD_LAUNCH_CHECK();
    if (!fused) {
        k_cv_normal<<<dim3(tiles, tiles, 3 * splits), dim3(16, 16), 0, s>>>(d_H, xx, n, bins, splits, d_part, cv->d_ata,
                                                                           cv->d_atb);
        BD_LAUNCH_CHECK();
    }
    if (!fused && splits > 1) {
        k_cv_reduce<<<div_up((long)sums, 64), 64, 0, s>>>(d_part, splits, (int)sums, cv->d_ata);
        BD_LAUNCH_CHECK();
    }
    BD_CUDA_TRY(w.wait());
    cv->samples++;
    return status_from_bits(*static_cast<volatile unsigned *>(&w.host->status));
}

int bd_cv3d_calculate_vector(bd_cv3d *cv) {
    if (!cv) return BD_ERR_ARG;
    if (cv->samples <= 0) return BD_ERR_STATE;  // the reference throws runtime_error
    const int N = cv->bins;
    std::vector<double> ata((size_t)3 * N * N + (size_t)3 * N);  // A^T A, then A^T b
    BD_CUDA_TRY(cudaMemcpy(ata.data(), cv->d_ata, sizeof(double) * ata.size(), cudaMemcpyDeviceToHost));
    const double *atb = ata.data() + (size_t)3 * N * N;
    std::vector<double> acc(N, 0.0), a, v, w;
    for (int c = 0; c < 3; c++) {
        a.assign(ata.begin() + (size_t)c * N * N, ata.begin() + (size_t)(c + 1) * N * N);  // symmetric: by columns too
        jacobi_svd(N, a, v, w);  // a <- U
        double wmax = 0;
        for (double x : w) wmax = std::max(wmax, std::fabs(x));
        std::vector<double> aux(N, 0.0);
        for (int j = 0; j < N; j++) {
            double s = 0;
            for (int i = 0; i < N; i++) s += a[(size_t)j * N + i] * atb[(size_t)c * N + i];
            double winv = (wmax > 0 && std::fabs(w[j] / wmax) > 1e-6) ? 1.0 / w[j] : 0.0;
            aux[j] = s * winv;
        }
        for (int i = 0; i < N; i++) {
            double s = 0;
            for (int k = 0; k < N; k++) s += v[(size_t)k * N + i] * aux[k];
            acc[i] += s;
        }
    }
    for (int i = 0; i < N; i++) cv->result[i] = (float)(acc[i] / 3.0);
    cv->calculated = true;
    return BD_OK;
}

int bd_cv3d_get_vector(const bd_cv3d *cv, float *out) {
    if (!cv || !out) return BD_ERR_ARG;
    if (!cv->calculated) return BD_ERR_STATE;  // the reference throws runtime_error
    std::memcpy(out, cv->result.data(), sizeof(float) * cv->bins);
    return BD_OK;
}

int bd_cv3d_destroy(bd_cv3d *cv) {
    if (!cv) return BD_ERR_ARG;
    if (cv->d_ata) cudaFree(cv->d_ata);
    if (cv->d_work) cudaFree(cv->d_work);
    delete cv;
    return BD_OK;
}

}  // extern "C"
