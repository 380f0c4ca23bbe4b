// gder.cu -- g(r) counts of the batched replica engine.
//
// get_gder_dev (get_gder.cu:69-127) tests every ordered pair (i, j) of two
// species against `range` with the minimum-image distance (r_i - r_j) and
// adds one count to bin (int)(dist / bin_size).  Two kernels give the same
// exact integer counts: k_gr_cells takes candidates from the cells within
// range (replicas whose box holds that region), k_gr_pairs every pair.
//
// k_gr_cells.  A block owns a brick of kGrBrick^3 cells (its "home"
// particles) and a slice of the cells within m = ceil(range / cell side)
// cells of the brick, skipping cells whose nearest point lies farther than
// `range` from the brick.  Every unordered pair of bricks is taken by one of
// the two: a candidate cell counts when its brick, as the region reaches it,
// comes after the home brick in (z, y, x) order of unwrapped brick positions.
// That order is reversed seen from the other brick, so each brick has half of
// its region, the same for every brick.  Within the home brick a pair counts
// for the smaller index.  Inside the range the minimum-image distance of
// (j, i) is the exact negation of that of (i, j), so one evaluation feeds
// both ordered counts.  The candidate region (kGrBrick + 2m cells per axis)
// must not wrap onto itself, so every cell appears at most once.
//
// A candidate cell that the region reaches across a face of the box carries
// the periodic shift s = L k (k = -1, 0, 1 per axis) of its image next to the
// brick.  Pairs are tested against the shifted (rounded) position x_j + s;
// where that does not settle the bin (gr_bins.cuh, with the rounding of the
// shift as the distance error), the difference is (x_i - x_j) - s, both
// roundings the reference's minimum image makes (d - L floor(d / L + 1/2),
// get_gder.cu:113-115) when its floor equals k.  For a pair within range that
// is always the case: a separation below the range is below L / 2, so the
// region's image of the cell is the minimum image; and a pair whose minimum
// image lies within range has its cell in the region at that image.
//
// Bound: issue slots.  A pair in range costs an estimated bin and one shared
// atomic; a group of four candidates out of range of all 32 home particles of
// a warp is left after the distances.  Hence compact groups: the brick's
// cells are numbered along a Z-order curve before its particles are cut into
// groups of 32 (a lane each), candidates are staged in cell order and, so
// that a candidate's species is the same for a whole loop, big ones from the
// front and small ones from the back of the tile.  (group, tile eighth) tasks
// are handed out by a counter: 9 groups on 8 warps would otherwise leave 7
// warps waiting for the ninth.  Every tested pair being one lane's work, the
// counts of 32 lanes meet in shared memory only: one histogram a block for
// bb, mixed (copied to bs and sb) and ss pairs, one count per unordered pair,
// doubled for equal species at the end.
// Measured, 8 x 32768 particles, 400 bins to 15 (1.1e9 unordered pairs in
// range): 2.6 ms, 78% of issue slots; 12.6 ms with a bin table looked up per
// pair, a branch per pair and candidates of every later brick.
//
// The bound assumes every particle lies in its cell to within
// kGrTol * cell side.  The engine's wrap keeps positions in [0, L], but a
// blown-up state can leave a coordinate outside the box by the rounding of
// x - L floor(x / L); each home particle checks its cell, and a replica with
// a misplaced particle is flagged and recounted by k_gr_pairs.
#include <algorithm>
#include <type_traits>

#include "engine_state.cuh"
#include "gr_bins.cuh"

namespace bd {

constexpr int kGrBrick = 4;
constexpr int kGrThreads = 256;
constexpr int kGrCells = 4 * kGrThreads;  // region cells scanned at a time (gr_scan's limit)
constexpr int kGrTile = 896;              // candidates staged at a time (four blocks fit an SM)
constexpr int kGrTileLen = kGrTile + 8;   // room to pad both species to groups of four
constexpr int kGrSlices = 8;              // tile slices per task
constexpr int kGrMaxCap = 24;
constexpr int kGrHomeMax = kGrBrick * kGrBrick * kGrBrick * kGrMaxCap;
constexpr double kGrTol = 1e-3;  // allowed stick-out of a particle from its cell, in cell sides

struct GrArgs {
    const SysDev *sys;
    const int *cnt;
    const float4 *pos;
    const int4 *bricks;  // (replica, ox, oy, oz)
    int cap;
    float range;
    GrBins bins;                 // without the shift's rounding, which depends on the replica (gr_with_shift)
    unsigned long long *counts;  // [R][4][nbins]
    const int *m_of;             // stencil reach in cells, per replica (-1: not counted here)
    int *misplaced;              // per replica: a particle lies outside its cell
    unsigned *status;
};

// Bounds of the estimate for positions shifted by a side of the box.  Per
// component, x_j + s is off by half an ulp and the reference, which rounds
// x_i - x_j first, by half an ulp of that.  At a distance d across a face the
// two are below L + d and L - d in size, so their errors add up to less than
// 2^-24 2 L (and reach it: on equal grids a tie may round either way).
__device__ __forceinline__ GrBins gr_with_shift(GrBins g, float side, float range) {
    const float err = 2.1e-7f * side;  // sqrt(3) 2^-24 2 L
    const float f = 1.f + err / range;
    g.near *= f * f;
    g.c0 += 1.1f * err * g.inv_bin;
    return g;
}

// Exclusive scan of a[0..n) in place (n <= 4 * kGrThreads); returns the total.
__device__ int gr_scan(int *a, int n, int *wsum) {
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    int v[4], s = 0;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int i = 4 * t + k;
        v[k] = i < n ? a[i] : 0;
        s += v[k];
    }
    int incl = s;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += y;
    }
    if (lane == 31) wsum[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const int nw = kGrThreads / 32;
        int w = lane < nw ? wsum[lane] : 0, wi = w;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, wi, off);
            if (lane >= off) wi += y;
        }
        if (lane < nw) wsum[lane] = wi - w;
        if (lane == nw - 1) wsum[nw] = wi;
    }
    __syncthreads();
    int base = wsum[warp] + incl - s;
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int i = 4 * t + k;
        if (i < n) a[i] = base;
        base += v[k];
    }
    const int total = wsum[kGrThreads / 32];
    __syncthreads();
    return total;
}

__device__ __forceinline__ int gr_find(const int *start, int n, int t) {  // last c in [0, n) with start[c] <= t
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (start[mid] <= t) lo = mid; else hi = mid - 1;
    }
    return lo;
}
// periodic shift along one axis: code 0, 1, 2 -> -L, 0, L
__device__ __forceinline__ float gr_shift(int code, int axis, float side) {
    return (float)(((code >> (2 * axis)) & 3) - 1) * side;
}

struct GrSmem {
    float4 home[kGrHomeMax];
    float x[kGrTileLen], y[kGrTileLen], z[kGrTileLen];  // shifted candidates: big from the front, small from the back
    int at[kGrTileLen];                                 // their bucket slots
    unsigned char code[kGrTileLen];                     // their shift codes
    int cstart[kGrCells + 1], cgc[kGrCells];
    unsigned char ccode[kGrCells];
    int wsum[kGrThreads / 32 + 1];
    int nbig, nsml, task;
    unsigned hist[1];  // [3][nbins + kGrSpare] bb, mixed, ss
};

// A warp's 32 home particles against candidates [c0, c1) (multiples of four)
// of one species; `row` (gr_row), `top` (gr_top): the lane's histogram row.
__device__ __forceinline__ void gr_warp_tile(const GrArgs &a, const GrBins &g, const GrSmem &sm, float4 pi, float side,
                                             int c0, int c1, unsigned row, unsigned top) {
    const f2 XI = f2_bcast(pi.x), YI = f2_bcast(pi.y), ZI = f2_bcast(pi.z);
    for (int c = c0; c < c1; c += 4) {
        const float4 x = *reinterpret_cast<const float4 *>(sm.x + c), y = *reinterpret_cast<const float4 *>(sm.y + c),
                     z = *reinterpret_cast<const float4 *>(sm.z + c);
        f2 D2[2];
        float d2[4];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const f2 DX = f2_sub(XI, u ? f2_make(x.z, x.w) : f2_make(x.x, x.y));
            const f2 DY = f2_sub(YI, u ? f2_make(y.z, y.w) : f2_make(y.x, y.y));
            const f2 DZ = f2_sub(ZI, u ? f2_make(z.z, z.w) : f2_make(z.x, z.y));
            D2[u] = f2_fma(DZ, DZ, f2_fma(DY, DY, f2_mul(DX, DX)));
            f2_split(D2[u], d2[2 * u], d2[2 * u + 1]);
        }
        bool in[4];
#pragma unroll
        for (int u = 0; u < 4; u++) in[u] = d2[u] < g.near;
        if (!__any_sync(0xffffffffu, in[0] | in[1] | in[2] | in[3])) continue;
        bool open[4];
        unsigned slot[4];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            unsigned sl[2];
            bool far[2];
            gr_estimate(D2[u], g, top, sl, far);
#pragma unroll
            for (int h = 0; h < 2; h++) {
                open[2 * u + h] = in[2 * u + h] & far[h];
                slot[2 * u + h] = sl[h];
                gr_count(row + 4u * sl[h], 1u);
            }
        }
        if (open[0] | open[1] | open[2] | open[3]) {
#pragma unroll 1
            for (int u = 0; u < 4; u++) {
                if (!(u == 0 ? open[0] : u == 1 ? open[1] : u == 2 ? open[2] : open[3])) continue;
                gr_uncount(row, u == 0 ? slot[0] : u == 1 ? slot[1] : u == 2 ? slot[2] : slot[3], 1u, g.nbins);
                const float4 pj = a.pos[sm.at[c + u]];
                const int code = sm.code[c + u];
                const float dx = __fsub_rn(__fsub_rn(pi.x, pj.x), gr_shift(code, 0, side));
                const float dy = __fsub_rn(__fsub_rn(pi.y, pj.y), gr_shift(code, 1, side));
                const float dz = __fsub_rn(__fsub_rn(pi.z, pj.z), gr_shift(code, 2, side));
                const float e2 = dist2_rn(dx, dy, dz);
                if (e2 < g.thr)
                    gr_count(row + 4u * (unsigned)(gr_bin_settled(e2, g) + __float_as_int(kRintMagic)), 1u);
            }
        }
    }
}

__global__ void __launch_bounds__(kGrThreads, 4) k_gr_cells(GrArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    GrSmem &sm = *reinterpret_cast<GrSmem *>(smem);
    const int tid = threadIdx.x, lane = tid & 31;
    const int4 br = a.bricks[blockIdx.x];
    const int m = a.m_of[br.x];
    if (m < 0) return;
    const SysDev &S = a.sys[br.x];
    const int nc = S.ncell;
    const int ox = br.y, oy = br.z, oz = br.w;
    const int wx = min(kGrBrick, nc - ox), wy = min(kGrBrick, nc - oy), wz = min(kGrBrick, nc - oz);
    const int nbins = a.bins.nbins;
    const float side = S.L;
    const GrBins g = gr_with_shift(a.bins, side, a.range);
    const int stride = nbins + kGrSpare;
    const unsigned top = gr_top(nbins, lane);
    // cells whose nearest point is farther than range: gap g (cells) with
    // g cs - 4 tol > range (cell units, with margin)
    const float cs = side / (float)nc;
    const float tol = (float)kGrTol * cs;
    const float lim = (a.range / cs) * 1.00001f + 4.0f * (float)kGrTol;
    const float lim2 = lim * lim;
    for (int b = tid; b < 3 * stride; b += kGrThreads) sm.hist[b] = 0;

    // 1. home particles of the brick, cells in Z order
    constexpr int nhc = kGrBrick * kGrBrick * kGrBrick;
    for (int c = tid; c < nhc; c += kGrThreads) {
        const int lx = (c & 1) | ((c >> 2) & 2), ly = ((c >> 1) & 1) | ((c >> 3) & 2), lz = ((c >> 2) & 1) | ((c >> 4) & 2);
        int k = 0, gc = 0;
        if (lx < wx && ly < wy && lz < wz) {
            gc = S.cell_base + (ox + lx) + nc * ((oy + ly) + nc * (oz + lz));
            k = a.cnt[gc];
            if (k > a.cap) { set_status(a.status, kStatCellOverflow); k = a.cap; }
        }
        sm.cstart[c] = max(k, 0);
        sm.cgc[c] = gc;
        sm.ccode[c] = (unsigned char)(lx | (ly << 2) | (lz << 4));
    }
    __syncthreads();
    const int H = gr_scan(sm.cstart, nhc, sm.wsum);
    if (tid == 0) { sm.cstart[nhc] = H; sm.task = 0; }
    __syncthreads();
    bool bad = false;
    for (int t = tid; t < H; t += kGrThreads) {
        const int c = gr_find(sm.cstart, nhc, t);
        const float4 v = a.pos[(size_t)sm.cgc[c] * a.cap + (t - sm.cstart[c])];
        sm.home[t] = v;
        const int lc = sm.ccode[c], lx = lc & 3, ly = (lc >> 2) & 3, lz = lc >> 4;
        const float x0 = (float)(ox + lx) * cs, y0 = (float)(oy + ly) * cs, z0 = (float)(oz + lz) * cs;
        bad |= !(v.x >= x0 - tol && v.x <= x0 + cs + tol && v.y >= y0 - tol && v.y <= y0 + cs + tol &&
                 v.z >= z0 - tol && v.z <= z0 + cs + tol);
    }
    if (__syncthreads_or(bad)) {
        if (tid == 0) a.misplaced[br.x] = 1;
        return;
    }
    if (H == 0) return;
    const int groups = (H + 31) >> 5;
    auto next_task = [&]() {
        int t = 0;
        if (lane == 0) t = atomicAdd(&sm.task, 1);
        return __shfl_sync(0xffffffffu, t, 0);
    };
    const float nan = __int_as_float(0x7fffffff);  // a distance from it is never within range
    auto home_of = [&](int group) {
        const int h = (group << 5) + lane;
        return h < H ? sm.home[h] : make_float4(nan, nan, nan, 0.f);
    };

    // 2. pairs inside the home brick (first slice only), each once: smaller index first; no shift
    if (blockIdx.y == 0) {
        for (int task = next_task(); task < groups * kGrSlices; task = next_task()) {
            const int group = task / kGrSlices, q = task % kGrSlices;
            const float4 pi = home_of(group);
            const int h = (group << 5) + lane;
            const unsigned ti = __float_as_uint(pi.w) >> 31;
            for (int c = max(group << 5, H * q / kGrSlices); c < H * (q + 1) / kGrSlices; c++) {
                const float4 pj = sm.home[c];
                const float e2 = dist2_rn(__fsub_rn(pi.x, pj.x), __fsub_rn(pi.y, pj.y), __fsub_rn(pi.z, pj.z));
                if (c > h && e2 < g.thr)
                    atomicAdd(&sm.hist[(ti + (__float_as_uint(pj.w) >> 31)) * stride + gr_bin_settled(e2, g)], 1u);
            }
        }
    }
    // 3. this slice of the half region of bricks after the home brick
    const int rx = wx + 2 * m, ry = wy + 2 * m, nreg = rx * ry * (wz + m);
    const int r0 = (int)((long long)nreg * blockIdx.y / gridDim.y), r1 = (int)((long long)nreg * (blockIdx.y + 1) / gridDim.y);
    for (int c0 = r0; c0 < r1; c0 += kGrCells) {
        const int ntc = min(kGrCells, r1 - c0);
        __syncthreads();  // the cell arrays are free
        for (int q = tid; q < ntc; q += kGrThreads) {
            const int qq = c0 + q;
            const int lx = qq % rx, ly = (qq / rx) % ry, lz = qq / (rx * ry);
            int k = 0, gc = 0, code = 1 | 1 << 2 | 1 << 4;
            const bool after = lz >= wz || ly >= m + wy || (ly >= m && lx >= m + wx);
            if (after) {
                // cell distance to the brick along each axis, minus one
                const int kx = max(0, max(m - lx, lx - (m + wx - 1)) - 1);
                const int ky = max(0, max(m - ly, ly - (m + wy - 1)) - 1);
                const int kz = max(0, lz - wz);
                if ((float)(kx * kx + ky * ky + kz * kz) <= lim2) {
                    int gx = ox - m + lx, gy = oy - m + ly, gz = oz + lz;
                    // a cell reached across a face: its image next to the
                    // brick is the stored position minus L (code 0) or plus L (2)
                    const int sx = gx < 0 ? -1 : gx >= nc, sy = gy < 0 ? -1 : gy >= nc, sz = gz >= nc;
                    gx -= sx * nc;
                    gy -= sy * nc;
                    gz -= sz * nc;
                    code = (sx + 1) | (sy + 1) << 2 | (sz + 1) << 4;
                    gc = S.cell_base + gx + nc * (gy + nc * gz);
                    k = min(max(a.cnt[gc], 0), a.cap);
                }
            }
            sm.cstart[q] = k;
            sm.cgc[q] = gc;
            sm.ccode[q] = (unsigned char)code;
        }
        __syncthreads();
        const int total = gr_scan(sm.cstart, ntc, sm.wsum);
        for (int p = 0; p < total; p += kGrTile) {
            __syncthreads();  // the last tile has been read
            if (tid == 0) sm.nbig = sm.nsml = sm.task = 0;
            for (int t = tid; t < kGrTileLen; t += kGrThreads) sm.x[t] = nan;  // padding
            __syncthreads();
            const int n = min(kGrTile, total - p);
            for (int t0 = tid & ~31; t0 < n; t0 += kGrThreads) {
                const int t = t0 + lane;
                const bool have = t < n;
                int code = 0, at = 0;
                float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
                if (have) {
                    const int c = gr_find(sm.cstart, ntc, p + t);
                    code = sm.ccode[c];
                    at = sm.cgc[c] * a.cap + (p + t - sm.cstart[c]);
                    v = a.pos[at];
                }
                const bool small = (__float_as_uint(v.w) >> 31) != 0u;
                const unsigned mb = __ballot_sync(0xffffffffu, have && !small), ms = __ballot_sync(0xffffffffu, have && small);
                int bb = 0, bs = 0;
                if (lane == 0) {
                    bb = atomicAdd(&sm.nbig, __popc(mb));
                    bs = atomicAdd(&sm.nsml, __popc(ms));
                }
                bb = __shfl_sync(0xffffffffu, bb, 0);
                bs = __shfl_sync(0xffffffffu, bs, 0);
                const unsigned below = (1u << lane) - 1u;
                const int d = small ? kGrTileLen - 1 - (bs + __popc(ms & below)) : bb + __popc(mb & below);
                if (have) {
                    sm.x[d] = v.x + gr_shift(code, 0, side);
                    sm.y[d] = v.y + gr_shift(code, 1, side);
                    sm.z[d] = v.z + gr_shift(code, 2, side);
                    sm.at[d] = at;
                    sm.code[d] = (unsigned char)code;
                }
            }
            __syncthreads();
            const int qb = (sm.nbig + 3) >> 2, s0 = (kGrTileLen - sm.nsml) & ~3, qs = (kGrTileLen - s0) >> 2;
            for (int task = next_task(); task < groups * kGrSlices; task = next_task()) {
                const int group = task / kGrSlices, q = task % kGrSlices;
                const float4 pi = home_of(group);
                const unsigned *rows = sm.hist + (__float_as_uint(pi.w) >> 31) * stride;
                gr_warp_tile(a, g, sm, pi, side, 4 * (qb * q / kGrSlices), 4 * (qb * (q + 1) / kGrSlices), gr_row(rows),
                             top);
                gr_warp_tile(a, g, sm, pi, side, s0 + 4 * (qs * q / kGrSlices), s0 + 4 * (qs * (q + 1) / kGrSlices),
                             gr_row(rows + stride), top);
            }
        }
    }
    __syncthreads();
    unsigned long long *out = a.counts + (size_t)br.x * 4 * nbins;  // bb, bs, sb, ss
    for (int b = tid; b < nbins; b += kGrThreads) {
        const unsigned long long bb = sm.hist[b], mx = sm.hist[stride + b], ss = sm.hist[2 * stride + b];
        if (bb) atomicAdd(&out[b], 2 * bb);
        if (mx) {
            atomicAdd(&out[nbins + b], mx);
            atomicAdd(&out[2 * nbins + b], mx);
        }
        if (ss) atomicAdd(&out[3 * nbins + b], 2 * ss);
    }
}

// Stencil reach of replica r for `range`, or -1 when the candidate region
// would wrap onto itself (the all-pairs kernel handles that replica).
int gder_cell_reach(const SysDev &S, float range) {
    const double cs = (double)S.L / S.ncell;
    // a pair closer than range can sit m cells apart when both particles
    // stick out of their cells by the tolerance
    const int m = (int)std::ceil(((double)range * (1.0 + 1e-5) + 2.0 * kGrTol * cs) / (cs * (1.0 - 1e-5)));
    if (kGrBrick + 2 * m > S.ncell) return -1;
    return m;
}

static size_t gder_cells_smem(int nbins) { return sizeof(GrSmem) + sizeof(unsigned) * 3 * ((size_t)nbins + kGrSpare); }

// ------------------------------------------------------------- all pairs
// Every unordered pair i < j of a replica in the reference order (big first),
// pairs as in the mirror's kernel: 256 particles a block, a chunk of partners
// staged in tiles of one species, packed minimum image by rounding to an
// integer, estimated bins.  Pairs at the edge of the image (a component
// beyond 0.49999 L) and tiles with a coordinate outside [-0.2 L, 1.2 L] take
// the reference's arithmetic in both directions (gr_pair_exact); the two
// orders may then fall in different bins.
constexpr int kGrPairTile = 1024;
struct GrPairArgs {
    const float4 *snap;  // [P] positions by global index
    const SysDev *sys;
    const int *reps;  // replica of blockIdx.z
    float range;
    GrBins bins;
    int jchunk;
    unsigned long long *counts;  // [R][4][nbins]
};
__device__ __forceinline__ int gr_bin_of(float dx, float dy, float dz, float side, float side_inv, const GrBins &g) {
    const float e2 = dist2_rn(min_image_gder(dx, side, side_inv), min_image_gder(dy, side, side_inv),
                              min_image_gder(dz, side, side_inv));
    return e2 < g.thr ? gr_bin_settled(e2, g) : -1;
}
__device__ __noinline__ void gr_pair_exact(const GrBins &g, float dx, float dy, float dz, float side, float side_inv,
                                           int ti, int tj, unsigned *hist, unsigned long long *out) {
    const int nbins = g.nbins, stride = nbins + kGrSpare;
    const int bf = gr_bin_of(dx, dy, dz, side, side_inv, g), bb = gr_bin_of(-dx, -dy, -dz, side, side_inv, g);
    if (bf == bb) {
        if (bf >= 0) atomicAdd(&hist[(ti + tj) * stride + bf], 1u);
        return;
    }
    if (bf >= 0) atomicAdd(&out[(ti * 2 + tj) * nbins + bf], 1ull);
    if (bb >= 0) atomicAdd(&out[(tj * 2 + ti) * nbins + bb], 1ull);
}
__global__ void __launch_bounds__(kGrThreads) k_gr_pairs(GrPairArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    const int r = a.reps[blockIdx.z];
    const SysDev &S = a.sys[r];
    const int n = S.n, n_big = S.n_big, nbins = a.bins.nbins;
    const int i0 = blockIdx.x * kGrThreads, i = i0 + threadIdx.x;
    const int j0 = max((int)blockIdx.y * a.jchunk, i0 + 1), j1 = min(n, (int)(blockIdx.y + 1) * a.jchunk);
    if (j0 >= j1) return;  // uniform over the block: no pair of this replica here
    const float4 *snap = a.snap + S.part_base;
    unsigned long long *out = a.counts + (size_t)r * 4 * nbins;
    float *tx = reinterpret_cast<float *>(smem), *ty = tx + kGrPairTile, *tz = ty + kGrPairTile;
    unsigned *hist = reinterpret_cast<unsigned *>(tz + kGrPairTile);  // [3][nbins + kGrSpare] bb, mixed, ss
    const int stride = nbins + kGrSpare;
    const unsigned top = gr_top(nbins, threadIdx.x & 31);
    for (int b = threadIdx.x; b < 3 * stride; b += kGrThreads) hist[b] = 0;
    const float side = S.L, side_inv = __double2float_rn(1.0 / (double)side);
    const float wild_lo = -0.2f * side, wild_hi = 1.2f * side;
    auto wild_at = [&](float v) { return !(v >= wild_lo && v <= wild_hi); };
    const float nan = __int_as_float(0x7fffffff);
    float xi = nan, yi = nan, zi = nan;
    bool wild = false;
    if (i < n) {
        const float4 v = snap[i];
        xi = v.x, yi = v.y, zi = v.z;
        wild = wild_at(xi) || wild_at(yi) || wild_at(zi);
    }
    const int ti = i < n_big ? 0 : 1;
    const f2 XI = f2_bcast(xi), YI = f2_bcast(yi), ZI = f2_bcast(zi);
    const f2 SINV = f2_bcast(side_inv), NSIDE = f2_bcast(-side), MAGIC = f2_bcast(kRintMagic);
    const float edge = 0.49999f * side, near = a.bins.near, edge_lo = 0.49998f * side;
    const bool check = !(near <= edge_lo * edge_lo);
    const float lim = check ? near * 1.0001f : near;
    for (int t0 = j0, tn; t0 < j1; t0 += tn) {
        tn = min(kGrPairTile, j1 - t0);
        if (t0 < n_big) tn = min(tn, n_big - t0);  // one species a tile
        const int tj = t0 < n_big ? 0 : 1, tp = (tn + 3) & ~3;
        __syncthreads();
        for (int t = threadIdx.x; t < tp; t += kGrThreads) {
            float4 v = make_float4(nan, nan, nan, 0.f);
            if (t < tn) {
                v = snap[t0 + t];
                wild = wild || wild_at(v.x) || wild_at(v.y) || wild_at(v.z);
            }
            tx[t] = v.x, ty[t] = v.y, tz[t] = v.z;
        }
        if (__syncthreads_or(wild)) {
            if (i < n)
                for (int t = 0; t < tn; t++)
                    if (t0 + t > i)
                        gr_pair_exact(a.bins, __fsub_rn(xi, tx[t]), __fsub_rn(yi, ty[t]), __fsub_rn(zi, tz[t]), side,
                                      side_inv, ti, tj, hist, out);
            continue;
        }
        const unsigned row = gr_row(hist + (ti + tj) * stride);
        auto image = [&](f2 d) { return f2_fma(f2_sub(f2_fma(d, SINV, MAGIC), MAGIC), NSIDE, d); };
        auto pairs = [&](auto diagonal, auto checked) {
            constexpr bool kDiag = decltype(diagonal)::value, kCheck = decltype(checked)::value;
            for (int t = 0; t < tp; t += 4) {
                const float4 x = *reinterpret_cast<const float4 *>(tx + t), y = *reinterpret_cast<const float4 *>(ty + t),
                             z = *reinterpret_cast<const float4 *>(tz + t);
                float dx[4], dy[4], dz[4];
                unsigned slot[4];
                bool open[4];
#pragma unroll
                for (int u = 0; u < 4; u += 2) {
                    const f2 DX = image(f2_sub(XI, u ? f2_make(x.z, x.w) : f2_make(x.x, x.y)));
                    const f2 DY = image(f2_sub(YI, u ? f2_make(y.z, y.w) : f2_make(y.x, y.y)));
                    const f2 DZ = image(f2_sub(ZI, u ? f2_make(z.z, z.w) : f2_make(z.x, z.y)));
                    const f2 D2 = f2_fma(DZ, DZ, f2_fma(DY, DY, f2_mul(DX, DX)));
                    f2_split(DX, dx[u], dx[u + 1]);
                    f2_split(DY, dy[u], dy[u + 1]);
                    f2_split(DZ, dz[u], dz[u + 1]);
                    float d2[2];
                    f2_split(D2, d2[0], d2[1]);
                    unsigned sl[2];
                    bool far[2];
                    gr_estimate(D2, a.bins, top, sl, far);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int v = u + h;
                        bool in = d2[h] < lim;
                        if (kDiag && t0 + t + v <= i) in = false, sl[h] = top;
                        if (kCheck) far[h] = far[h] | (fmaxf(fmaxf(fabsf(dx[v]), fabsf(dy[v])), fabsf(dz[v])) > edge);
                        open[v] = in & far[h];
                        slot[v] = sl[h];
                        gr_count(row + 4u * sl[h], 1u);
                    }
                }
                if (open[0] | open[1] | open[2] | open[3]) {
#pragma unroll
                    for (int u = 0; u < 4; u++) {
                        if (!open[u]) continue;
                        gr_uncount(row, slot[u], 1u, nbins);
                        if (kCheck && fmaxf(fmaxf(fabsf(dx[u]), fabsf(dy[u])), fabsf(dz[u])) > edge) {
                            gr_pair_exact(a.bins, __fsub_rn(xi, tx[t + u]), __fsub_rn(yi, ty[t + u]),
                                          __fsub_rn(zi, tz[t + u]), side, side_inv, ti, tj, hist, out);
                            continue;
                        }
                        const float e2 = dist2_rn(dx[u], dy[u], dz[u]);
                        if (e2 < a.bins.thr) atomicAdd(&hist[(ti + tj) * stride + gr_bin_settled(e2, a.bins)], 1u);
                    }
                }
            }
        };
        const bool diag = t0 <= i0 + kGrThreads - 1;
        if (diag && check) pairs(std::true_type{}, std::true_type{});
        else if (diag) pairs(std::true_type{}, std::false_type{});
        else if (check) pairs(std::false_type{}, std::true_type{});
        else pairs(std::false_type{}, std::false_type{});
    }
    __syncthreads();
    for (int b = threadIdx.x; b < nbins; b += kGrThreads) {
        const unsigned long long bb = hist[b], mx = hist[stride + b], ss = hist[2 * stride + b];
        if (bb) atomicAdd(&out[b], 2 * bb);
        if (mx) {
            atomicAdd(&out[nbins + b], mx);
            atomicAdd(&out[2 * nbins + b], mx);
        }
        if (ss) atomicAdd(&out[3 * nbins + b], 2 * ss);
    }
}

// ------------------------------------------------------------- host side
// Device buffer of at least n bytes kept by the engine.
static int gr_reserve(void *&buf, size_t &cap, size_t n) {
    if (cap >= n) return BD_OK;
    if (buf) cudaFree(buf);
    buf = nullptr;
    cap = 0;
    BD_CUDA_TRY(cudaMalloc(&buf, n));
    cap = n;
    return BD_OK;
}

// Counts [R][4][nbins] of every replica into counts_host: replicas with
// m_of[r] >= 0 by k_gr_cells, the others (and those k_gr_cells finds with a
// misplaced particle) by k_gr_pairs.  The cell buckets and displacements are
// up to date.  The engine keeps the brick table (geometry only) and the
// buffers between calls.
int run_gder(bd_engine *e, std::vector<int> &m_of, int nbins, float range, unsigned long long *counts_host) {
    const size_t per = (size_t)4 * nbins, nc = per * e->R;
    cudaStream_t st = e->stream;
    if (e->cap > kGrMaxCap) std::fill(m_of.begin(), m_of.end(), -1);
    const bool any_cells = std::any_of(m_of.begin(), m_of.end(), [](int m) { return m >= 0; });
    // counts, reach and misplaced flag per replica, replicas of the all-pairs launch
    if (int rc = gr_reserve(e->gr_buf, e->gr_cap, nc * sizeof(unsigned long long) + 3 * sizeof(int) * e->R)) return rc;
    unsigned long long *d_counts = static_cast<unsigned long long *>(e->gr_buf);
    int *d_m = reinterpret_cast<int *>(d_counts + nc), *d_bad = d_m + e->R, *d_reps = d_bad + e->R;
    BD_CUDA_TRY(cudaMemsetAsync(d_counts, 0, nc * sizeof(unsigned long long), st));
    const GrBins bins = gr_bins(range, nbins, 0.0);
    if (any_cells) {
        if (!e->gr_bricks) {
            std::vector<int4> bricks;
            for (int r = 0; r < e->R; r++) {
                const int n = e->sysh[r].ncell;
                for (int z = 0; z < n; z += kGrBrick)
                    for (int y = 0; y < n; y += kGrBrick)
                        for (int x = 0; x < n; x += kGrBrick) bricks.push_back(make_int4(r, x, y, z));
            }
            BD_CUDA_TRY(cudaMalloc(&e->gr_bricks, sizeof(int4) * bricks.size()));
            BD_CUDA_TRY(cudaMemcpyAsync(e->gr_bricks, bricks.data(), sizeof(int4) * bricks.size(),
                                        cudaMemcpyHostToDevice, st));
            BD_CUDA_TRY(cudaStreamSynchronize(st));  // the host table goes out of scope
            e->gr_nbricks = (int)bricks.size();
        }
        BD_CUDA_TRY(cudaMemcpyAsync(d_m, m_of.data(), sizeof(int) * e->R, cudaMemcpyHostToDevice, st));
        BD_CUDA_TRY(cudaMemsetAsync(d_bad, 0, sizeof(int) * e->R, st));
        const size_t sm = gder_cells_smem(nbins);
        if (int rc = allow_smem(k_gr_cells, sm)) return rc;
        GrArgs a;
        a.sys = e->d_sys;
        a.cnt = e->cnt[obs_buf(e)];
        a.pos = e->pos[obs_buf(e)];
        a.bricks = e->gr_bricks;
        a.cap = e->cap;
        a.range = range;
        a.bins = bins;
        a.counts = d_counts;
        a.m_of = d_m;
        a.misplaced = d_bad;
        a.status = e->status;
        // region slices until the grid holds about six rounds of the 4 blocks
        // resident on each SM, so that the last round is a small part
        const int slices = std::max(1, std::min(8, div_up(148 * 4 * 6, e->gr_nbricks)));
        k_gr_cells<<<dim3(e->gr_nbricks, slices), kGrThreads, sm, st>>>(a);
        BD_LAUNCH_CHECK();
        std::vector<int> bad(e->R, 0);
        BD_CUDA_TRY(cudaMemcpyAsync(bad.data(), d_bad, sizeof(int) * e->R, cudaMemcpyDeviceToHost, st));
        BD_CUDA_TRY(cudaMemcpyAsync(counts_host, d_counts, nc * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
        BD_CUDA_TRY(cudaStreamSynchronize(st));
        for (int r = 0; r < e->R; r++) {
            if (!bad[r]) continue;
            m_of[r] = -1;
            BD_CUDA_TRY(cudaMemsetAsync(d_counts + per * r, 0, per * sizeof(unsigned long long), st));
        }
    }
    std::vector<int> reps;
    int nmax = 0;
    double pairs = 0.0;
    for (int r = 0; r < e->R; r++)
        if (m_of[r] < 0) {
            reps.push_back(r);
            const int n = e->sysh[r].n;
            nmax = std::max(nmax, n);
            pairs += 0.5 * (double)n * n;
        }
    if (reps.empty()) return BD_OK;  // counts_host is complete
    if (int rc = export_snap(e)) return rc;
    BD_CUDA_TRY(cudaMemcpyAsync(d_reps, reps.data(), sizeof(int) * reps.size(), cudaMemcpyHostToDevice, st));
    GrPairArgs a;
    a.snap = e->snap;
    a.sys = e->d_sys;
    a.reps = d_reps;
    a.range = range;
    a.bins = bins;
    a.counts = d_counts;
    // partners per block, as in the mirror's kernel: about 8 blocks for each SM
    const double want = pairs / (kGrThreads * 148.0 * 8.0);
    a.jchunk = (int)std::min(8192.0, std::max(64.0, 64.0 * std::ceil(want / 64.0)));
    const size_t sm = 3 * kGrPairTile * sizeof(float) + sizeof(unsigned) * 3 * ((size_t)nbins + kGrSpare);
    if (sm > 48 * 1024)
        if (int rc = allow_smem(k_gr_pairs, sm)) return rc;
    const int most = 65535;  // grid limit of y and z
    a.jchunk = std::max(a.jchunk, div_up(nmax, most));
    for (size_t first = 0; first < reps.size(); first += most) {
        a.reps = d_reps + first;
        const dim3 grid(div_up(nmax, kGrThreads), div_up(nmax, a.jchunk),
                        (unsigned)std::min<size_t>(most, reps.size() - first));
        k_gr_pairs<<<grid, kGrThreads, sm, st>>>(a);
        BD_LAUNCH_CHECK();
    }
    BD_CUDA_TRY(cudaMemcpyAsync(counts_host, d_counts, nc * sizeof(unsigned long long), cudaMemcpyDeviceToHost, st));
    BD_CUDA_TRY(cudaStreamSynchronize(st));
    return BD_OK;
}

}  // namespace bd
