// mirror.cu -- the reference's entry points (encabezados.h:86-158) as sm_100a
// kernels behind the C ABI of include/bd_aging.h.  Same argument meaning and
// float3 array-of-structs layout as the reference; status codes instead of
// exit(); explicit streams; no write ever leaves its buffer.
#include <cuda.h>
#include <curand_kernel.h>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <type_traits>
#include <vector>

#include "gr_bins.cuh"
#include "runtime.cuh"

namespace bd {

// ------------------------------------------------------------ workspace
unsigned long long current_context_id() {
    using GetCurrent = CUresult (*)(CUcontext *);
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = (GetCurrent)f;
        f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &f, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = (GetId)f;
    });
    if (!get_current || !get_id) return 0;
    CUcontext c = nullptr;
    if (get_current(&c) != CUDA_SUCCESS || !c) {
        int dev = 0;  // no context yet on this thread: make the device's primary context current
        if (cudaGetDevice(&dev) != cudaSuccess || cudaSetDevice(dev) != cudaSuccess) return 0;
        if (get_current(&c) != CUDA_SUCCESS || !c) return 0;
    }
    unsigned long long id = 0;
    return get_id(c, &id) == CUDA_SUCCESS ? id + 1 : 0;  // +1: a valid id is never 0 here
}

namespace {
constexpr int kSlots = 32;
struct SlotState {
    std::atomic_flag busy = ATOMIC_FLAG_INIT;
};
struct SlotWords {  // on the device
    unsigned counter, pad[31];
    CallStatus status;
};
static_assert(sizeof(SlotWords) == 256, "on their own lines");
struct ContextSlots {
    HostWords *host = nullptr, *dev = nullptr;  // [kSlots] words, 128 bytes apart
    double *accum = nullptr;                    // [kSlots][kWorkAccum], then SlotWords [kSlots]
    unsigned long long ctx = 0;                 // context the pointers belong to
    SlotState slot[kSlots];
    ContextSlots *next = nullptr;
};
constexpr size_t kWordStride = 128 / sizeof(HostWords);
static_assert(128 % sizeof(HostWords) == 0, "slots on their own lines");

bool init_slots(void *acc, size_t sums, HostWords *dev) {
    SlotWords w[kSlots];
    std::memset(w, 0, sizeof(w));
    for (int k = 0; k < kSlots; k++) w[k].status.word = &dev[k * kWordStride].status;
    return cudaMemset(acc, 0, sums) == cudaSuccess &&
           cudaMemcpy(static_cast<char *>(acc) + sums, w, sizeof(w), cudaMemcpyHostToDevice) == cudaSuccess;
}

// The current context's slots, made on first use and never changed after: a
// context's id is its own for the life of the process, so one that was destroyed
// (its memory with it) leaves an entry that no call finds again.
ContextSlots *context_slots() {
    static std::mutex mu;
    static ContextSlots *all = nullptr;
    const unsigned long long ctx = current_context_id();
    if (!ctx) return nullptr;
    std::lock_guard<std::mutex> lock(mu);
    for (ContextSlots *d = all; d; d = d->next)
        if (d->ctx == ctx) return d;
    ContextSlots *d = new (std::nothrow) ContextSlots();
    if (!d) return nullptr;
    void *h = nullptr, *p = nullptr, *acc = nullptr;
    const size_t sums = sizeof(double) * kWorkAccum * kSlots, bytes = sums + sizeof(SlotWords) * kSlots;
    if (cudaHostAlloc(&h, 128 * kSlots, cudaHostAllocMapped) != cudaSuccess ||
        cudaHostGetDevicePointer(&p, h, 0) != cudaSuccess || cudaMalloc(&acc, bytes) != cudaSuccess ||
        !init_slots(acc, sums, static_cast<HostWords *>(p)) || cudaDeviceSynchronize() != cudaSuccess) {
        if (h) cudaFreeHost(h);
        if (acc) cudaFree(acc);
        delete d;
        return nullptr;
    }
    d->host = static_cast<HostWords *>(h);
    d->dev = static_cast<HostWords *>(p);
    d->accum = static_cast<double *>(acc);
    d->ctx = ctx;
    d->next = all;
    all = d;
    return d;
}
}  // namespace

CallSlot::CallSlot(cudaStream_t s) : stream(s) {
    ContextSlots *d = context_slots();
    if (!d) return;
    int k = 0;
    while (d->slot[k].busy.test_and_set(std::memory_order_acquire)) {
        if (++k == kSlots) {
            k = 0;
            std::this_thread::yield();
        }
    }
    state = &d->slot[k];
    host = d->host + k * kWordStride;
    dev = d->dev + k * kWordStride;
    accum = d->accum + (size_t)k * kWorkAccum;
    SlotWords *w = reinterpret_cast<SlotWords *>(d->accum + (size_t)kSlots * kWorkAccum) + k;
    counter = &w->counter;
    status = &w->status;
    host->status = 0;
}
cudaError_t CallSlot::wait() {
    waited = true;
    return cudaStreamSynchronize(stream);
}
CallSlot::~CallSlot() {
    if (!state) return;
    if (!waited) cudaStreamSynchronize(stream);
    if (*static_cast<volatile unsigned *>(&host->status)) {
        cudaMemsetAsync(status->seen, 0, sizeof(status->seen), stream);
        cudaStreamSynchronize(stream);
    }
    static_cast<SlotState *>(state)->busy.clear(std::memory_order_release);
}

// Waits for the call's kernels and maps their status.
static int read_status(CallSlot &w) {
    BD_CUDA_TRY(w.wait());
    return status_from_bits(*static_cast<volatile unsigned *>(&w.host->status));
}

// ------------------------------------------------------------ cell list
// cell_locate_dev (cell_locate.cu:155-209): cell (int)(cell_side_inv * x)
// with the inverse side a double division narrowed to float, ==ncell clamp,
// linear index i + n(j + n k), slot by atomic increment of nocup.
__global__ void k_cell_bin(const float *__restrict__ rr, int n, float csi, int ncell, int ntags, int *nocup,
                           int *cell_vec, CallStatus *st) {
    int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n) return;
    float x = rr[3 * m], y = rr[3 * m + 1], z = rr[3 * m + 2];
    if (!isfinite(x) || !isfinite(y) || !isfinite(z)) set_status(st, kStatNumeric);
    int ii = (int)__fmul_rn(csi, x), jj = (int)__fmul_rn(csi, y), kk = (int)__fmul_rn(csi, z);
    if (ii == ncell) ii--;
    if (jj == ncell) jj--;
    if (kk == ncell) kk--;
    if ((unsigned)ii >= (unsigned)ncell || (unsigned)jj >= (unsigned)ncell || (unsigned)kk >= (unsigned)ncell) {
        // outside the box: the reference would write out of bounds here
        set_status(st, kStatArg);
        ii = min(max(ii, 0), ncell - 1);
        jj = min(max(jj, 0), ncell - 1);
        kk = min(max(kk, 0), ncell - 1);
    }
    int c = ii + ncell * (jj + ncell * kk);
    int s = atomicAdd(&nocup[c], 1);
    if (s < ntags) cell_vec[(long)c * ntags + s] = m;
    if (s + 1 >= ntags) set_status(st, kStatCellOverflow);  // main.cu:655 (nocup_max >= ntags)
}
// Slots in ascending particle order (the order cell_locate_hst produces), the
// unused ones -1.  G lanes per cell (ntags <= G): a lane holds a slot's entry
// and counts the smaller ones by shuffles, so a cell is one load and one store
// per slot, and the clear of cell_vec before the binning is saved.
template <int G>
__global__ void k_cell_sort(const int *nocup, int *cell_vec, int nc3, int ntags) {
    const int c = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) / G), t = threadIdx.x % G;
    const bool live = c < nc3;
    const int k = live ? min(nocup[c], ntags) : 0;
    int *v = cell_vec + (size_t)c * ntags;
    const int key = t < k ? v[t] : INT_MAX;
    int rank = 0;
    const int most = __reduce_max_sync(0xffffffffu, k);  // of the warp's cells: two or three, not G
    for (int u = 0; u < most; u++) rank += __shfl_sync(0xffffffffu, key, u, G) < key;
    if (t < k) v[rank] = key;
    else if (live && t < ntags) v[t] = -1;
}
// The same for more slots per cell or many cells, a thread per cell (unused
// slots cleared before the binning).
__global__ void k_cell_sort_long(const int *nocup, int *cell_vec, int nc3, int ntags) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nc3) return;
    int k = min(nocup[c], ntags);
    int *v = cell_vec + (long)c * ntags;
    for (int a = 1; a < k; a++) {
        int key = v[a], b = a - 1;
        while (b >= 0 && v[b] > key) { v[b + 1] = v[b]; b--; }
        v[b + 1] = key;
    }
}

// ------------------------------------------------------------ forces
// get_forces_same_dev / get_forces_diff_dev (get_forces.cu:297-558): G lanes
// per particle share the (2 nrange + 1)^3 cells around its own cell of the
// partner species; pair selection with the reference's rounding (min_image_f,
// dist2_rn), WCA-modified pair; results ADDED to ff/vir/pot.
// Bound: the chain of loads position -> cell count -> cell entry -> partner
// position, which a thread per particle walks 27 or 125 times with 110 threads
// on an SM (16384 particles).  A warp per particle walks it once or four times
// and fills the chip; with more particles fewer lanes each, and so fewer
// instructions, win (launch_forces).  12 blocks an SM (40 registers): a thread
// per particle over 1.5 million waits for memory, 719 us with 48 warps on an SM,
// 799 with the 40 that 46 registers allow.
constexpr int kForceThreads = 128;
template <int G>  // the aligned group of G lanes that `lane` belongs to
__host__ __device__ constexpr unsigned lanes_of_group(int lane) {
    return (unsigned)(((1ull << G) - 1ull) << (lane & ~(G - 1)));
}
static_assert(lanes_of_group<32>(5) == 0xffffffffu && lanes_of_group<8>(0) == 0xffu &&
                  lanes_of_group<8>(15) == 0xff00u && lanes_of_group<8>(31) == 0xff000000u,
              "a particle's lanes");
template <bool SAME, int G, int W>
__global__ void __launch_bounds__(kForceThreads, 12) k_forces(const float *__restrict__ rr, float *ff, float *vir, float *pot,
                         const float *__restrict__ rr_o, const int *__restrict__ nocup,
                         const int *__restrict__ cell_vec, int n, int ncell, int ntags, int nrange, float csi,
                         float sigma, float side, CallStatus *st) {
    const int m = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) / G), sub = threadIdx.x % G;
    if (m >= n) return;  // the lanes of a particle leave together
    const float side_inv = __fdiv_rn(1.0f, side);
    const float cut2 = __fmul_rn(sigma, sigma);
    float rx = rr[3 * (size_t)m], ry = rr[3 * (size_t)m + 1], rz = rr[3 * (size_t)m + 2];
    int ii = (int)__fmul_rn(csi, rx), jj = (int)__fmul_rn(csi, ry), kk = (int)__fmul_rn(csi, rz);
    if (ii == ncell) ii--;
    if (jj == ncell) jj--;
    if (kk == ncell) kk--;
    if ((unsigned)ii >= (unsigned)ncell || (unsigned)jj >= (unsigned)ncell || (unsigned)kk >= (unsigned)ncell) {
        set_status(st, kStatArg);
        ii = min(max(ii, 0), ncell - 1);
        jj = min(max(jj, 0), ncell - 1);
        kk = min(max(kk, 0), ncell - 1);
    }
    float fx = 0.f, fy = 0.f, fz = 0.f, v = 0.f, p = 0.f;
    if (G == 1) fx = ff[3 * (size_t)m], fy = ff[3 * (size_t)m + 1], fz = ff[3 * (size_t)m + 2], v = vir[m], p = pot[m];
    const int w = W > 0 ? W : 2 * nrange + 1, reach = W > 0 ? W / 2 : nrange;
    auto wrap = [&](int k) {
        while (k < 0) k += ncell;
        while (k >= ncell) k -= ncell;
        return k;
    };
    auto visit = [&](int c) {
        int occ = min(nocup[c], ntags);
        const int *cv = cell_vec + (long)c * ntags;
#pragma unroll 2
        for (int t = 0; t < occ; t++) {
            int nn = cv[t];
            if (SAME && nn == m) continue;
            float dx = min_image_f(__fsub_rn(rr_o[3 * (size_t)nn], rx), side, side_inv);
            float dy = min_image_f(__fsub_rn(rr_o[3 * (size_t)nn + 1], ry), side, side_inv);
            float dz = min_image_f(__fsub_rn(rr_o[3 * (size_t)nn + 2], rz), side, side_inv);
            float d2 = dist2_rn(dx, dy, dz);
            if (d2 < cut2) {
                PairOut o = wca_modified_pair(sigma, d2, dx, dy, dz);
                fx += o.fx;
                fy += o.fy;
                fz += o.fz;
                p += o.pot;
                v += o.vir;
            }
        }
    };
    if (G == 1) {  // the reference's order of sums
        for (int di = -reach; di <= reach; di++) {
            const int ip = wrap(ii + di);
            for (int dj = -reach; dj <= reach; dj++) {
                const int jp = wrap(jj + dj);
                for (int dk = -reach; dk <= reach; dk++) visit(ip + ncell * (jp + ncell * wrap(kk + dk)));
            }
        }
    } else {  // consecutive lanes take cells that follow one another in memory (x runs fastest)
        for (int t0 = sub; t0 < w * w * w; t0 += G)
            visit(wrap(ii + t0 % w - reach) +
                  ncell * (wrap(jj + t0 / w % w - reach) + ncell * wrap(kk + t0 / (w * w) - reach)));
    }
    if (G > 1) {
        // this particle's lanes: they left together at m >= n, and the loop has not
        // rejoined them, which the shuffles do for the lanes they name
        const unsigned mask = lanes_of_group<G>(threadIdx.x & 31);
#pragma unroll
        for (int o = G / 2; o; o >>= 1) {
            fx += __shfl_xor_sync(mask, fx, o);
            fy += __shfl_xor_sync(mask, fy, o);
            fz += __shfl_xor_sync(mask, fz, o);
            v += __shfl_xor_sync(mask, v, o);
            p += __shfl_xor_sync(mask, p, o);
        }
        if (sub != 0) return;
        fx += ff[3 * (size_t)m], fy += ff[3 * (size_t)m + 1], fz += ff[3 * (size_t)m + 2], v += vir[m], p += pot[m];
    }
    ff[3 * (size_t)m] = fx;
    ff[3 * (size_t)m + 1] = fy;
    ff[3 * (size_t)m + 2] = fz;
    vir[m] = v;
    pot[m] = p;
}
template <bool SAME, int G>
static auto forces_kernel(int nrange) {
    return nrange == 1 ? k_forces<SAME, G, 3> : nrange == 2 ? k_forces<SAME, G, 5> : k_forces<SAME, G, 0>;
}
template <bool SAME>
static int launch_forces(const float *rr, float *ff, float *vir, float *pot, const float *rr_o, const int *nocup,
                         const int *cell_vec, int n, int ncell, int ntags, int nrange, float csi, float sigma, float side,
                         cudaStream_t s) {
    CallSlot w(s);
    if (!w.ok()) return BD_ERR_NOMEM;
    // lanes per particle.  A call's time (us) with 32, 8 and 1 lanes over 27
    // cells: 20, 24, 68 at 6000 particles; 30, 27, 74 at 16384; 64, 49, 76 at
    // 60000; 255, 163, 159 at 300000; over 125 cells: 26, 41, 193 at 6000; 45,
    // 46, 220 at 16384; 112, 106, 226 at 60000; 487, 402, 494 at 300000; with 8
    // and 1 lanes 546, 585 at 500000; 950, 893 at 800000; 2125, 1985 at 1.5 million.
    const int lanes = nrange > 1 ? (n <= 32768 ? 32 : n <= 655360 ? 8 : 1) : n <= 8192 ? 32 : n <= 131072 ? 8 : 1;
    auto kern = lanes == 32 ? forces_kernel<SAME, 32>(nrange) : lanes == 8 ? forces_kernel<SAME, 8>(nrange)
                                                                          : forces_kernel<SAME, 1>(nrange);
    kern<<<div_up((long)n * lanes, kForceThreads), kForceThreads, 0, s>>>(rr, ff, vir, pot, rr_o, nocup, cell_vec, n, ncell, ntags, nrange, csi,
                                                      sigma, side, w.status);
    BD_LAUNCH_CHECK();
    return read_status(w);
}

// ------------------------------------------------------------ update
__global__ void k_setup_rng(curandState *states, unsigned long long seed, int n) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) curand_init(seed, i, 0, &states[i]);
}
// update_ermak_dev (update_ermak.cu:91-160) with the reference's cuRAND
// stream; the expression is the reference's, so the compiler treats it alike.
__global__ void k_update_curand(float *rr, float *raw, const float *__restrict__ ff, curandState *states, int n,
                                float side, float side_inv, float dinv, float dt, float amplitude) {
    int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n) return;
    curandState s = states[m];
    float rx = amplitude * curand_normal(&s);
    float ry = amplitude * curand_normal(&s);
    float rz = amplitude * curand_normal(&s);
    states[m] = s;
    float tx = ff[3 * m] * dinv * dt + rx;
    float ty = ff[3 * m + 1] * dinv * dt + ry;
    float tz = ff[3 * m + 2] * dinv * dt + rz;
    float x = rr[3 * m] + tx, y = rr[3 * m + 1] + ty, z = rr[3 * m + 2] + tz;
    raw[3 * m] += tx;
    raw[3 * m + 1] += ty;
    raw[3 * m + 2] += tz;
    x -= side * floorf(side_inv * x);
    y -= side * floorf(side_inv * y);
    z -= side * floorf(side_inv * z);
    rr[3 * m] = x;
    rr[3 * m + 1] = y;
    rr[3 * m + 2] = z;
}
// update_ermak_hst (update_ermak.cu:8-77) with injected N(0,1) values, every
// operation rounded separately as on the host: bit-identical to it.
__global__ void k_update_noise(float *rr, float *raw, const float *__restrict__ ff, const float *__restrict__ noise,
                               int n, float side, float side_inv, float dinv, float dt, float amplitude) {
    int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= n) return;
#pragma unroll
    for (int k = 0; k < 3; k++) {
        float rnd = __fmul_rn(amplitude, noise[3 * m + k]);
        float tot = __fadd_rn(__fmul_rn(__fmul_rn(ff[3 * m + k], dinv), dt), rnd);
        float x = __fadd_rn(rr[3 * m + k], tot);
        raw[3 * m + k] = __fadd_rn(raw[3 * m + k], tot);
        rr[3 * m + k] = __fsub_rn(x, __fmul_rn(side, floorf(__fmul_rn(side_inv, x))));
    }
}

// ------------------------------------------------------------ g(r)
// get_gder_dev (get_gder.cu:69-127) as an exact integer histogram over all
// pairs.  A thread owns one particle of `ra` (256 a block); the partners
// [j0, j1) of the block are staged in shared memory and read as broadcasts,
// two per packed operation.  SAME: unordered pairs j > i, each counted in
// both directions.
//
// Bound: issue slots (no DRAM traffic to speak of).  What keeps a pair cheap:
//  - the minimum image is taken as fma(rint(d / L), -L, d).  When every
//    component of the result lies within 0.49999 L of zero, d / L is within
//    0.499995 of an integer k in {-1, 0, 1} (its rounding errors are below
//    4e-7), the reference's floor equals k and L k is exact, so the rounded
//    difference is the reference's, and that of the reverse pair is its
//    negation.  Pairs beyond that (they matter only when the range reaches
//    L / 2) and tiles with a coordinate outside [-0.2 L, 1.2 L] take the
//    reference's arithmetic in both directions (gder_pair_exact);
//  - the bin comes from an estimate (gr_bins.cuh), without a branch;
//  - every pair adds to its estimated slot with a plain shared atomic, into a
//    histogram copy per warp (fewer copies when they would pass 32 KB); an
//    open pair takes that count back.
// Blocks are cut over the partners until the grid has several per SM.
// Measured at 4095 + 4099 particles, 200 bins to L / 2, the four species
// pairs: 10.46 -> 0.11 ms (before: 16 to 128 blocks of 8192 partners, a square
// root and a divide per pair, a __match_any_sync histogram).
constexpr int kGderThreads = 256, kGderTile = 1024, kGderMaxCopies = kGderThreads / 32;
__device__ __forceinline__ int gder_bin(float dx, float dy, float dz, float side, float side_inv, float range,
                                        float range2_hi, float bin_size, int nbins) {
    dx = min_image_gder(dx, side, side_inv);
    dy = min_image_gder(dy, side, side_inv);
    dz = min_image_gder(dz, side, side_inv);
    float d2 = dist2_rn(dx, dy, dz);
    if (!(d2 <= range2_hi)) return -1;
    float dist = __fsqrt_rn(d2);
    if (!(dist < range)) return -1;
    int bin = (int)__fdiv_rn(dist, bin_size);
    if (bin == nbins) bin--;
    return bin;
}
struct GderArgs {
    const float *ra, *rb;
    int na, nb;
    float side, side_inv, range, range2_hi;
    GrBins bins;
    int jchunk, copies;
    unsigned long long *counts;
};
// one pair in the reference's arithmetic, both directions when SAME
template <bool SAME>
__device__ __noinline__ void gder_pair_exact(const GderArgs &a, float dx, float dy, float dz, unsigned *hist) {
    const int bf = gder_bin(dx, dy, dz, a.side, a.side_inv, a.range, a.range2_hi, a.bins.bin_size,
                            a.bins.nbins);
    if (bf >= 0) atomicAdd(&hist[bf], 1u);
    if (SAME) {
        const int br = gder_bin(-dx, -dy, -dz, a.side, a.side_inv, a.range, a.range2_hi, a.bins.bin_size,
                            a.bins.nbins);
        if (br >= 0) atomicAdd(&hist[br], 1u);
    }
}
template <bool SAME, bool CHECK>
__global__ void __launch_bounds__(kGderThreads) k_gder(const GderArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    float *tx = reinterpret_cast<float *>(smem);
    float *ty = tx + kGderTile, *tz = ty + kGderTile;
    unsigned *hist0 = reinterpret_cast<unsigned *>(tz + kGderTile);  // [copies][nbins + kGrSpare]
    const int i0 = blockIdx.x * kGderThreads, i = i0 + threadIdx.x;
    int j0 = blockIdx.y * a.jchunk;
    const int j1 = min(a.nb, j0 + a.jchunk);
    if (SAME) j0 = max(j0, i0 + 1);  // partners before the block's first particle: other blocks count them
    if (j0 >= j1) return;
    const int nbins = a.bins.nbins;
    const int stride = nbins + kGrSpare;
    unsigned *hist = hist0 + ((threadIdx.x >> 5) * a.copies / kGderMaxCopies) * stride;
    const unsigned row = gr_row(hist), top = gr_top(nbins, threadIdx.x & 31);
    for (int b = threadIdx.x; b < a.copies * stride; b += kGderThreads) hist0[b] = 0;
    const float wild_lo = -0.2f * a.side, wild_hi = 1.2f * a.side;
    auto wild_at = [&](float v) { return !(v >= wild_lo && v <= wild_hi); };
    const float nan = __int_as_float(0x7fffffff);  // a distance from it is never within range
    float xi = nan, yi = nan, zi = nan;
    bool wild = false;
    if (i < a.na) {
        xi = a.ra[3 * (size_t)i], yi = a.ra[3 * (size_t)i + 1], zi = a.ra[3 * (size_t)i + 2];
        wild = wild_at(xi) || wild_at(yi) || wild_at(zi);
    }
    const f2 XI = f2_bcast(xi), YI = f2_bcast(yi), ZI = f2_bcast(zi);
    const f2 SINV = f2_bcast(a.side_inv), NSIDE = f2_bcast(-a.side), MAGIC = f2_bcast(kRintMagic);
    const float edge = 0.49999f * a.side;
    const float lim = a.bins.near * (CHECK ? 1.0001f : 1.0f);
    constexpr unsigned kWeight = SAME ? 2u : 1u;
    for (int t0 = j0; t0 < j1; t0 += kGderTile) {
        const int tn = min(kGderTile, j1 - t0), tp = (tn + 3) & ~3;
        __syncthreads();
        for (int t = threadIdx.x; t < tp; t += kGderThreads) {
            float x = nan, y = nan, z = nan;  // padding
            if (t < tn) {
                const size_t j = 3 * (size_t)(t0 + t);
                x = a.rb[j], y = a.rb[j + 1], z = a.rb[j + 2];
                wild = wild || wild_at(x) || wild_at(y) || wild_at(z);
            }
            tx[t] = x, ty[t] = y, tz[t] = z;
        }
        if (__syncthreads_or(wild)) {
            if (i < a.na)
                for (int t = 0; t < tn; t++)
                    if (!SAME || t0 + t > i)
                        gder_pair_exact<SAME>(a, __fsub_rn(xi, tx[t]), __fsub_rn(yi, ty[t]), __fsub_rn(zi, tz[t]),
                                              hist);
            continue;
        }
        auto image = [&](f2 d) {
            return f2_fma(f2_sub(f2_fma(d, SINV, MAGIC), MAGIC), NSIDE, d);
        };
        // a pair whose estimate does not settle its bin
        auto settle = [&](unsigned slot, float dx, float dy, float dz, int t) {
            gr_uncount(row, slot, kWeight, nbins);
            if (CHECK && fmaxf(fmaxf(fabsf(dx), fabsf(dy)), fabsf(dz)) > edge) {
                gder_pair_exact<SAME>(a, __fsub_rn(xi, tx[t]), __fsub_rn(yi, ty[t]), __fsub_rn(zi, tz[t]), hist);
                return;
            }
            const float e2 = dist2_rn(dx, dy, dz);
            if (e2 < a.bins.thr) atomicAdd(&hist[gr_bin_settled(e2, a.bins)], kWeight);
        };
        auto pairs = [&](auto diagonal) {  // diagonal: some partner of the tile may not come after i
            constexpr bool kDiag = decltype(diagonal)::value;
            for (int t = 0; t < tp; t += 4) {
                const float4 x = *reinterpret_cast<const float4 *>(tx + t),
                             y = *reinterpret_cast<const float4 *>(ty + t),
                             z = *reinterpret_cast<const float4 *>(tz + t);
                float d2[4], dx[4], dy[4], dz[4];
                unsigned slot[4];
                bool open[4];
#pragma unroll
                for (int u = 0; u < 4; u += 2) {
                    const f2 DX = image(f2_sub(XI, u ? f2_make(x.z, x.w) : f2_make(x.x, x.y)));
                    const f2 DY = image(f2_sub(YI, u ? f2_make(y.z, y.w) : f2_make(y.x, y.y)));
                    const f2 DZ = image(f2_sub(ZI, u ? f2_make(z.z, z.w) : f2_make(z.x, z.y)));
                    const f2 D2 = f2_fma(DZ, DZ, f2_fma(DY, DY, f2_mul(DX, DX)));
                    f2_split(D2, d2[u], d2[u + 1]);
                    f2_split(DX, dx[u], dx[u + 1]);
                    f2_split(DY, dy[u], dy[u + 1]);
                    f2_split(DZ, dz[u], dz[u + 1]);
                    unsigned sl[2];
                    bool far[2];
                    gr_estimate(D2, a.bins, top, sl, far);
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int v = u + h;
                        bool in = d2[v] < lim;
                        if (kDiag && t0 + t + v <= i) in = false, sl[h] = top;
                        if (CHECK) far[h] = far[h] | (fmaxf(fmaxf(fabsf(dx[v]), fabsf(dy[v])), fabsf(dz[v])) > edge);
                        open[v] = in & far[h];
                        slot[v] = sl[h];
                        gr_count(row + 4u * sl[h], kWeight);
                    }
                }
                const bool any = open[0] | open[1] | open[2] | open[3];
                if (any) {
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (open[u]) settle(slot[u], dx[u], dy[u], dz[u], t + u);
                }
            }
        };
        if (SAME && t0 <= i0 + kGderThreads - 1) pairs(std::true_type{});
        else pairs(std::false_type{});
    }
    __syncthreads();
    for (int b = threadIdx.x; b < nbins; b += kGderThreads) {
        unsigned long long v = 0;
        for (int c = 0; c < a.copies; c++) v += hist0[c * stride + b];
        if (v) atomicAdd(&a.counts[b], v);
    }
}

// ------------------------------------------------------------ F_s, MSD
// fself_isotropic (fself.cu:3-21) and the MSD loop (main.cu:776-792): per
// particle float terms as in the reference, summed in FP64.
// One FP64 partial per block; the last block to finish adds the partials in
// index order into the call's host word, so the result does not depend on the
// order in which blocks finish.
constexpr int kDispThreads = 256, kDispMaxBlocks = 148 * 8;
static_assert(kDispMaxBlocks <= kWorkAccum, "partials fit the workspace");
template <int KIND>  // 0: F_s, 1: MSD
__global__ void __launch_bounds__(kDispThreads) k_disp_reduce(const float *__restrict__ raw,
                                                              const float *__restrict__ r0, int n, float q,
                                                              double *part, unsigned *counter, double *result) {
    double s = 0.0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float dx = raw[3 * i] - r0[3 * i], dy = raw[3 * i + 1] - r0[3 * i + 1], dz = raw[3 * i + 2] - r0[3 * i + 2];
        float d2 = dist2_rn(dx, dy, dz);
        if (KIND == 0) {
            float mag = __fsqrt_rn(d2);
            s += (double)(sinf(q * mag) / (q * mag));
        } else {
            s += (double)d2;
        }
    }
    for (int o = 16; o; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    __shared__ double red[kDispThreads];
    __shared__ bool last;
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kDispThreads / 32; w++) t += red[w];
        part[blockIdx.x] = t;
        __threadfence();
        last = atomicAdd(counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    s = 0.0;
    for (int b = threadIdx.x; b < gridDim.x; b += blockDim.x) s += __ldcg(part + b);
    red[threadIdx.x] = s;
    __syncthreads();
    for (int w = kDispThreads / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        *result = red[0];
        *counter = 0u;
    }
}

static int disp_reduce(int kind, const float *raw, const float *r0, int n, float q, double *out, cudaStream_t s) {
    CallSlot w(s);
    if (!w.ok()) return BD_ERR_NOMEM;
    const int blocks = std::min(div_up(n, kDispThreads), kDispMaxBlocks);
    auto kern = kind == 0 ? k_disp_reduce<0> : k_disp_reduce<1>;
    kern<<<blocks, kDispThreads, 0, s>>>(raw, r0, n, q, w.accum, w.counter, &w.dev->value);
    BD_LAUNCH_CHECK();
    BD_CUDA_TRY(w.wait());
    *out = *static_cast<volatile double *>(&w.host->value);
    return BD_OK;
}


// ------------------------------------------------------------ colours
// calculate_color / between (colors.cu:8-110) for every big particle, one
// thread each, in the reference's float operation order (rounding
// intrinsics: no contraction).  ids: 0 blue, 1 green, 2 red.
__device__ __forceinline__ bool between_dev(const float3 r1, const float3 r2, const float3 *__restrict__ rs, int ns,
                                            float side, float side_inv, float max_big, float max_line) {
    float ux = min_image_f(__fsub_rn(r1.x, r2.x), side, side_inv);
    float uy = min_image_f(__fsub_rn(r1.y, r2.y), side, side_inv);
    float uz = min_image_f(__fsub_rn(r1.z, r2.z), side, side_inv);
    const float ua = __fsqrt_rn(dist2_rn(ux, uy, uz));
    ux = __fdiv_rn(ux, ua);
    uy = __fdiv_rn(uy, ua);
    uz = __fdiv_rn(uz, ua);
    for (int i = 0; i < ns; i++) {
        const float3 r = rs[i];
        const float ax = min_image_f(__fsub_rn(r.x, r1.x), side, side_inv);
        const float ay = min_image_f(__fsub_rn(r.y, r1.y), side, side_inv);
        const float az = min_image_f(__fsub_rn(r.z, r1.z), side, side_inv);
        if (__fsqrt_rn(dist2_rn(ax, ay, az)) > max_big) continue;
        const float bx = min_image_f(__fsub_rn(r.x, r2.x), side, side_inv);
        const float by = min_image_f(__fsub_rn(r.y, r2.y), side, side_inv);
        const float bz = min_image_f(__fsub_rn(r.z, r2.z), side, side_inv);
        if (__fsqrt_rn(dist2_rn(bx, by, bz)) > max_big) continue;
        const float cx = __fsub_rn(__fmul_rn(ay, uz), __fmul_rn(az, uy));
        const float cy = __fadd_rn(__fmul_rn(-ax, uz), __fmul_rn(az, ux));
        const float cz = __fsub_rn(__fmul_rn(ax, uy), __fmul_rn(ay, ux));
        if (__fsqrt_rn(dist2_rn(cx, cy, cz)) > max_line) continue;
        return true;
    }
    return false;
}

__global__ void k_colors(const float3 *__restrict__ rb, int nb, const float3 *__restrict__ rs, int ns, float side,
                         float sigma_big, float sigma_sml, int *ids, unsigned *counts) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= nb) return;
    const float side_inv_c = __double2float_rn(1.0 / (double)side);  // calculate_color: 1.0 / side
    const float side_inv_b = __fdiv_rn(1.0f, side);                  // between: 1 / side
    const float max_big = __double2float_rn(0.5 * (double)sigma_big + 2.0 * (double)sigma_sml);
    const float max_line = __double2float_rn(0.35 * (double)sigma_big);
    const double near2 = (double)sigma_big + 2.0 * (double)sigma_sml;
    const float3 rm = rb[m];
    int cid = 0;
    bool near = false;
    for (int n = 0; n < nb; n++) {
        if (n == m) continue;
        const float3 rn = rb[n];
        const float dx = min_image_f(__fsub_rn(rn.x, rm.x), side, side_inv_c);
        const float dy = min_image_f(__fsub_rn(rn.y, rm.y), side, side_inv_c);
        const float dz = min_image_f(__fsub_rn(rn.z, rm.z), side, side_inv_c);
        if ((double)dist2_rn(dx, dy, dz) > near2) continue;  // squared distance against a length, as written
        cid += between_dev(rm, rn, rs, ns, side, side_inv_b, max_big, max_line) ? 1 : -1;
        near = true;
    }
    const int id = near ? (cid > 0 ? 2 : 1) : 0;
    if (ids) ids[m] = id;
    atomicAdd(&counts[id], 1u);
}

}  // namespace bd

using namespace bd;

// ====================================================================== ABI
extern "C" {

const char *bd_status_string(int s) {
    switch (s) {
        case BD_OK: return "ok";
        case BD_ERR_ARG: return "invalid argument";
        case BD_ERR_CUDA: return "CUDA runtime error";
        case BD_ERR_CELL_OVERFLOW: return "ntags reached limit (cell capacity exceeded)";
        case BD_ERR_NOMEM: return "out of memory";
        case BD_ERR_STATE: return "call out of order";
        case BD_ERR_TIMEOUT: return "bounded device wait expired";
        case BD_ERR_FILE: return "file missing or unreadable";
        case BD_ERR_FORMAT: return "malformed input";
        case BD_ERR_NUMERIC: return "non-finite position";
        default: return "unknown status";
    }
}
int bd_abi_version(void) { return BD_ABI_VERSION; }

// main.cu:155-163, 244-298, 348-349
int bd_setup_params(bd_parametros *p, float side, int nb, int ns, float sigma_big, float sigma_sml, float mass_big,
                    float mass_sml, int ntags_big, int ntags_sml, int nbins_gder, float range_gder, double dt,
                    float temp0) {
    if (!p || nb < 0 || ns < 0 || !(side > 0) || !(sigma_big > 0) || !(sigma_sml > 0) || nbins_gder < 1)
        return BD_ERR_ARG;
    std::memset(p, 0, sizeof(*p));
    p->dt = (float)dt;
    p->temp_set = temp0;
    p->nbins_gder = nbins_gder;
    p->range_gder = range_gder;
    p->ntags_big = ntags_big;
    p->ntags_sml = ntags_sml;
    p->bin_size_gder = range_gder / ((float)nbins_gder);
    p->side = side;
    p->ngrain_big = nb;
    p->ngrain_sml = ns;
    p->ngrain_tot = nb + ns;
    p->sigma_big = sigma_big;
    p->sigma_sml = sigma_sml;
    p->mass_big = mass_big;
    p->mass_sml = mass_sml;
    float cutoff = sigma_big;
    int ncb = (int)(side / (1.05 * cutoff));
    p->ncell_big = ncb;
    p->cell_side_big = side / ((float)ncb);
    cutoff = sigma_sml;
    int ncs = (int)(side / (1.05 * cutoff));
    p->ncell_sml = ncs;
    p->cell_side_sml = side / ((float)ncs);
    p->nrange_bb = 1;
    float aux = (float)((sigma_big + sigma_sml) / 2.0);
    p->nrange_bs = 1 + (int)(aux / p->cell_side_sml);
    p->nrange_sb = 1;
    p->nrange_ss = 1;
    p->NH = 256;
    return (ncb < 1 || ncs < 1) ? BD_ERR_ARG : BD_OK;
}

int bd_cell_locate(char type, const float *rr, int *nocup, int *cell_vec, const bd_parametros *p, void *stream) {
    if (!p || (type != 'b' && type != 's') || !nocup || !cell_vec) return BD_ERR_ARG;
    const bool b = type == 'b';
    const int n = b ? p->ngrain_big : p->ngrain_sml, ncell = b ? p->ncell_big : p->ncell_sml;
    const int ntags = b ? p->ntags_big : p->ntags_sml;
    if (ncell < 1 || ntags < 1 || n < 0 || (n > 0 && !rr)) return BD_ERR_ARG;
    const float csi = (float)(1.0 / (b ? p->cell_side_big : p->cell_side_sml));
    const int nc3 = ncell * ncell * ncell;
    cudaStream_t s = as_stream(stream);
    CallSlot w(s);
    if (!w.ok()) return BD_ERR_NOMEM;
    BD_CUDA_TRY(cudaMemsetAsync(nocup, 0, sizeof(int) * (size_t)nc3, s));
    // 16 or 32 lanes per cell (a call's time, us, lanes / a thread per cell: 16
    // slots 27 / 32 at 343 cells, 25 / 30 at 35937, 29 / 30 at 68921, 35 / 31 at
    // 250047, 110 / 53 at 1.8 million; 32 slots 25 / 33 at 9261, 28 / 28 at 35937,
    // 46 / 32 at 250047): up to a million lanes the launch and clear saved count
    // more, beyond it the lanes that hold no entry do
    const int lanes = ntags <= 16 ? 16 : 32;
    const bool by_lanes = ntags <= 32 && (long long)nc3 * lanes <= 1 << 20;
    if (!by_lanes) BD_CUDA_TRY(cudaMemsetAsync(cell_vec, 0xff, sizeof(int) * (size_t)nc3 * ntags, s));
    if (n > 0) {
        k_cell_bin<<<div_up(n, 256), 256, 0, s>>>(rr, n, csi, ncell, ntags, nocup, cell_vec, w.status);
        BD_LAUNCH_CHECK();
    }
    if (by_lanes && lanes == 16) k_cell_sort<16><<<div_up((long)nc3 * 16, 256), 256, 0, s>>>(nocup, cell_vec, nc3, ntags);
    else if (by_lanes) k_cell_sort<32><<<div_up((long)nc3 * 32, 256), 256, 0, s>>>(nocup, cell_vec, nc3, ntags);
    else k_cell_sort_long<<<div_up(nc3, 256), 256, 0, s>>>(nocup, cell_vec, nc3, ntags);
    BD_LAUNCH_CHECK();
    return read_status(w);
}

int bd_get_forces_same(char type, const float *rr, float *ff, float *vir, float *pot, const int *nocup,
                       const int *cell_vec, const bd_parametros *p, void *stream) {
    if (!p || (type != 'b' && type != 's')) return BD_ERR_ARG;
    const bool b = type == 'b';
    const int n = b ? p->ngrain_big : p->ngrain_sml;
    if (n == 0) return BD_OK;
    if (!rr || !ff || !vir || !pot || !nocup || !cell_vec) return BD_ERR_ARG;
    const float sigma = b ? p->sigma_big : p->sigma_sml;
    const float csi = 1.0f / (b ? p->cell_side_big : p->cell_side_sml);
    const int ntags = b ? p->ntags_big : p->ntags_sml, ncell = b ? p->ncell_big : p->ncell_sml;
    const int nrange = b ? p->nrange_bb : p->nrange_ss;
    return launch_forces<true>(rr, ff, vir, pot, rr, nocup, cell_vec, n, ncell, ntags, nrange, csi, sigma, p->side,
                               as_stream(stream));
}

int bd_get_forces_diff(char type, char type_other, const float *rr, float *ff, const float *rr_other, float *vir,
                       float *pot, const int *nocup_o, const int *cell_o, const bd_parametros *p, void *stream) {
    if (!p || (type != 'b' && type != 's') || (type_other != 'b' && type_other != 's') || type == type_other)
        return BD_ERR_ARG;
    const bool b = type == 'b';
    const int n = b ? p->ngrain_big : p->ngrain_sml;
    if (n == 0) return BD_OK;
    if (!rr || !ff || !vir || !pot || !nocup_o || !cell_o || !rr_other) return BD_ERR_ARG;
    const float csi = 1.0f / (b ? p->cell_side_sml : p->cell_side_big);
    const float sigma = b ? 0.5f * (p->sigma_big + p->sigma_sml) : 0.5f * (p->sigma_sml + p->sigma_big);
    const int ntags = b ? p->ntags_sml : p->ntags_big, ncell = b ? p->ncell_sml : p->ncell_big;
    const int nrange = b ? p->nrange_bs : p->nrange_sb;
    return launch_forces<false>(rr, ff, vir, pot, rr_other, nocup_o, cell_o, n, ncell, ntags, nrange, csi, sigma, p->side,
                                as_stream(stream));
}

size_t bd_rng_state_size(void) { return sizeof(curandState); }

int bd_setup_rng(void *states, unsigned long long seed, int n, void *stream) {
    if (n < 0 || (n > 0 && !states)) return BD_ERR_ARG;
    if (n == 0) return BD_OK;
    k_setup_rng<<<div_up(n, 256), 256, 0, as_stream(stream)>>>((curandState *)states, seed, n);
    BD_LAUNCH_CHECK();
    return BD_OK;
}

static int update_common(char type, const bd_parametros *p, int &n, float &side_inv, float &dinv, float &amp) {
    if (!p || (type != 'b' && type != 's')) return BD_ERR_ARG;
    n = type == 'b' ? p->ngrain_big : p->ngrain_sml;
    float diameter = type == 'b' ? p->sigma_big : p->sigma_sml;
    side_inv = 1.0f / p->side;
    dinv = 1.0f / diameter;
    amp = (float)std::sqrt(2.0 * p->temp_set * dinv * p->dt);  // update_ermak.cu:114
    return BD_OK;
}

int bd_update_ermak(char type, float *rr, float *rr_raw, const float *ff, void *states, const bd_parametros *p,
                    void *stream) {
    int n;
    float side_inv, dinv, amp;
    int rc = update_common(type, p, n, side_inv, dinv, amp);
    if (rc) return rc;
    if (n == 0) return BD_OK;
    if (!rr || !rr_raw || !ff || !states) return BD_ERR_ARG;
    k_update_curand<<<div_up(n, 256), 256, 0, as_stream(stream)>>>(rr, rr_raw, ff, (curandState *)states, n, p->side,
                                                                   side_inv, dinv, p->dt, amp);
    BD_LAUNCH_CHECK();
    return BD_OK;
}

int bd_update_ermak_noise(char type, float *rr, float *rr_raw, const float *ff, const float *noise,
                          const bd_parametros *p, void *stream) {
    int n;
    float side_inv, dinv, amp;
    int rc = update_common(type, p, n, side_inv, dinv, amp);
    if (rc) return rc;
    if (n == 0) return BD_OK;
    if (!rr || !rr_raw || !ff || !noise) return BD_ERR_ARG;
    k_update_noise<<<div_up(n, 256), 256, 0, as_stream(stream)>>>(rr, rr_raw, ff, noise, n, p->side, side_inv, dinv,
                                                                  p->dt, amp);
    BD_LAUNCH_CHECK();
    return BD_OK;
}

float bd_calculate_temp_linear(float T0, float Tf, float t0, float tf, float t) {
    return temp_linear(T0, Tf, t0, tf, t);
}
// set_temp.cu:14-23
float bd_calculate_temp_sine(float T0, float Tf, float t0, float tf, float period, float t) {
    if (t < t0) return T0;
    if (t > tf) return Tf;
    float a = (float)(0.5 * (T0 + Tf));
    float b = (float)(0.5 * (Tf - T0));
    float argument = (float)(2 * kRefPi * (t / period - 0.25));
    volatile float sn = sinf(argument);
    volatile float bs = b * sn;
    return a + bs;
}

int bd_get_gder(char type, char type_other, const float *rr, const float *rr_other, unsigned long long *counts,
                const bd_parametros *p, void *stream) {
    if (!p || (type != 'b' && type != 's') || (type_other != 'b' && type_other != 's') || !counts) return BD_ERR_ARG;
    const int na = type == 'b' ? p->ngrain_big : p->ngrain_sml;
    const int nb = type_other == 'b' ? p->ngrain_big : p->ngrain_sml;
    const int nbins = p->nbins_gder;
    if (nbins < 1 || nbins > 8192 || !(p->range_gder > 0)) return BD_ERR_ARG;
    if (na == 0 || nb == 0) return BD_OK;
    if (!rr || !rr_other) return BD_ERR_ARG;
    GderArgs a;
    a.ra = rr;
    a.rb = rr_other;
    a.na = na;
    a.nb = nb;
    a.side = p->side;
    a.side_inv = (float)(1.0 / a.side);
    a.range = p->range_gder;
    a.range2_hi = a.range * a.range * 1.00001f;
    a.bins = gr_bins(a.range, nbins, 0.0);
    a.counts = counts;
    const bool same = type == type_other;
    // partners per block: enough blocks for 8 of 256 threads on each SM (half
    // of the grid of equal species is empty), in tiles of at least 64 so that
    // the histogram's clear and flush stay a small part
    const int rows = div_up(na, kGderThreads);
    const long want = (long)148 * 8 * (same ? 2 : 1);
    const long per = ((long)rows * nb / want + 63) / 64 * 64;
    a.jchunk = (int)std::min(8192L, std::max(64L, per));
    a.copies = kGderMaxCopies;  // a power of two
    while (a.copies > 1 && (size_t)a.copies * (nbins + kGrSpare) * sizeof(unsigned) > 32 * 1024) a.copies /= 2;
    const dim3 grid(rows, div_up(nb, a.jchunk));
    const size_t sm = 3 * kGderTile * sizeof(float) + (size_t)a.copies * (nbins + kGrSpare) * sizeof(unsigned);
    cudaStream_t s = as_stream(stream);
    // pairs at the edge of the minimum image may be within range
    const float edge = 0.49998f * a.side;
    const bool check = !(a.bins.near <= edge * edge);
    auto kern = same ? (check ? k_gder<true, true> : k_gder<true, false>)
                     : (check ? k_gder<false, true> : k_gder<false, false>);
    if (sm > 48 * 1024)
        if (int rc = allow_smem(kern, sm)) return rc;
    kern<<<grid, kGderThreads, sm, s>>>(a);
    BD_LAUNCH_CHECK();
    return BD_OK;
}

// main.cu:847-877 for one sample (host arithmetic as in the reference)
int bd_gder_normalize(const double *counts, int nbins, float bin_size, float side, int nb, int ns, float sigma_big,
                      float sigma_sml, int n_configs, float *gder) {
    if (!counts || !gder || nbins < 1 || n_configs < 1) return BD_ERR_ARG;
    const float volume = side * side * side, xb = (float)nb, xs = (float)ns;
    for (int k = 0; k < nbins; k++) {
        float xnb = (float)k;
        volatile float xnb2 = xnb * xnb;
        float shell_vol = (float)(4.0 * kRefPi * bin_size * bin_size * bin_size * ((1.0 / 3.0) + xnb2 + xnb));
        float g[4];
        for (int j = 0; j < 4; j++) g[j] = (float)counts[j * nbins + k];
        float sigma = sigma_big;
        float vol_free = (float)(volume - (4.0 / 3.0) * kRefPi * sigma * sigma * sigma);
        g[0] = g[0] / shell_vol;
        g[0] = (float)(g[0] / (xb * (xb - 1.0) / vol_free));
        sigma = (float)(0.5 * (sigma_big + sigma_sml));
        vol_free = (float)(volume - (4.0 / 3.0) * kRefPi * sigma * sigma * sigma);
        g[1] = g[1] / shell_vol;
        g[2] = g[2] / shell_vol;
        volatile float pbs = xb * xs, psb = xs * xb;
        g[1] /= (pbs / vol_free);
        g[2] /= (psb / vol_free);
        sigma = sigma_sml;
        vol_free = (float)(volume - (4.0 / 3.0) * kRefPi * sigma * sigma * sigma);
        g[3] = g[3] / shell_vol;
        g[3] = (float)(g[3] / (xs * (xs - 1.0) / vol_free));
        for (int j = 0; j < 4; j++) gder[j * nbins + k] = g[j] / n_configs;
    }
    return BD_OK;
}

int bd_fself_isotropic(const float *rr_raw, const float *rr0, int ngrain, float *fself_host, int sample_number,
                       float qmax, void *stream) {
    if (ngrain <= 0 || !rr_raw || !rr0 || !fself_host || sample_number < 0) return BD_ERR_ARG;
    double sum = 0.0;
    int rc = disp_reduce(0, rr_raw, rr0, ngrain, qmax, &sum, as_stream(stream));
    if (rc) return rc;
    fself_host[sample_number] += (float)(sum / ngrain);
    return BD_OK;
}

int bd_color_statistics(const float *rr_big, const float *rr_sml, int *color_ids, int *counts_host,
                        const bd_parametros *p, void *stream) {
    if (!p || !counts_host || p->ngrain_big < 0 || p->ngrain_sml < 0) return BD_ERR_ARG;
    counts_host[0] = counts_host[1] = counts_host[2] = 0;
    const int nb = p->ngrain_big, ns = p->ngrain_sml;
    if (nb == 0) return BD_OK;
    if (!rr_big || (ns > 0 && !rr_sml)) return BD_ERR_ARG;
    cudaStream_t s = as_stream(stream);
    unsigned *d_counts = nullptr;
    BD_CUDA_TRY(cudaMalloc(&d_counts, 3 * sizeof(unsigned)));
    cudaError_t ce = cudaMemsetAsync(d_counts, 0, 3 * sizeof(unsigned), s);
    if (ce == cudaSuccess) {
        k_colors<<<div_up(nb, 128), 128, 0, s>>>(reinterpret_cast<const float3 *>(rr_big), nb,
                                                 reinterpret_cast<const float3 *>(rr_sml), ns, p->side,
                                                 p->sigma_big, p->sigma_sml, color_ids, d_counts);
        ce = cudaGetLastError();
    }
    unsigned h[3] = {0, 0, 0};
    if (ce == cudaSuccess) ce = cudaMemcpyAsync(h, d_counts, sizeof(h), cudaMemcpyDeviceToHost, s);
    if (ce == cudaSuccess) ce = cudaStreamSynchronize(s);
    cudaFree(d_counts);
    if (ce != cudaSuccess) return BD_ERR_CUDA;
    for (int k = 0; k < 3; k++) counts_host[k] = (int)h[k];
    return BD_OK;
}

int bd_msd(const float *rr_raw, const float *rr0, int ngrain, float *msd_host, void *stream) {
    if (ngrain <= 0 || !rr_raw || !rr0 || !msd_host) return BD_ERR_ARG;
    double sum = 0.0;
    int rc = disp_reduce(1, rr_raw, rr0, ngrain, 0.0f, &sum, as_stream(stream));
    if (rc) return rc;
    *msd_host = (float)(sum / ngrain);
    return BD_OK;
}

}  // extern "C"
