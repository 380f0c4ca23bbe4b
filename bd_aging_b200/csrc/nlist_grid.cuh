// nlist_grid.cuh -- list steps of mid-size batches, resident on the whole grid.
//
// Between the replicas that fit a cluster (nlist_cluster.cuh) and the batches
// that fill the chip for tens of microseconds per step, a step of the per-step
// path is its four launches: 9.1 us for one replica of 32768 particles, whose
// arithmetic is 1.5 us of the chip's issue slots.  Here one cooperative launch
// runs a whole batch of steps, a thread per particle:
//  - the particle's state (position, remainder, build position, crossings)
//    stays in registers, its list in shared memory; positions are exchanged
//    through the two by-id buffers in global memory;
//  - one grid barrier per step (arrivals counted in an L2 word) publishes the
//    new positions; the count's upper half tells whether any particle left
//    half the skin, so the rebuild decision needs no other exchange;
//  - as many threads again draw the next step's Gaussians meanwhile (blocks of
//    up to 256 particles; larger ones draw between their arrival and the wait);
//  - a rebuild clears and bins the flagged replicas' cells between two more
//    grid barriers, then every thread of a flagged replica scans its 27 cells.
//    Buckets stay unsorted: hits are inserted in storage-id order within their
//    cell, the order of the sorted builds.
// Lists, force sums, updates and rebuild decisions are those of the other
// launches, so the bits are the same.  The barrier's wait has a limit, after
// which the kernel raises the timeout status and returns.
// Measured at T = 0.1, us a step (per-step launches): 3.1 (8.4) at 4000
// particles, 3.3 (8.7) at 16000, 3.6 (9.1) at 32768 and 4.7 (10.0) at 2 x 32768.
#pragma once

namespace bd {

constexpr int kGridMaxOwners = 512;            // particles per block; threads per block (128 registers each)
// polls of a barrier (a second or so).  A constant: as a launch argument it made
// 192 steps of 4000 particles 587 us instead of 567
constexpr unsigned kGridSpinLimit = 1u << 21;

__host__ __device__ inline size_t grid_smem_bytes(int owners) { return (size_t)(kMaxNbr * 4 + 24) * owners; }

struct ListGrid {  // lists in shared memory, positions in global memory; entries are storage ids (np: absent)
    const float4 *pos;
    const int4 *list;
    int stride, none;
    __device__ __forceinline__ void words(int k0, int (&jn)[kGather]) const {
        const int4 w = list[(k0 >> 2) * stride];
        jn[0] = w.x;
        jn[1] = w.y;
        jn[2] = w.z;
        jn[3] = w.w;
    }
    __device__ __forceinline__ void gather(const int (&jn)[kGather], int (&jj)[kGather], float4 (&pj)[kGather]) const {
#pragma unroll
        for (int u = 0; u < kGather; u++) {
            jj[u] = jn[u];
            pj[u] = pos[jj[u]];
        }
    }
};

// Grid barrier on two words used in turn: arrivals in the low half, arrivals
// that ask for a rebuild in the high half, both counting up from zero at the
// launch.  A block that runs ahead arrives at the next barrier on the other
// word and waits there, so a slow block reads exactly this barrier's askers.
struct GridBarrier {
    unsigned long long *word;
    unsigned phase = 0, rounds = 0;  // word of the next barrier, barriers it has completed
    __device__ __forceinline__ explicit GridBarrier(unsigned long long *w) : word(w) {}
    // by one thread of the block, after a block barrier
    __device__ __forceinline__ void arrive(bool ask) {
        __threadfence();
        atomicAdd(word + phase, 1ull + (ask ? 1ull << 32 : 0ull));
    }
    // by the same thread: false when the limit is reached
    __device__ __forceinline__ bool wait(unsigned long long &v) const {
        const int target = (int)((rounds + 1u) * gridDim.x);
        for (unsigned k = 0; k < kGridSpinLimit; k++) {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(word + phase) : "memory");
            if ((int)(unsigned)v >= target) return true;
        }
        return false;
    }
    // by every thread, after the wait
    __device__ __forceinline__ void next() {
        rounds += phase;
        phase ^= 1u;
    }
};

// Partners of the particle at v from unsorted cell buckets, in the staged
// sweep's order (rows dz, dy of three cells dx, each cell by storage id), into
// list words put(k, j) / get(k); returns their number (words up to kMaxNbr).
template <class PUT, class GET>
__device__ __forceinline__ int bucket_partners(const SysDev &S, float4 v, const int *cnt, const float4 *bucket, int cap,
                                               PUT put, GET get) {
    const int nc = S.ncell;
    const int sid = (int)(__float_as_uint(v.w) & 0x7fffffffu);
    const int tm = (int)(__float_as_uint(v.w) >> 31);
    const float cut_b = S.lcut2[tm], cut_s = S.lcut2[tm + 1];  // towards a big / a small partner
    const float L = S.L;
    const int3 c = list_cell_of(v, S);
    int found = 0;
#pragma unroll 1
    for (int row = 0; row < 9; row++) {
        float shy, shz, shx[3];
        const int gz = wrap_cell(c.z + row / 3 - 1, nc, L, shz), gy = wrap_cell(c.y + row % 3 - 1, nc, L, shy);
        const bool wrap = c.x == 0 || c.x == nc - 1 || shy != 0.f || shz != 0.f;
        int cell[3], m[3];
#pragma unroll
        for (int d = 0; d < 3; d++) {
            cell[d] = S.cell_base + wrap_cell(c.x + d - 1, nc, L, shx[d]) + nc * (gy + nc * gz);
            m[d] = cnt[cell[d]];
        }
#pragma unroll
        for (int d = 0; d < 3; d++) {
            const float4 *b = bucket + (size_t)cell[d] * cap;
            const int n = min(m[d], cap), first = found;
            for (int k0 = 0; k0 < n; k0 += 4) {
                float4 q[4];
#pragma unroll
                for (int u = 0; u < 4; u++) q[u] = b[min(k0 + u, n - 1)];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const unsigned w = __float_as_uint(q[u].w);
                    const int sj = (int)(w & 0x7fffffffu);
                    const float ex = __fsub_rn(__fsub_rn(q[u].x, v.x), shx[d]);
                    const float ey = __fsub_rn(__fsub_rn(q[u].y, v.y), shy);
                    const float ez = __fsub_rn(__fsub_rn(q[u].z, v.z), shz);
                    if (k0 + u < n && sj != sid &&
                        list_build_d2(ex, ey, ez, wrap) < ((w >> 31) ? cut_s : cut_b)) {
                        if (found < kMaxNbr) {
                            int k = found;
                            for (; k > first; k--) {
                                const int p = get(k - 1);
                                if (p < sj) break;
                                put(k, p);
                            }
                            put(k, sj);
                        }
                        found++;
                    }
                }
            }
        }
    }
    return found;
}

// nsteps steps (at most the amplitude table's batch) of every replica, Philox
// noise.  The first T threads of a block own a particle each; with HELP the
// other T draw the noise of the step after theirs.
template <bool EXTRA, bool HELP>
__global__ void __launch_bounds__(kGridMaxOwners, 1)
    k_list_grid(ListArgs a, ListPersist lp, const long long *ni_base, int nsteps, unsigned long long *bar_word) {
    extern __shared__ __align__(16) unsigned char dsm[];
    __shared__ unsigned long long s_word;
    __shared__ int s_ok;
    const int T = HELP ? (int)blockDim.x >> 1 : (int)blockDim.x;
    const bool owner = !HELP || threadIdx.x < T;
    const int tid = owner ? threadIdx.x : threadIdx.x - T;
    int4 *s_list = reinterpret_cast<int4 *>(dsm);                                   // [kMaxNbr / 4][T]
    float *s_noise = reinterpret_cast<float *>(s_list + (size_t)(kMaxNbr / 4) * T);  // [2][3][T]
    const int first = (int)((long long)a.np * blockIdx.x / gridDim.x);
    const int count = (int)((long long)a.np * (blockIdx.x + 1) / gridDim.x) - first;
    const bool live = tid < count;
    const int sid = first + (live ? tid : 0);
    const int rep = a.rep_of_sid[sid];
    const SysDev &S = a.sys[rep];
    int *my_list = reinterpret_cast<int *>(s_list + tid);
    auto list_at = [&](int k) { return ((size_t)(k >> 2) * T) * 4 + (k & 3); };
    const float4 *pos0 = lp.pos[0], *pos1 = lp.pos[1];
    float4 pi = (lp.cur0 & 1) ? pos1[sid] : pos0[sid];
    const int tm = (int)(__float_as_uint(pi.w) >> 31);
    const int gid = a.gid_of[sid], pid = gid - S.part_base;
    const long long ni0 = *ni_base;
    const unsigned long long seed = S.seed;
    auto draw_noise = [&](int s) {  // amplitude times the Gaussians of step s
        if (!live || s >= nsteps) return;
        const float3 xi = gauss3(seed, (uint32_t)pid, (uint64_t)(ni0 + s), a.rng_stream);
        const float amp = __ldg(a.amp_tab + ((size_t)s * a.nrep + rep) * 2 + tm);
        float *z = s_noise + (s & 1) * 3 * T + tid;
        z[0] = __fmul_rn(amp, xi.x);
        z[T] = __fmul_rn(amp, xi.y);
        z[2 * T] = __fmul_rn(amp, xi.z);
    };
    float4 pb = a.pbuild[sid];
    float lx = a.lo_x[sid], ly = a.lo_y[sid], lz = a.lo_z[sid];
    int ix = a.img[sid], iy = a.img[a.np + sid], iz = a.img[2 * a.np + sid];
    int nl = min(a.nnb[sid], kMaxNbr);
    bool rebuilt = false;
    auto pad_list = [&]() {
        for (int k = nl; k % kClusterGroup != 0; k++) my_list[list_at(k)] = a.np;
    };
    bool need = a.flag[a.nrep] != 0;  // some replica needs a rebuild: the same in every block
    if (!HELP || !owner) draw_noise(0);
    if (owner && live && a.flag[rep] == 0) {
        for (int k = 0; k < nl; k += kGather)
            s_list[(size_t)(k >> 2) * T + tid] = reinterpret_cast<const int4 *>(a.nbr)[(size_t)(k >> 2) * a.np + sid];
        pad_list();
    }
    const float L = S.L, Linv = S.Linv, mob = S.mob[tm], dt = S.dt;
    const float sg0 = tm ? S.sig[1] : S.sig[0], sg1 = tm ? S.sig[2] : S.sig[1];
    const float c0 = tm ? S.cut2[1] : S.cut2[0], c1 = tm ? S.cut2[2] : S.cut2[1];
    const bool general = (EXTRA && S.pot != kPotWcaModified) || S.fcap > 0.f;
    const float skin_half2 = S.skin_half2;
    GridBarrier bar(bar_word);
    unsigned asked0 = 0, asked1 = 0;  // askers so far on either word
    // the whole grid waits; true (and the word) unless the limit was reached
    auto grid_wait = [&]() {
        if (threadIdx.x == 0) {
            unsigned long long v = 0;
            s_ok = bar.wait(v) ? 1 : 0;
            s_word = v;
            if (!s_ok) set_status(a.status, kStatTimeout);
        }
        __syncthreads();
        bar.next();
        return s_ok != 0;
    };
    auto grid_sync = [&]() {
        __syncthreads();
        if (threadIdx.x == 0) bar.arrive(false);
        return grid_wait();
    };
    __syncthreads();
    for (int s = 0; s < nsteps; s++) {
        const bool odd = ((lp.cur0 + s) & 1) != 0;
        const float4 *cur = odd ? pos1 : pos0;
        float4 *nxt = odd ? lp.pos[0] : lp.pos[1];
        if (need) {
            const bool mine = a.flag[rep] != 0;
            const int me = blockIdx.x * blockDim.x + threadIdx.x, all = gridDim.x * blockDim.x;
            // a flagged replica's particles clear its cells (a walk over the
            // replicas by every thread took 0.15 us a replica, 38 us at 300)
            if (owner && live && mine) {
                const int cells = S.ncell * S.ncell * S.ncell, n = S.n, base = S.cell_base;
                for (int c = sid - S.part_base; c < cells; c += n) lp.cnt[base + c] = 0;
            }
            if (!grid_sync()) return;
            if (me < a.nrep || (blockIdx.x == 0 && threadIdx.x == 0)) {  // every block has read the flags
                for (int r = me; r < a.nrep; r += all)
                    if (a.flag[r]) {
                        atomicAdd((unsigned long long *)lp.builds, 1ull);
                        a.flag[r] = 0;
                    }
                if (me == 0) lp.step_rebuilt[s] = 1;
            }
            if (owner && live && mine) {
                const int3 c = list_cell_of(pi, S);
                const int cell = S.cell_base + c.x + S.ncell * (c.y + S.ncell * c.z);
                const int slot = atomicAdd(lp.cnt + cell, 1);
                if (slot < lp.cap) lp.bucket[(size_t)cell * lp.cap + slot] = pi;
                else set_status(a.status, kStatCellOverflow);
            }
            if (!grid_sync()) return;
            if (owner && live && mine) {
                const int found = bucket_partners(
                    S, pi, lp.cnt, lp.bucket, lp.cap, [&](int k, int j) { my_list[list_at(k)] = j; },
                    [&](int k) { return my_list[list_at(k)]; });
                if (found > kMaxNbr) set_status(a.status, kStatCellOverflow);
                nl = min(found, kMaxNbr);
                pad_list();
                pb = pi;
                rebuilt = true;
            }
        }
        bool beyond = false;
        if (!owner) {
            draw_noise(s + 1);
        } else if (live) {
            const float *z = s_noise + (s & 1) * 3 * T + tid;
            const float nx = z[0], ny = z[T], nz = z[2 * T];
            float fx, fy, fz;
            const ListGrid src{cur, s_list + tid, T, a.np};
            if (general) {
                int jn[kGather];
                src.words(0, jn);
                list_force<EXTRA>(src, S, nl, jn, pi, tm, fx, fy, fz);
            } else {
                list_forces_wide(src, nl, pi, L, Linv, sg0 * sg0, sg1 * sg1, c0, c1, fx, fy, fz);
            }
            if (ni0 + s == 0) {  // origin of the unwrapped positions (main.cu:497-506)
                a.x0[3 * (size_t)gid] = (double)pi.x + (double)lx;
                a.x0[3 * (size_t)gid + 1] = (double)pi.y + (double)ly;
                a.x0[3 * (size_t)gid + 2] = (double)pi.z + (double)lz;
                ix = iy = iz = 0;
            }
            const float ex = __fadd_rn(__fmul_rn(__fmul_rn(fx, mob), dt), nx);
            const float ey = __fadd_rn(__fmul_rn(__fmul_rn(fy, mob), dt), ny);
            const float ez = __fadd_rn(__fmul_rn(__fmul_rn(fz, mob), dt), nz);
            ix += (int)advance_wrap(pi.x, lx, ex, L, Linv);
            iy += (int)advance_wrap(pi.y, ly, ey, L, Linv);
            iz += (int)advance_wrap(pi.z, lz, ez, L, Linv);
            nxt[sid] = pi;
            if (!(isfinite(pi.x) && isfinite(pi.y) && isfinite(pi.z))) set_status(a.status, kStatNumeric);
            beyond = list_beyond(pi.x, pi.y, pi.z, pb, L, Linv, skin_half2);
            if (beyond) a.flag[rep] = 1;
        }
        const bool ask = __syncthreads_or(beyond) != 0;
        if (threadIdx.x == 0) bar.arrive(ask);
        if (!HELP) draw_noise(s + 1);
        if (!grid_wait()) return;
        const unsigned now = (unsigned)(s_word >> 32);
        unsigned &before = bar.phase ? asked0 : asked1;  // the barrier was on the other word
        need = now != before;
        before = now;
    }
    if (owner && live) {
        a.lo_x[sid] = lx;
        a.lo_y[sid] = ly;
        a.lo_z[sid] = lz;
        a.img[sid] = ix;
        a.img[a.np + sid] = iy;
        a.img[2 * a.np + sid] = iz;
        if (rebuilt) {
            for (int k = 0; k < nl; k += kGather)
                reinterpret_cast<int4 *>(lp.nbr)[(size_t)(k >> 2) * a.np + sid] = s_list[(size_t)(k >> 2) * T + tid];
            lp.nnb[sid] = nl;
            lp.pbuild[sid] = pb;
        }
    }
}

}  // namespace bd
