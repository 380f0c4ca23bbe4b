// nlist_cluster.cuh -- list steps of small replicas, resident in a
// thread-block cluster.
//
// A small replica's time step is latency: a thousand particles are one
// instruction stream's worth of work per SM, and the per-step path pays four
// launches (8.4 us) for it, the per-replica block of variants 3-5 a chain of
// global loads and a whole replica on one SM (6.1 us at N = 1000).  Here a
// cluster of C CTAs runs a whole batch of steps of one replica:
//  - a thread owns one particle, whose state (position, remainder, build
//    position, crossings) stays in registers for the launch;
//  - every CTA holds all positions of the replica in shared memory, double
//    buffered, and its own particles' lists as 16-bit local indices, so a
//    step reads nothing from global memory but its noise amplitude;
//  - a thread stores its new position into the next buffer of all C CTAs
//    (distributed shared memory); one cluster barrier per step publishes them;
//  - as many threads again draw the next step's Gaussians meanwhile (1500
//    cycles in one stream, as long as the rest of a step);
//  - a particle beyond half the skin raises a word in every CTA; after the
//    barrier each CTA sorts the replica by cell (into the free buffer) and
//    rebuilds its own particles' lists, with one more cluster barrier before
//    that buffer is written again.
// Lists, force sums, updates and rebuild decisions are those of the other
// launches (replica_partners_rows, list_force, advance_wrap, list_beyond), so the
// bits are the same.  Lists and state go back to global memory at the end of
// the launch.
// Measured, one replica at T = 0.1: 1.57, 1.86 and 2.78 us a step at N = 500,
// 1000 and 2000 (8.4 with the per-step launches).  At N = 1000 the force takes
// about 1100 cycles (two groups of eight partners), the update 270, the stores
// to the peers 300, the barrier 400; a rebuild takes 20000.  Tried: four
// partners at a time with a branch per pair (3200 cycles of force), the noise
// in the owner's own stream (1500 cycles on the critical path).
#pragma once

namespace bd {

constexpr int kClusterMaxOwners = 256;  // particles per CTA (512 threads of 128 registers)
constexpr int kClusterMaxCtas = 8;       // portable cluster size
constexpr int kClusterMarks = 32;        // rebuilding steps noted before they go to global memory

// dynamic shared memory: two position buffers (with the zero position), lists
// [kMaxNbr / 4][owners][4], noise [2][3][owners], cell starts and counters of
// a rebuild
__host__ __device__ inline size_t cluster_smem_bytes(int nmax, int cells, int owners) {
    return 2 * (size_t)(nmax + 1) * 16 + (size_t)(kMaxNbr * 2 + 24) * owners +
           (((size_t)(2 * cells + 1) * 4 + 15) & ~(size_t)15);
}

struct ListShared {  // lists and positions in shared memory; entries are local particle indices
    const float4 *pos;
    const ushort4 *list;  // chunk k / 4 of this thread at [(k / 4) * stride]
    int stride, none;
    __device__ __forceinline__ void words(int k0, int (&jn)[kGather]) const {
        const ushort4 w = list[(k0 >> 2) * stride];
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

// list_forces_wca for one warp per scheduler: eight partners at a time
// without a branch, so that their chains overlap (partners out of range and
// padding get a zero factor, which leaves the sums as they are), always with
// the minimum image (it returns the plain difference where that is nearest).
// The list is padded to a multiple of eight.
constexpr int kClusterGroup = 8;
template <class SRC>
__device__ __forceinline__ void list_forces_wide(const SRC &src, int n, float4 pi, float L, float Linv, float sq0,
                                                 float sq1, float c0, float c1, float &fx, float &fy, float &fz) {
    const f2 PX = f2_bcast(pi.x), PY = f2_bcast(pi.y), PZ = f2_bcast(pi.z), M12 = f2_bcast(-12.0f);
    const f2 LINV = f2_bcast(Linv), NEGL = f2_bcast(-L);
    f2 FX = 0ull, FY = 0ull, FZ = 0ull;  // (0.f, 0.f)
    for (int k0 = 0; k0 < n; k0 += kClusterGroup) {
        int jn[kClusterGroup];
        float4 q[kClusterGroup];
#pragma unroll
        for (int u = 0; u < kClusterGroup; u += kGather) {
            int w[kGather];
            src.words(k0 + u, w);
#pragma unroll
            for (int v = 0; v < kGather; v++) jn[u + v] = w[v];
        }
#pragma unroll
        for (int u = 0; u < kClusterGroup; u++) q[u] = src.pos[jn[u]];
        f2 dX[kClusterGroup / 2], dY[kClusterGroup / 2], dZ[kClusterGroup / 2], GM[kClusterGroup / 2];
#pragma unroll
        for (int p = 0; p < kClusterGroup / 2; p++) {
            const float4 qa = q[2 * p], qb = q[2 * p + 1];
            dX[p] = min_image_pair(f2_sub(f2_make(qa.x, qb.x), PX), LINV, NEGL);
            dY[p] = min_image_pair(f2_sub(f2_make(qa.y, qb.y), PY), LINV, NEGL);
            dZ[p] = min_image_pair(f2_sub(f2_make(qa.z, qb.z), PZ), LINV, NEGL);
            const f2 D2 = f2_fma(dZ[p], dZ[p], f2_fma(dX[p], dX[p], f2_mul(dY[p], dY[p])));
            float d2a, d2b, ra, rb;
            f2_split(D2, d2a, d2b);
            const bool ta = (__float_as_uint(qa.w) >> 31) != 0u, tb = (__float_as_uint(qb.w) >> 31) != 0u;
            const bool oka = (jn[2 * p] != src.none) & (d2a < (ta ? c1 : c0));
            const bool okb = (jn[2 * p + 1] != src.none) & (d2b < (tb ? c1 : c0));
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ra) : "f"(d2a));
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rb) : "f"(d2b));
            const f2 R2 = f2_make(ra, rb);
            const f2 S2 = f2_mul(R2, f2_make(ta ? sq1 : sq0, tb ? sq1 : sq0));
            const f2 S6 = f2_mul(f2_mul(S2, S2), S2);
            const f2 G = f2_mul(f2_mul(M12, f2_sub(f2_mul(S6, S6), S6)), R2);
            float ga, gb;
            f2_split(G, ga, gb);
            GM[p] = f2_make(oka ? ga : 0.f, okb ? gb : 0.f);
        }
#pragma unroll
        for (int p = 0; p < kClusterGroup / 2; p++) {
            FX = f2_fma(GM[p], dX[p], FX);
            FY = f2_fma(GM[p], dY[p], FY);
            FZ = f2_fma(GM[p], dZ[p], FZ);
        }
    }
    float ea, eb;
    f2_split(FX, ea, eb);
    fx = __fadd_rn(ea, eb);
    f2_split(FY, ea, eb);
    fy = __fadd_rn(ea, eb);
    f2_split(FZ, ea, eb);
    fz = __fadd_rn(ea, eb);
}

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_map(unsigned addr, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// nsteps steps (at most the amplitude table's batch) of replica
// order[blockIdx.x / C] by the C CTAs of a cluster, Philox noise.  The first
// half of the block's threads own a particle each (at least ceil(n / C)); the
// others draw the noise of the step after theirs.
template <bool EXTRA>
__global__ void __launch_bounds__(2 * kClusterMaxOwners, 1)
    k_list_cluster(ListArgs a, ListPersist lp, const long long *ni_base, int nsteps, int nmax, int cmax, int C) {
    extern __shared__ __align__(16) unsigned char dsm[];
    __shared__ int s_marks[kClusterMarks];
    __shared__ unsigned s_need[3];  // step s: some particle is beyond half the skin, word s % 3
    const int T = blockDim.x >> 1, tid = threadIdx.x < T ? threadIdx.x : threadIdx.x - T;
    const bool owner = threadIdx.x < T;
    const int rep = lp.order[blockIdx.x / C];
    const unsigned q = cluster_rank();
    // parameters in shared memory: the barrier's acquire empties L1, and a
    // step would wait for them from L2 again
    __shared__ SysDev S;
    for (int k = threadIdx.x; k < (int)(sizeof(SysDev) / 4); k += blockDim.x)
        reinterpret_cast<int *>(&S)[k] = reinterpret_cast<const int *>(a.sys + rep)[k];
    __syncthreads();
    const int n = S.n, base = S.part_base;
    float4 *s_pos0 = reinterpret_cast<float4 *>(dsm);  // [2][nmax + 1]
    ushort4 *s_list = reinterpret_cast<ushort4 *>(s_pos0 + 2 * (nmax + 1));  // [kMaxNbr / 4][T]
    float *s_noise = reinterpret_cast<float *>(s_list + (size_t)(kMaxNbr / 4) * T);  // [2][3][T]
    int *s_start = reinterpret_cast<int *>(s_noise + 6 * T), *s_fill = s_start + cmax + 1;
    const int first = (int)((long long)n * q / C), count = (int)((long long)n * (q + 1) / C) - first;
    const bool live = tid < count;
    const int lid = first + (live ? tid : 0), sid = base + lid;
    unsigned short *my_list = reinterpret_cast<unsigned short *>(s_list + tid);
    auto list_at = [&](int k) { return ((size_t)(k >> 2) * T) * 4 + (k & 3); };

    // positions of the launch's first step, own state, lists
    const float4 *pos_in = (lp.cur0 & 1) ? lp.pos[1] : lp.pos[0];
    for (int i = threadIdx.x; i < n; i += blockDim.x) s_pos0[i] = pos_in[base + i];
    if (threadIdx.x < 2) s_pos0[threadIdx.x * (nmax + 1) + n] = make_float4(0.f, 0.f, 0.f, 0.f);  // the zero position
    if (threadIdx.x < 3) s_need[threadIdx.x] = 0u;
    bool need = a.flag[rep] != 0;
    const int gid = a.gid_of[sid], pid = gid - base;
    float4 pi = pos_in[sid];
    const int tm = (int)(__float_as_uint(pi.w) >> 31);
    const long long ni0 = *ni_base;
    auto draw_noise = [&](int s) {  // amplitude times the Gaussians of step s
        if (!live || s >= nsteps) return;
        const float3 xi = gauss3(S.seed, (uint32_t)pid, (uint64_t)(ni0 + s), a.rng_stream);
        const float amp = __ldg(a.amp_tab + ((size_t)s * a.nrep + rep) * 2 + tm);
        float *z = s_noise + (s & 1) * 3 * T + tid;
        z[0] = __fmul_rn(amp, xi.x);
        z[T] = __fmul_rn(amp, xi.y);
        z[2 * T] = __fmul_rn(amp, xi.z);
    };
    bool rebuilt = false;
    float4 pb = a.pbuild[sid];
    float lx = a.lo_x[sid], ly = a.lo_y[sid], lz = a.lo_z[sid];
    int ix = a.img[sid], iy = a.img[a.np + sid], iz = a.img[2 * a.np + sid];
    int nl = min(a.nnb[sid], kMaxNbr);
    auto pad_list = [&]() {
        for (int k = nl; k % kClusterGroup != 0; k++) my_list[list_at(k)] = (unsigned short)n;
    };
    if (!owner) draw_noise(0);
    if (owner && live && !need) {
        for (int k = 0; k < nl; k += kGather) {
            const int4 w = reinterpret_cast<const int4 *>(a.nbr)[(size_t)(k >> 2) * a.np + sid];
            auto local = [&](int j) { return (unsigned short)min((unsigned)(j - base), (unsigned)n); };
            s_list[(size_t)(k >> 2) * T + tid] = make_ushort4(local(w.x), local(w.y), local(w.z), local(w.w));
        }
        pad_list();
    }
    const float L = S.L, Linv = S.Linv, mob = S.mob[tm], dt = S.dt;
    const float sg0 = tm ? S.sig[1] : S.sig[0], sg1 = tm ? S.sig[2] : S.sig[1];
    const float c0 = tm ? S.cut2[1] : S.cut2[0], c1 = tm ? S.cut2[2] : S.cut2[1];
    const bool general = (EXTRA && S.pot != kPotWcaModified) || S.fcap > 0.f;
    const float skin_half2 = S.skin_half2;
    // steps that rebuilt, noted in shared memory: a global store before a
    // cluster barrier would hold its arrive back
    int builds = 0;
    auto flush_marks = [&]() {
        if (q != 0 || threadIdx.x != 0) return;
        const int m = builds % kClusterMarks == 0 && builds ? kClusterMarks : builds % kClusterMarks;
        atomicAdd((unsigned long long *)lp.builds, (unsigned long long)m);
        for (int k = 0; k < m; k++) lp.step_rebuilt[s_marks[k]] = 1;
    };
    // every CTA's buffers exist and are loaded before a peer writes to them
    cluster_arrive();
    cluster_wait();
    for (int s = 0; s < nsteps; s++) {
        float4 *cur = s_pos0 + (s & 1) * (nmax + 1), *nxt = s_pos0 + ((s & 1) ^ 1) * (nmax + 1);
        if (need) {  // the same in every CTA of the cluster
            replica_sort(S, [&](int i) { return cur[i]; }, lp.cap, a.status, s_start, s_fill, nxt);
            // an owner scans the first five rows of its cells, its helper the
            // others, into the list's end in reverse
            const CellsShared cells{s_start, nxt};
            int *helped = reinterpret_cast<int *>(s_noise + ((s + 1) & 1) * 3 * T);  // free until this step's draw
            const float4 v = owner ? pi : cur[lid];
            int found = 0;
            if (live)
                found = replica_partners_rows(S, v, cells, owner ? 0 : 5, owner ? 5 : 9, [&](int k, int sj) {
                    if (k < kMaxNbr / 2) my_list[list_at(owner ? k : kMaxNbr - 1 - k)] = (unsigned short)(sj - base);
                });
            if (!owner) helped[tid] = found;
            __syncthreads();
            if (owner && live) {
                const int more = helped[tid];
                if (found <= kMaxNbr / 2 && more <= kMaxNbr / 2 && found + 2 * more <= kMaxNbr) {
                    for (int k = 0; k < more; k++) my_list[list_at(found + k)] = my_list[list_at(kMaxNbr - 1 - k)];
                    found += more;
                } else {  // a long list: both halves into its front
                    found = replica_partners_rows(S, v, cells, 0, 9, [&](int k, int sj) {
                        if (k < kMaxNbr) my_list[list_at(k)] = (unsigned short)(sj - base);
                        else set_status(a.status, kStatCellOverflow);
                    });
                }
                nl = min(found, kMaxNbr);
                pad_list();
                pb = pi;
            }
            rebuilt = true;
            if (threadIdx.x == 0) s_marks[builds % kClusterMarks] = s;
            if (++builds % kClusterMarks == 0) flush_marks();
            __syncwarp();
            cluster_arrive();  // `nxt` is free in every CTA after the wait
            cluster_wait();
        }
        if (threadIdx.x == 0) s_need[(s + 1) % 3] = 0u;  // last read two barriers ago, next raised after this step's barrier
        if (!owner) {
            draw_noise(s + 1);
        } else if (live) {
            const float *z = s_noise + (s & 1) * 3 * T + tid;
            const float nx = z[0], ny = z[T], nz = z[2 * T];
            float fx, fy, fz;
            const ListShared src{cur, s_list + tid, T, n};
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
            const unsigned at = (unsigned)__cvta_generic_to_shared(nxt + lid);
#pragma unroll
            for (int c = 0; c < kClusterMaxCtas; c++)
                if (c < C)
                    asm volatile("st.shared::cluster.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_map(at, c)),
                                 "f"(pi.x), "f"(pi.y), "f"(pi.z), "f"(pi.w)
                                 : "memory");
            if (!(isfinite(pi.x) && isfinite(pi.y) && isfinite(pi.z))) set_status(a.status, kStatNumeric);
            if (list_beyond(pi.x, pi.y, pi.z, pb, L, Linv, skin_half2)) {
                const unsigned word = (unsigned)__cvta_generic_to_shared(s_need + s % 3);
                for (int c = 0; c < C; c++)
                    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_map(word, c)), "r"(1u) : "memory");
            }
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        need = s_need[s % 3] != 0u;
    }
    if (owner && live) {
        float4 *pos_out = ((lp.cur0 + nsteps) & 1) ? lp.pos[1] : lp.pos[0];
        pos_out[sid] = pi;
        a.lo_x[sid] = lx;
        a.lo_y[sid] = ly;
        a.lo_z[sid] = lz;
        a.img[sid] = ix;
        a.img[a.np + sid] = iy;
        a.img[2 * a.np + sid] = iz;
        if (rebuilt) {
            auto global = [&](int j) { return j == n ? a.np : base + j; };
            for (int k = 0; k < nl; k += kGather) {
                const ushort4 w = s_list[(size_t)(k >> 2) * T + tid];
                reinterpret_cast<int4 *>(lp.nbr)[(size_t)(k >> 2) * a.np + sid] =
                    make_int4(global(w.x), global(w.y), global(w.z), global(w.w));
            }
            lp.nnb[sid] = nl;
            lp.pbuild[sid] = pb;
        }
    }
    if (builds % kClusterMarks != 0) flush_marks();
    if (q == 0 && threadIdx.x == 0) a.flag[rep] = need ? 1 : 0;
}

}  // namespace bd
