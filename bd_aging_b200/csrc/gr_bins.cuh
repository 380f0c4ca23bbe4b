// gr_bins.cuh -- g(r) bins of squared distances, shared by the mirror's and
// the engine's pair kernels.
//
// The reference bins a pair at (int)(sqrt(d2) / bin_size), both operations
// correctly rounded, when the square root is below the range; a bin equal to
// nbins goes to the last one (get_gder.cu:116-121).  Per pair the kernels only
// estimate q = sqrt(d2) / bin_size with an approximate rsqrt of a fused d2, and round
// q - 1/2 to the nearest integer: floor(q) unless q lies within
// eps = c1 q + c0 of an integer.  Such a pair (about one in a thousand; the
// range itself is the integer nbins) is settled with the reference's
// operations.  Relative errors of q: 2^-22.9 of the rsqrt, 2^-24 of each of the
// other roundings (three of d2, halved; three of q) and as much again for the
// reference's own roundings, 8e-7 in all at most; c1 = 1e-6.  c0 covers an
// absolute error of the distance (positions shifted to a periodic image are
// rounded).
#pragma once
#include <cmath>
#include <cstring>

#include "common.cuh"

namespace bd {

constexpr float kGrC1 = 1e-6f;

struct GrBins {
    float thr;       // smallest squared distance at or beyond the range
    float near;      // estimates of d2 at or beyond it are out of range
    float inv_bin;   // 1 / bin_size (estimate only)
    float bin_size;  // range / nbins, float division as in the reference
    float c0;
    int nbins;
};

inline GrBins gr_bins(float range, int nbins, double dist_err) {
    // smallest float >= 0 whose square root is not below `range`, by
    // bisection over the bit patterns of the non-negative floats
    unsigned lo = 0u, hi = 0x7f800000u;  // +0 .. +inf
    float x;
    while (lo < hi) {
        const unsigned mid = lo + ((hi - lo) >> 1);
        std::memcpy(&x, &mid, 4);
        if (!(std::sqrt(x) < range)) hi = mid;
        else lo = mid + 1;
    }
    std::memcpy(&x, &lo, 4);
    GrBins g;
    g.thr = x;
    g.nbins = nbins;
    g.bin_size = range / (float)nbins;
    g.inv_bin = 1.0f / g.bin_size;
    g.near = (float)((double)x * (1.0 + 1.2e-6 + 2.0 * dist_err / (double)range));
    g.c0 = (float)(1.1 * dist_err / (double)g.bin_size + 1e-6);
    return g;
}

// bin of an exactly rounded squared distance below the range
__device__ __forceinline__ int gr_bin_settled(float d2, const GrBins &g) {
    const int bin = (int)__fdiv_rn(__fsqrt_rn(d2), g.bin_size);
    return bin == g.nbins ? bin - 1 : bin;
}
// A histogram row holds nbins counts and a spare word for each lane, where
// pairs out of range add instead of branching.  gr_top: the largest slot word
// of the lane; gr_row: what to add to 4 x a slot word for its shared address.
constexpr int kGrSpare = 32;
__device__ __forceinline__ unsigned gr_top(int nbins, int lane) {
    return (unsigned)__float_as_int(kRintMagic) + (unsigned)(nbins + lane);
}
__device__ __forceinline__ unsigned gr_row(const unsigned *row) {
    return (unsigned)__cvta_generic_to_shared(row) - 4u * (unsigned)__float_as_int(kRintMagic);
}
// Estimates of two squared distances: slot words (bits of bin + kRintMagic,
// at most `top`; NaN too) and whether the bin is still open (also for d2 = 0).
__device__ __forceinline__ void gr_estimate(f2 D2, const GrBins &g, unsigned top, unsigned (&slot)[2], bool (&open)[2]) {
    float a, b;
    f2_split(D2, a, b);
    asm("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(a));  // a subnormal d2 gives a NaN estimate: open
    asm("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(b));
    const f2 Q = f2_fma(f2_mul(D2, f2_make(a, b)), f2_bcast(g.inv_bin), f2_bcast(-0.5f));
    const f2 QM = f2_add(Q, f2_bcast(kRintMagic)), R = f2_sub(Q, f2_sub(QM, f2_bcast(kRintMagic)));
    const f2 H = f2_fma(Q, f2_bcast(-kGrC1), f2_bcast(0.5f - kGrC1 - g.c0));
    float qa, qb, ra, rb, ha, hb;
    f2_split(QM, qa, qb);
    f2_split(R, ra, rb);
    f2_split(H, ha, hb);
    slot[0] = min(__float_as_uint(qa), top);
    slot[1] = min(__float_as_uint(qb), top);
    open[0] = !(fabsf(ra) <= ha);
    open[1] = !(fabsf(rb) <= hb);
}
// one count at a shared-memory byte address
__device__ __forceinline__ void gr_count(unsigned addr, unsigned weight) {
    asm volatile("red.shared.add.u32 [%0], %1;" ::"r"(addr), "r"(weight));
}
// takes an estimated count back (one in a spare word may stay)
__device__ __forceinline__ void gr_uncount(unsigned row, unsigned slot, unsigned weight, int nbins) {
    if (slot - (unsigned)__float_as_int(kRintMagic) < (unsigned)nbins) gr_count(row + 4u * slot, 0u - weight);
}

}  // namespace bd
