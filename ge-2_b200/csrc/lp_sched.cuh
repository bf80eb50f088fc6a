// How the scores kernels of the link-prediction step share out their work: the (row block, negative tile) units of the whole step are
// numbered consecutively and dealt to persistent CTAs as contiguous ranges of equal length.
#pragma once
#include "lp_internal.cuh"

namespace ge2 {

constexpr int kMaxParts = 8;  // most CTAs that can share one row block in the logsumexp pass; size of a row's partial list

// How the units of a launch are dealt to its CTAs: CTA k takes units [k * units / grid, (k + 1) * units / grid).
struct Sched {
    int RB, T, ZC;       // row blocks per chunk, negative tiles per chunk, sides * chunks
    int unitsA, gridA;   // lse pass: unit = (zc, row block, tile), numbered (zc * RB + rb) * T + tile
    int unitsB, gridB;   // gradient pass: the same units (X = Q block, stream over the K tiles)
};
__host__ __device__ __forceinline__ int range_begin(int k, int units, int grid) { return (int)(((long long)k * units) / grid); }
__host__ __device__ __forceinline__ int cta_of_unit(int u, int units, int grid) { return (int)((((long long)u + 1) * grid - 1) / units); }

// what a CTA needs to know about one unit of the lse pass
struct UnitA {
    int item, tile, rb, zc;
};
__device__ __forceinline__ UnitA decode_a(int u, const Sched& sc) {
    UnitA r;
    r.item = u / sc.T;
    r.tile = u - r.item * sc.T;
    r.zc = r.item / sc.RB;
    r.rb = r.item - r.zc * sc.RB;
    return r;
}
// The loops walk their units with these instead of decoding every index (no divisions inside the pipelines).
struct IterA {
    int item, tile, rb, zc;
    __device__ __forceinline__ IterA(int u, const Sched& sc) {
        const UnitA un = decode_a(u, sc);
        item = un.item, tile = un.tile, rb = un.rb, zc = un.zc;
    }
    __device__ __forceinline__ void next(const Sched& sc) {
        if (++tile == sc.T) {
            tile = 0;
            item++;
            if (++rb == sc.RB) rb = 0, zc++;
        }
    }
};

}  // namespace ge2
