// The short range's work plan: the units that its warps take.  Written by
// whichever kernel knows the cell offsets first (the cell order's, or a plan
// kernel of its own).
#pragma once

#include "common.cuh"

namespace cuco {

// A unit is kUnitMin to kUnitMax targets; the units of a segment of more than
// kDense targets are one group each (their boxes hardly grow with the group,
// as a dense cell's slices are thin) and listed ahead of the others.
constexpr int kUnitMin = 8, kUnitMax = 32;
constexpr uint32_t kDense = 128;

// The work plan of one launch, by the warps of a grid over all segments: the
// units of one segment (nt targets from sorted index tb on, first cell at
// (ix, iy, iz) of box `box`), appended in any order (which warp computes
// a target does not change its result): the slices of a dense segment from the
// front of the list, the others' from its back.  A unit's record holds
// everything its warp needs to start (box < 2^24, cells < 2^16 per axis: a
// grid's 32-bit cell numbers end at 1625 an axis), so that no unit repeats the
// divisions.  slice: the targets of a unit of this segment's box, which may
// differ between the lanes.  Every lane of the warp calls it together (nt = 0:
// nothing).
__device__ __forceinline__ void plan_segment(uint32_t tb, uint32_t nt, uint32_t box, uint32_t ix, uint32_t iy,
                                             uint32_t iz, uint32_t slice, const SRWork &w) {
    constexpr unsigned kAll = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t xy = ix | iy << 16;
    const bool dense = nt > kDense;
    // this lane's first place among the places of the warp's lanes
    auto place = [&](uint32_t c, uint32_t *counter) {
        uint32_t incl = c;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const uint32_t v = __shfl_up_sync(kAll, incl, off);
            if (lane >= (uint32_t)off) incl += v;
        }
        uint32_t first = 0;
        if (lane == 31 && incl) first = atomicAdd(counter, incl);
        return __shfl_sync(kAll, first, 31) + incl - c;
    };
    const uint32_t c = dense ? 0u : (nt + slice - 1) / slice;
    const uint32_t o = place(c, &w.ctl[2]);
    for (uint32_t k = 0; k < c; ++k)
        w.units[CUCO_IDX(w.cap - 1u - (o + k), w.cap)] =
            make_uint4(tb + k * slice, min(slice, nt - k * slice) | box << 8, xy, iz);
    uint32_t any = __ballot_sync(kAll, dense);
    if (!any) return;
    const uint32_t cd = dense ? (nt + slice - 1) / slice : 0u;
    const uint32_t od = place(cd, &w.ctl[0]);
    // the warp writes one dense segment's slices after the other
    for (; any; any &= any - 1) {
        const int src = __ffs(any) - 1;
        const uint32_t cs = __shfl_sync(kAll, cd, src), os = __shfl_sync(kAll, od, src), ts = __shfl_sync(kAll, tb, src),
                       ns = __shfl_sync(kAll, nt, src), ls = __shfl_sync(kAll, slice, src),
                       xys = __shfl_sync(kAll, xy, src), zs = __shfl_sync(kAll, iz, src), bs = __shfl_sync(kAll, box, src);
        for (uint32_t k = lane; k < cs; k += 32)
            w.units[CUCO_IDX(os + k, w.cap)] = make_uint4(ts + k * ls, min(ls, ns - k * ls) | bs << 8, xys, zs);
    }
}

// Segment `seg` of a box of G^3 cells (segments are numbered in cell order).
// hold (or null): where it is not 0, nothing is planned.
__device__ __forceinline__ void plan_box_segment(const SRPlan &plan, uint32_t seg, const uint32_t *__restrict__ cell_off,
                                                 uint32_t cell_base, uint32_t box, const SRWork &w,
                                                 const uint32_t *__restrict__ hold = nullptr) {
    uint32_t tb = 0, nt = 0, ix = 0, iy = 0, iz = 0;
    if (seg < plan.nseg) {
        const uint32_t c0 = cell_base + seg * (uint32_t)plan.S;
        tb = cell_off[c0];
        nt = cell_off[c0 + plan.S] - tb;
        if (hold && *hold) nt = 0;
        const uint32_t segs = plan.G / plan.S, row = seg / segs;
        iz = (seg - row * segs) * plan.S;
        ix = row / plan.G;
        iy = row - ix * plan.G;
    }
    plan_segment(tb, nt, box, ix, iy, iz, plan.slice, w);
}

}  // namespace cuco
