// vt_lane.cuh — per-lane ray state machine of the persistent tracers (sm_103a).
//
// A persistent warp keeps one ray per lane.  Each pass of its loop advances every live lane by
// one unit of traversal — one occupied brick walked voxel by voxel, or one empty region crossed
// per axis (skip_cross) — so lanes whose rays end can be refilled with new rays between
// units instead of idling until the longest ray of the warp is done.  The units are the loop
// body of dda_skip(), split so that the loop state lives in LaneRay; results are identical.
#pragma once

#include "vt_device.cuh"

namespace vt {

enum : int { kRayRunning = 0, kRayHit = 1, kRayMiss = 2 };

struct LaneRay {
    float o[3], d[3];
    SkipRay S;
    uint32_t slot;
    int32_t entry_axis;  // slab entry face axis, -1 when the origin is inside the grid
    float t_entry;
    bool mx, my, mz;     // axes stepped on the final iteration
    uint32_t flags;      // VT_HIT_FLAG_INVALID for rejected input
};

// Validity, slab entry and DDA set-up (trace.frag:68-71).  Returns kRayRunning, or the final
// status when the ray is already decided (rejected input, grid missed, or a degenerate direction
// resolved by the literal loop).
__device__ __forceinline__ int ray_begin(const GridView& g, const float o[3], const float d[3],
                                         LaneRay& R) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        R.o[a] = o[a];
        R.d[a] = d[a];
    }
    R.flags = 0;
    R.mx = R.my = R.mz = false;
    R.slot = kEmptyBit;
    if (!finite3(o) || !finite3(d)) {
        R.flags = VT_HIT_FLAG_INVALID;
        return kRayMiss;
    }
    float pos[3];
    int axis;
    const int kind = slab_entry(g, o, d, pos, R.t_entry, axis);
    if (kind == 0) return kRayMiss;
    R.entry_axis = kind == 1 ? axis : -1;
    const float len = __fsqrt_rn(
        __fadd_rn(__fadd_rn(__fmul_rn(d[0], d[0]), __fmul_rn(d[1], d[1])), __fmul_rn(d[2], d[2])));
    SkipRay& S = R.S;
    dda_setup_axis(pos[0], d[0], g.nx, len, S.vx, S.stx, S.dlx, S.sx);
    dda_setup_axis(pos[1], d[1], g.ny, len, S.vy, S.sty, S.dly, S.sy);
    dda_setup_axis(pos[2], d[2], g.nz, len, S.vz, S.stz, S.dlz, S.sz);
    if (skip_degenerate(S.sx, S.sy, S.sz)) {
        DDAResult r;
        dda_degenerate(g, S, r);
        S.vx = r.vx;
        S.vy = r.vy;
        S.vz = r.vz;
        R.slot = r.slot;
        R.mx = (r.last & 1) != 0;
        R.my = (r.last & 2) != 0;
        R.mz = (r.last & 4) != 0;
        return r.hit ? kRayHit : kRayMiss;
    }
    skip_setup(d, len, S);
    return grid_inside(g, S.vx, S.vy, S.vz) ? kRayRunning : kRayMiss;
}

// Directory entry of the lane's current brick.
__device__ __forceinline__ uint32_t ray_entry(const GridView& g, const LaneRay& R) {
    return __ldg(g.dir + skip_brick(g, R.S));
}

// One unit of traversal: the rest of the current occupied brick voxel by voxel, or the crossing
// of the empty region around the current brick (`e`: its directory entry, ray_entry()).  Same
// arithmetic as dda_skip().
__device__ __forceinline__ int ray_unit(const GridView& g, LaneRay& R, uint32_t e) {
    if (!brick_empty(e)) {
        if (skip_walk(g, R.S, e, R.mx, R.my, R.mz)) {
            R.slot = e;
            return kRayHit;
        }
    } else {
        skip_cross(g, R.S, R.d, e, skip_brick(g, R.S), R.mx, R.my, R.mz);
    }
    return grid_inside(g, R.S.vx, R.S.vy, R.S.vz) ? kRayRunning : kRayMiss;
}

__device__ __forceinline__ int ray_unit(const GridView& g, LaneRay& R) {
    return ray_unit(g, R, ray_entry(g, R));
}

// Record of a finished ray (unshaded colour; misses carry `miss_rgba`).
__device__ __forceinline__ HitRec ray_record(const GridView& g, const LaneRay& R, int status,
                                             uint32_t miss_rgba) {
    if (status != kRayHit) return miss_rec(R.flags, miss_rgba);
    const int32_t last = (R.mx ? 1 : 0) | (R.my ? 2 : 0) | (R.mz ? 4 : 0);
    return hit_record(g, R.o, R.d, R.S.vx, R.S.vy, R.S.vz, last, R.slot, R.entry_axis, R.t_entry);
}

// Warp-aggregated work fetch: every idle lane of the warp gets the next item index from
// `counter` (one atomic per warp).  Returns the number of items handed out to the warp; an idle
// lane's item is `first + rank`, valid when below `total`.
__device__ __forceinline__ uint64_t warp_fetch(unsigned long long* counter, uint32_t idle,
                                               uint32_t lane, uint64_t& my_item) {
    const uint32_t n = __popc(idle);
    const int leader = __ffs(idle) - 1;
    unsigned long long base = 0;
    if ((int)lane == leader) base = atomicAdd(counter, (unsigned long long)n);
    base = __shfl_sync(0xFFFFFFFFu, base, leader);
    my_item = base + __popc(idle & ((1u << lane) - 1u));
    return base;
}

// Passes a unit kind may be passed over in trace_persistent.
constexpr int kUnitWait = 4;

// Resident-warp tracing of `n` rays: a ray per lane, lanes whose rays ended refilled from `counter`
// once `refill_min` of the warp's lanes are idle.  `io.load(item, o, d)` gives an item's ray and
// `io.store(item, R, status)` takes its result; every lane of the warp calls this together.  Only the
// first `lanes` lanes take rays (lanes_per_warp()).
template <class Io>
__device__ __forceinline__ void trace_persistent(const GridView& g, const Io& io, uint64_t n,
                                                 unsigned long long* __restrict__ counter,
                                                 uint32_t refill_min, uint32_t lanes) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t all = lanes >= 32u ? 0xFFFFFFFFu : (1u << lanes) - 1u;
    const int refill = (int)min(refill_min, lanes);
    LaneRay R;
    bool busy = false;
    typename Io::Index idx = 0;
    bool more = true;
    int wait_w = 0, wait_c = 0;  // warp-uniform: iterations a unit kind was passed over
    for (;;) {
        uint32_t idle = __ballot_sync(0xFFFFFFFFu, !busy) & all;
        while (more && __popc(idle) >= refill) {
            uint64_t item;
            const uint64_t base = warp_fetch(counter, idle, lane, item);
            if (base + __popc(idle) >= n) more = false;
            if (!busy && lane < lanes && item < n) {
                float o[3], d[3];
                io.load((typename Io::Index)item, o, d);
                const int st = ray_begin(g, o, d, R);
                if (st == kRayRunning) {
                    busy = true;
                    idx = (typename Io::Index)item;
                } else {
                    io.store((typename Io::Index)item, R, st);
                }
            }
            idle = __ballot_sync(0xFFFFFFFFu, !busy) & all;
        }
        if (!more && idle == all) break;
        // One kind of unit per pass: the lanes whose next unit is the more common kind (walk or
        // crossing) run it, the others wait, unless their kind has already waited kUnitWait
        // passes.  A warp then issues one kind's instructions per pass instead of both; every
        // pass with busy lanes runs at least one unit.  2% faster on the 16M incoherent rays.
        const uint32_t e = busy ? ray_entry(g, R) : kEmptyBit;
        const bool walk = busy && !brick_empty(e);
        const uint32_t wb = __ballot_sync(0xFFFFFFFFu, walk);
        const uint32_t cb = __ballot_sync(0xFFFFFFFFu, busy && !walk);
        bool run_walk = __popc(wb) >= __popc(cb);
        if (run_walk ? (cb && wait_c >= kUnitWait) : (wb && wait_w >= kUnitWait)) run_walk = !run_walk;
        if (run_walk) {
            wait_w = 0;
            wait_c = cb ? wait_c + 1 : 0;
        } else {
            wait_c = 0;
            wait_w = wb ? wait_w + 1 : 0;
        }
        if (busy && walk == run_walk) {
            const int st = ray_unit(g, R, e);
            if (st != kRayRunning) {
                io.store(idx, R, st);
                busy = false;
            }
        }
    }
}

}  // namespace vt
