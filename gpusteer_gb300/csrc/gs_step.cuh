// Device pieces shared by the fused step's kernels: the thread-per-agent ones
// (gs_step.cu) and the lane-group ones (gs_lanes.cu).
#pragma once

#include "gs_behaviours.cuh"
#include "gs_launch.h"
#include "gs_scan.cuh"

namespace gs {

__device__ __forceinline__ unsigned u(float x) { return __float_as_uint(x); }
__device__ __forceinline__ float fb(unsigned x) { return __uint_as_float(x); }

// Adds 1 to the scan tile total of `cell`, once per group of active lanes in
// the same tile (a warp's agents are mostly in one).
__device__ __forceinline__ void add_to_tile(unsigned* tile, unsigned cell) {
    const unsigned t = cell / kScanTile;
    const unsigned peers = __match_any_sync(__activemask(), t);
    if ((threadIdx.x & 31u) == unsigned(__ffs(int(peers)) - 1))
        atomicAdd(tile + t, unsigned(__popc(int(peers))));
}

// The agent's cell for the next step's counting sort: counted (the old count
// is its rank in the cell) and, given tile totals (tile not null), added to
// its tile's total.
__device__ __forceinline__ unsigned count_next(const Scene& sc, V3 pos, int wrap_mode,
                                               unsigned* count, unsigned* tile, unsigned& cell) {
    const V3 wp = wrap_world(pos, sc.grid.ws, wrap_mode);
    cell = sc.cell_offset + cell_of(sc.grid, wp);
    if (tile) add_to_tile(tile, cell);
    return atomicAdd(count + cell, 1u);
}

__device__ __forceinline__ void store_next(const FusedLaunch& L, unsigned s, const Self& me,
                                           unsigned id, unsigned scene, const Scene& sc,
                                           int wrap_mode) {
    // the cell count's atomic first: its round trip overlaps the state stores
    unsigned cell;
    const unsigned rank = count_next(sc, me.pos, wrap_mode, L.count, L.tile, cell);
    L.A.f[0][s] = make_float4(me.pos.x, me.pos.y, me.pos.z, fb(id));
    L.A.f[1][s] = make_float4(me.dir.x, me.dir.y, me.dir.z, me.speed);
    L.A.f[2][s] = make_float4(me.side.x, me.side.y, me.side.z, me.radius);
    L.A.f[3][s] = make_float4(me.up.x, me.up.y, me.up.z, me.mass);
    L.A.f[4][s] = make_float4(me.max_speed, me.max_force, fb(0u), fb(scene));
    L.cellrank[s] = make_uint2(cell, rank);
}

// The scene number alone (f4.w): the KNN needs position, index and scene;
// the rest of the state is loaded after it, so it is not held in registers
// through the scan.
__device__ __forceinline__ unsigned load_scene(const Fused& B, unsigned s) {
    return __float_as_uint(reinterpret_cast<const float*>(B.f[4] + s)[3]);
}

// Everything but position and index, after the KNN.
__device__ __forceinline__ Self load_rest(const Fused& B, unsigned s, V3 pos, float4& f4v) {
    const float4 f1 = B.f[1][s], f2 = B.f[2][s], f3 = B.f[3][s];
    f4v = B.f[4][s];
    Self me;
    me.pos = pos;
    me.dir = v3(f1);
    me.speed = f1.w;
    me.side = v3(f2);
    me.radius = f2.w;
    me.up = v3(f3);
    me.mass = f3.w;
    me.max_speed = f4v.x;
    me.max_force = f4v.y;
    return me;
}

// NEEDC: the behaviours that read the neighbour list, fixed at compile time
// (kNeedRuntime: taken from p.need).
constexpr unsigned kNeedRuntime = ~0u;
constexpr unsigned kNeedList = NEED_SEP | NEED_ALI | NEED_COH | NEED_AVOID | NEED_CLOSE;

}  // namespace gs
