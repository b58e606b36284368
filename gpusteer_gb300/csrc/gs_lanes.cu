// The fused step of small groups: a group of lanes per agent (gs_lanes.cuh).
//
// Same phases, same buffers between them and the same results as the
// thread-per-agent kernels of gs_step.cu; only the neighbour lists between the
// wall and the rest phase lie agent by agent (knn_slot[s * k + r]), which a
// lane group writes and reads in one access.
#include "gs_lanes.cuh"
#include "gs_launch.h"
#include "gs_step.cuh"

namespace gs {

constexpr unsigned kLaneBlock = 128;

// ---- whole step without walls -----------------------------------------------------------
template <int G, int R, unsigned NEEDC>
__global__ void __launch_bounds__(kLaneBlock) k_lanes_step(FusedLaunch L, StepDev p) {
    after_previous();
    __shared__ unsigned row_sh[R ? 1 : kLaneBlock / G * kLaneRowWords];
    unsigned* rows = row_sh + (R ? 0u : threadIdx.x / G * kLaneRowWords);
    __shared__ __align__(16) float sh[kLaneBlock / G * LaneSums<G>::kWords];
    const unsigned need = NEEDC == kNeedRuntime ? p.need : NEEDC;
    const unsigned lane = threadIdx.x & unsigned(G - 1);
    const unsigned a = (blockIdx.x * kLaneBlock + threadIdx.x) / G;
    const bool act = a < L.n;  // the last warps' spare groups run along and store nothing
    const unsigned s = act ? a : L.n - 1;
    const float4 f0 = L.B.f[0][s];
    const unsigned id = __float_as_uint(f0.w);
    float4 f4v;
    Self me = load_rest(L.B, s, v3(f0), f4v);
    const unsigned scene = __float_as_uint(f4v.w);
    const Scene sc = L.scenes[scene];
    unsigned ix, iy, iz;
    cell_coords(sc.grid, me.pos, ix, iy, iz);
    const Box box = cell_box(sc.grid, ix, iy, iz, p.r);
    const LaneEntry<G> nb = lanes_knn<G, R>(p.k, lane, me.pos, id, sc.grid, box, sc.cell_offset,
                                            L.start, L.B.f[0], rows);
    const bool ok = lane < p.k && nb.slot != UINT_MAX;
    const unsigned bs = ok ? nb.slot : s;
    const float4 b0 = L.B.f[0][bs], b1 = L.B.f[1][bs];
    const float br = (need & (NEED_AVOID | NEED_CLOSE))
                         ? reinterpret_cast<const float*>(L.B.f[2] + bs)[3] : 0.f;
    if (L.rec_knn && act) {
        if (lane < p.k) L.rec_knn[size_t(id) * p.k + lane] = ok ? __float_as_uint(b0.w) : UINT_MAX;
        if (lane == 0) {
            L.rec_pos[id] = make_float4(me.pos.x, me.pos.y, me.pos.z, me.speed);
            L.rec_dir[id] = make_float4(me.dir.x, me.dir.y, me.dir.z, 0.f);
        }
    }
    unsigned applied = p.clear_applied ? 0u : __float_as_uint(f4v.z);
    V3 steer = p.dirty ? v3(L.B.f[5][s]) : v3(0.f, 0.f, 0.f);
    const LaneNeighbour n{ok, v3(b0), v3(b1), b1.w, br, key_dist(nb.key)};
    lanes_behaviours<G, R == 3>(p, need, 0, me, lane, n, LaneSums<G>::of(sh), applied, steer);
    integrate<R == 3>(me, steer, p.dt);
    if (act && lane == 0) store_next(L, s, me, id, scene, sc, p.wrap_mode);
}

// ---- wall phase ---------------------------------------------------------------------------
template <int G, int R>
__global__ void __launch_bounds__(kLaneBlock) k_lanes_walls(FusedLaunch L, StepDev p) {
    after_previous();
    __shared__ unsigned row_sh[R ? 1 : kLaneBlock / G * kLaneRowWords];
    unsigned* rows = row_sh + (R ? 0u : threadIdx.x / G * kLaneRowWords);
    const unsigned lane = threadIdx.x & unsigned(G - 1);
    const unsigned a = (blockIdx.x * kLaneBlock + threadIdx.x) / G;
    const bool act = a < L.n;
    const unsigned s = act ? a : L.n - 1;
    const float4 f0 = L.B.f[0][s];
    const unsigned id = __float_as_uint(f0.w);
    float4 f4v;
    Self me = load_rest(L.B, s, v3(f0), f4v);
    const Scene sc = L.scenes[__float_as_uint(f4v.w)];
    unsigned ix, iy, iz;
    cell_coords(sc.grid, me.pos, ix, iy, iz);
    const Box box = cell_box(sc.grid, ix, iy, iz, p.r);
    const LaneEntry<G> nb = lanes_knn<G, R>(p.k, lane, me.pos, id, sc.grid, box, sc.cell_offset,
                                            L.start, L.B.f[0], rows);
    if (act && lane < p.k) {
        L.knn_slot[size_t(s) * p.k + lane] = nb.slot;
        // the KNN distance (before any wall correction moves agents), read by
        // avoid-close-neighbours only
        if (p.need & NEED_CLOSE) L.knn_dist[size_t(s) * p.k + lane] = key_dist(nb.key);
    }
    unsigned applied = p.clear_applied ? 0u : __float_as_uint(f4v.z);
    V3 steer = p.dirty ? v3(L.B.f[5][s]) : v3(0.f, 0.f, 0.f);
    lanes_walls<G, R>(WallRefs{L.w_start, L.w_end, L.w_normal, L.w_pos_id, L.w_cell_start}, sc, p, me,
                      lane, box, applied, steer, rows);
    if (act && lane == 0) {
        L.w0[s] = make_float4(me.pos.x, me.pos.y, me.pos.z, me.radius);
        L.w1[s] = make_float4(me.dir.x, me.dir.y, me.dir.z, me.speed);
        L.w2[s] = make_float4(steer.x, steer.y, steer.z, __uint_as_float(applied));
    }
}

// ---- rest of the step after the wall phase -------------------------------------------------
template <int G, unsigned NEEDC>
__global__ void __launch_bounds__(kLaneBlock) k_lanes_rest(FusedLaunch L, StepDev p) {
    after_previous();
    __shared__ __align__(16) float sh[kLaneBlock / G * LaneSums<G>::kWords];
    const unsigned need = NEEDC == kNeedRuntime ? p.need : NEEDC;
    const unsigned lane = threadIdx.x & unsigned(G - 1);
    const unsigned a = (blockIdx.x * kLaneBlock + threadIdx.x) / G;
    const bool act = a < L.n;
    const unsigned s = act ? a : L.n - 1;
    const unsigned slot = lane < p.k ? L.knn_slot[size_t(s) * p.k + lane] : UINT_MAX;
    const bool ok = slot != UINT_MAX;
    const unsigned bs = ok ? slot : s;
    const float4 b0 = L.w0[bs], b1 = L.w1[bs];
    const float kd = (need & NEED_CLOSE) && lane < p.k ? L.knn_dist[size_t(s) * p.k + lane] : 0.f;
    const float4 w0 = L.w0[s], w1 = L.w1[s], w2 = L.w2[s];
    float4 f4v;
    Self me = load_rest(L.B, s, v3(w0), f4v);
    me.radius = w0.w;
    me.dir = v3(w1);
    me.speed = w1.w;
    const unsigned id = __float_as_uint(reinterpret_cast<const float*>(L.B.f[0] + s)[3]);
    const unsigned scene = __float_as_uint(f4v.w);
    unsigned applied = __float_as_uint(w2.w);
    V3 steer = v3(w2);
    const LaneNeighbour n{ok, v3(b0), v3(b1), b1.w, b0.w, kd};
    lanes_behaviours<G, true>(p, need, 1, me, lane, n, LaneSums<G>::of(sh), applied, steer);
    integrate<true>(me, steer, p.dt);
    const Scene sc = L.scenes[scene];
    if (act && lane == 0) store_next(L, s, me, id, scene, sc, p.wrap_mode);
}

// ---- one behaviour per launch ------------------------------------------------------------------
// The per-function behaviours of small groups (whose worlds may be flat: they
// divide vectors as flat ones): lane r of an agent's group takes
// list entry r.  An index past the other group ends the list, as in the
// reference's kernels.
template <int G>
__device__ __forceinline__ bool lanes_entry(const unsigned* knn, unsigned i,
                                            unsigned n, unsigned k, unsigned n_other,
                                            unsigned lane, unsigned& b) {
    b = lane < k ? knn[i + size_t(lane) * n] : UINT_MAX;
    const unsigned bad = lanes_ballot<G>(b >= n_other);
    const bool ok = bad == 0 || lane < unsigned(__ffs(int(bad)) - 1);
    if (!ok) b = 0;
    return ok;
}

// Agent, lane and validity of the thread; spare groups run along as the last
// agent and store nothing.
template <int G>
__device__ __forceinline__ bool lanes_agent(unsigned n, unsigned& i, unsigned& lane) {
    const unsigned a = (blockIdx.x * kLaneBlock + threadIdx.x) / G;
    lane = threadIdx.x & unsigned(G - 1);
    i = a < n ? a : n - 1;
    return a < n;
}

// KIND: 0 separation, 1 alignment, 2 cohesion
template <int G, int KIND>
__global__ void __launch_bounds__(kLaneBlock) k_flock_lanes(GroupView g,
                                                            const unsigned* knn,
                                                            unsigned k, OtherView o,
                                                            FlockParams fp) {
    after_previous();
    __shared__ __align__(16) float sh[kLaneBlock / G * LaneSums<G>::kWords];
    constexpr unsigned need = KIND == 0 ? NEED_SEP : KIND == 1 ? NEED_ALI : NEED_COH;
    unsigned i, lane, b;
    const bool act = lanes_agent<G>(g.n, i, lane);
    LaneNeighbour nb;
    nb.ok = lanes_entry<G>(knn, i, g.n, k, o.n, lane, b);
    unsigned applied = g.applied[i];
    Self me;
    me.pos = v3(g.position[i]);
    me.dir = v3(g.direction[i]);
    V3 steer = v3(g.steering[i]);
    nb.pos = nb.ok ? v3(o.position[b]) : me.pos;
    nb.dir = nb.ok && KIND == 1 ? v3(o.direction[b]) : me.dir;
    V3 r_sep, r_ali, r_coh;
    lanes_flock<true>(need, fp, fp, fp, me, lane, nb, LaneSums<G>::of(sh), r_sep, r_ali, r_coh);
    if (!act || lane != 0 || (applied & fp.mask)) return;
    flock_apply(KIND == 0 ? r_sep : KIND == 1 ? r_ali : r_coh, fp,
                KIND == 0 ? SEPARATION_BIT : KIND == 1 ? ALIGNMENT_BIT : COHESION_BIT, applied,
                steer);
    g.steering[i] = f4(steer, 0.f);
    g.applied[i] = applied;
}

// steerToAvoidNeighbors: the close pass (CLOSE) or the main pass.
template <int G, bool CLOSE>
__global__ void __launch_bounds__(kLaneBlock) k_avoid_lanes(GroupView g,
                                                            const unsigned* knn,
                                                            const float* knn_dist,
                                                            unsigned k, OtherView o, float limit,
                                                            float w, unsigned mask) {
    after_previous();
    unsigned i, lane, b;
    const bool act = lanes_agent<G>(g.n, i, lane);
    LaneNeighbour nb;
    nb.ok = lanes_entry<G>(knn, i, g.n, k, o.n, lane, b);
    nb.dist = CLOSE && nb.ok ? knn_dist[i + size_t(lane) * g.n] : 0.f;
    unsigned applied = g.applied[i];
    Self me;
    me.pos = v3(g.position[i]);
    me.dir = v3(g.direction[i]);
    me.speed = g.speed[i];
    me.radius = g.radius[i];
    const float3 sd = g.side[i];
    me.side = v3(sd.x, sd.y, sd.z);
    V3 steer = v3(g.steering[i]);
    if (nb.ok) {
        nb.pos = v3(o.position[b]);
        nb.radius = o.radius[b];
        if (!CLOSE) {
            nb.dir = v3(o.direction[b]);
            nb.speed = o.speed[b];
        }
    } else {
        nb.pos = nb.dir = v3(0.f, 0.f, 0.f);
        nb.speed = nb.radius = 0.f;
    }
    if constexpr (CLOSE) {
        const CloseAcc c = lanes_close<G>(me, limit, nb);
        if (!act || lane != 0 || (applied & mask)) return;
        close_finish<true>(c, w, mask, applied, steer);
    } else {
        const AvoidAcc a = lanes_avoid<G, true>(me, limit, k, nb);
        if (!act || lane != 0 || a.threat == UINT_MAX) return;
        avoid_finish<true>(a, w, mask, me, applied, steer);
    }
    g.steering[i] = f4(steer, 0.f);
    g.applied[i] = applied;
}

template <int G>
__global__ void __launch_bounds__(kLaneBlock) k_avoid_walls_lanes(
    GroupView g, const unsigned* knw, unsigned kw, const float4* ls,
    const float4* le, const float4* ln, unsigned n_lines, float min_time,
    float w, unsigned mask) {
    after_previous();
    unsigned i, lane, line;
    const bool act = lanes_agent<G>(g.n, i, lane);
    const bool ok = lanes_entry<G>(knw, i, g.n, kw, n_lines, lane, line);
    unsigned applied = g.applied[i];
    Self me;
    me.pos = v3(g.position[i]);
    me.dir = v3(g.direction[i]);
    me.speed = g.speed[i];
    me.radius = g.radius[i];
    const float3 sd = g.side[i];
    me.side = v3(sd.x, sd.y, sd.z);
    V3 steer = v3(g.steering[i]);
    const unsigned lines = __popc(lanes_ballot<G>(ok));
    const unsigned most = __reduce_max_sync(kAllLanes, lines);
    WallAcc wa;
    walls_init(wa, me, min_time);
    for (unsigned r = 0; r < most; ++r) {
        const unsigned at = __shfl_sync(kAllLanes, line, int(r), G);
        const bool on = r < lines;
        const unsigned s = on ? at : 0u;
        lanes_wall_line<G>(wa, me, lane, at, on, v3(ls[s]), v3(le[s]), v3(ln[s]));
    }
    if (!act || lane != 0 || (applied & mask)) return;
    walls_finish(wa, w, mask, me, applied, steer);
    g.steering[i] = f4(steer, 0.f);
    g.position[i] = f4(me.pos, 0.f);
    g.direction[i] = f4(me.dir, 0.f);
    g.applied[i] = applied;
}

template <int G>
static void flock_lanes_go(int kind, GroupView g, const unsigned* knn, unsigned k, OtherView o,
                           FlockParams fp, cudaStream_t st) {
    const unsigned nb = blocks_for(g.n, kLaneBlock / G);
    if (kind == 0) launch_after(k_flock_lanes<G, 0>, nb, kLaneBlock, 0, st, g, knn, k, o, fp);
    else if (kind == 1) launch_after(k_flock_lanes<G, 1>, nb, kLaneBlock, 0, st, g, knn, k, o, fp);
    else launch_after(k_flock_lanes<G, 2>, nb, kLaneBlock, 0, st, g, knn, k, o, fp);
}
void launch_flock_lanes(int kind, GroupView g, const unsigned* knn, unsigned k, OtherView o,
                        FlockParams fp, cudaStream_t st) {
    if (k <= 8) flock_lanes_go<8>(kind, g, knn, k, o, fp, st);
    else if (k <= 16) flock_lanes_go<16>(kind, g, knn, k, o, fp, st);
    else flock_lanes_go<32>(kind, g, knn, k, o, fp, st);
}

template <int G>
static void avoid_lanes_go(GroupView g, const unsigned* knn, const float* knn_dist, unsigned k,
                           OtherView o, float min_time, float min_sep, bool close, float w,
                           unsigned mask, cudaStream_t st) {
    const unsigned nb = blocks_for(g.n, kLaneBlock / G);
    if (close)
        launch_after(k_avoid_lanes<G, true>, nb, kLaneBlock, 0, st, g, knn, knn_dist, k, o, min_sep, w, mask);
    launch_after(k_avoid_lanes<G, false>, nb, kLaneBlock, 0, st, g, knn, nullptr, k, o, min_time, w, mask);
}
void launch_avoid_lanes(GroupView g, const unsigned* knn, const float* knn_dist, unsigned k,
                        OtherView o, float min_time, float min_sep, bool close, float w,
                        unsigned mask, cudaStream_t st) {
    if (k <= 8) avoid_lanes_go<8>(g, knn, knn_dist, k, o, min_time, min_sep, close, w, mask, st);
    else if (k <= 16)
        avoid_lanes_go<16>(g, knn, knn_dist, k, o, min_time, min_sep, close, w, mask, st);
    else avoid_lanes_go<32>(g, knn, knn_dist, k, o, min_time, min_sep, close, w, mask, st);
}

void launch_avoid_walls_lanes(GroupView g, const unsigned* knw, unsigned kw, const float4* start,
                              const float4* end, const float4* normal, unsigned n_lines,
                              float min_time, float w, unsigned mask, cudaStream_t st) {
    launch_after(k_avoid_walls_lanes<8>, blocks_for(g.n, kLaneBlock / 8), kLaneBlock, 0, st, g, knw, kw, start, end, normal, n_lines, min_time, w, mask);
}

// ---- MultiGroup frames ------------------------------------------------------------------------
// One group's part of a frame (Group::update, plugins/MultiGroup.cpp:558-610) in
// two launches instead of one for steering, one for the update and three for
// each group's anti-penetration: 72 launches and copies a frame of three groups
// took 400 us, almost all of it between kernels.
//
// The first: steering as k_multigroup_steer (each list gathered once, lane r
// its entry r), the update, and anti-penetration against the groups before
// this one, whose agents have moved.  Other agents of this group read its
// position, heading and speed of before the update meanwhile, so the new ones
// go to M.next.
//
// Anti-penetration (AntiPenetrationAgentsCUDAKernel.cu:72-108, as k_antipen)
// takes the groups one after another, but what it reads of each does not depend
// on the ones before: lane t loads group first + t's nearest neighbour, then the
// pushes are applied in order.
template <int G>
__device__ __forceinline__ void lanes_push_apart(const MultiSteer& M, unsigned a, unsigned lane,
                                                 unsigned first, unsigned last, V3& pos,
                                                 float radius, unsigned& applied) {
    bool near = false;
    V3 at = v3(0.f, 0.f, 0.f);
    float overlap = 0.f;
    unsigned bits = 0;
    const unsigned j = first + lane;
    if (j < last) {
        const OtherView& o = M.o[j];
        const bool own = j == M.self;  // this group's agents have moved to M.next
        const unsigned b = M.idx[j][a];
        const float d = M.dist[j][a];
        if (b < o.n) {
            at = v3(own ? M.next.position[b] : o.position[b]);
            bits = own ? M.next.applied[b] : o.applied[b];
            overlap = radius + o.radius[b] - d;
            near = !(overlap < 0.f);
        }
    }
    const unsigned m = lanes_ballot<G>(near);
    for (unsigned t = 0; t < last - first; ++t) {
        const V3 other = lanes_get<G>(at, t);
        const float over = __shfl_sync(kAllLanes, overlap, int(t), G);
        const unsigned ob = __shfl_sync(kAllLanes, bits, int(t), G);
        if (!((m >> t) & 1u) || (applied & M.mask_antipen)) continue;
        const V3 unit = normalize(sub(pos, other));
        pos = add(pos, mul(unit, (ob & M.mask_antipen) ? over : 0.5f * over));
        applied |= ANTI_PENETRATION_AGENT;
    }
}

template <int G>
__global__ void __launch_bounds__(kLaneBlock) k_group_move(const __grid_constant__ MultiSteer M) {
    after_previous();
    __shared__ __align__(16) float sh[kLaneBlock / G * LaneSums<G>::kWords];
    const GroupView& g = M.g;
    unsigned a, lane;
    const bool act = lanes_agent<G>(g.n, a, lane);
    const LaneSums<G> sums = LaneSums<G>::of(sh);
    unsigned applied = g.applied[a];
    V3 steer = v3(g.steering[a]);
    Self me;
    me.pos = v3(g.position[a]);
    me.dir = v3(g.direction[a]);
    me.speed = g.speed[a];
    me.radius = g.radius[a];
    const float3 sd = g.side[a];
    me.side = v3(sd.x, sd.y, sd.z);
    V3 mine = v3(0.f, 0.f, 0.f), r_ali = mine, r_coh = mine;  // lane j: separation from group j
    auto neighbour = [&](unsigned j) {
        const OtherView& o = M.o[j];
        LaneNeighbour nb;
        unsigned b;
        nb.ok = lanes_entry<G>(M.idx[j], a, g.n, M.k[j], o.n, lane, b);
        nb.pos = nb.dir = v3(0.f, 0.f, 0.f);
        nb.speed = nb.radius = nb.dist = 0.f;
        if (nb.ok) {
            nb.pos = v3(o.position[b]);
            nb.dir = v3(o.direction[b]);
            nb.speed = o.speed[b];
            nb.radius = o.radius[b];
            nb.dist = M.dist[j][a + size_t(lane) * g.n];
        }
        return nb;
    };
    // the next group's neighbours are on their way while one group is taken
    LaneNeighbour nb = neighbour(0), next;
    for (unsigned j = 0; j < M.n_groups; ++j, nb = next) {
        next = neighbour(j + 1 < M.n_groups ? j + 1 : j);
        V3 r_sep, none;
        if (j != M.self) {
            lanes_flock(NEED_SEP, M.sep, M.sep, M.sep, me, lane, nb, sums, r_sep, none, none);
            if (M.avoid_close) {
                const CloseAcc c = lanes_close<G>(me, M.min_sep, nb);
                close_finish(c, M.w_avoid, M.mask_avoid, applied, steer);
            }
            const AvoidAcc v = lanes_avoid<G>(me, M.min_time, M.k[j], nb);
            avoid_finish(v, M.w_avoid, M.mask_avoid, me, applied, steer);
        } else {
            lanes_flock(NEED_SEP | NEED_ALI | NEED_COH, M.sep, M.ali, M.coh, me, lane, nb, sums,
                        r_sep, r_ali, r_coh);
        }
        if (lane == j) mine = r_sep;
    }
    for (unsigned j = 0; j < M.n_groups; ++j)
        flock_apply(lanes_get<G>(mine, j), M.sep, SEPARATION_BIT, applied, steer);
    flock_apply(r_ali, M.ali, ALIGNMENT_BIT, applied, steer);
    flock_apply(r_coh, M.coh, COHESION_BIT, applied, steer);
    if (M.has_path) {
        follow_path_finish(M.path, M.path_time, M.w_path, M.mask_path, me, applied, steer);
        seek_finish(v3(M.seek_target[0], M.seek_target[1], M.seek_target[2]), M.w_seek, M.mask_seek,
                    me, applied, steer);
    }
    const float3 up = g.up[a];
    me.up = v3(up.x, up.y, up.z);
    me.max_speed = g.max_speed[a];
    me.max_force = g.max_force[a];
    me.mass = g.mass[a];
    integrate(me, steer, M.dt);
    applied = 0u;
    lanes_push_apart<G>(M, a, lane, 0, M.self, me.pos, me.radius, applied);
    if (!act || lane != 0) return;
    M.next.position[a] = f4(me.pos, 0.f);
    M.next.direction[a] = f4(me.dir, 0.f);
    M.next.speed[a] = me.speed;
    M.next.applied[a] = applied;
    g.side[a] = make_float3(me.side.x, me.side.y, me.side.z);
    g.up[a] = make_float3(me.up.x, me.up.y, me.up.z);
    g.steering[a] = make_float4(0.f, 0.f, 0.f, 0.f);
}

// The second: anti-penetration within the group, whose agents have all moved
// now, then against the groups after it, which have not; the result goes to
// the group's arrays.
__global__ void __launch_bounds__(kLaneBlock) k_group_settle(const __grid_constant__ MultiSteer M) {
    after_previous();
    const GroupView& g = M.g;
    unsigned a, lane;
    const bool act = lanes_agent<8>(g.n, a, lane);
    V3 pos = v3(M.next.position[a]);
    unsigned applied = M.next.applied[a];
    const float4 dir = M.next.direction[a];
    const float speed = M.next.speed[a];
    lanes_push_apart<8>(M, a, lane, M.self, M.n_groups, pos, g.radius[a], applied);
    if (!act || lane != 0) return;
    g.position[a] = f4(pos, 0.f);
    g.direction[a] = dir;
    g.speed[a] = speed;
    g.applied[a] = applied;
}
static_assert(kMaxGroups <= 8, "a lane per group");

// k <= 32 for every list; a group of a few agents a lane group each, larger
// groups keep one thread per agent (k_multigroup_steer and the calls after it).
bool lanes_multigroup(const MultiSteer& M) {
    for (unsigned j = 0; j < M.n_groups; ++j)
        if (M.k[j] > 32) return false;
    return M.g.n <= 65536;
}

gs_status launch_group_frame(const MultiSteer& M, cudaStream_t st) {
    if (M.g.n == 0) return GS_OK;
    unsigned k = 0;
    for (unsigned j = 0; j < M.n_groups; ++j) k = M.k[j] > k ? M.k[j] : k;
    if (k <= 8) launch_after(k_group_move<8>, blocks_for(M.g.n, kLaneBlock / 8), kLaneBlock, 0, st, M);
    else if (k <= 16) launch_after(k_group_move<16>, blocks_for(M.g.n, kLaneBlock / 16), kLaneBlock, 0, st, M);
    else launch_after(k_group_move<32>, blocks_for(M.g.n, kLaneBlock / 32), kLaneBlock, 0, st, M);
    launch_after(k_group_settle, blocks_for(M.g.n, kLaneBlock / 8), kLaneBlock, 0, st, M);
    GS_LAUNCHED("group_frame");
    return GS_OK;
}

// Under ncu, lanes / threads (us; a launch's floor is about 3): one flocking
// behaviour, k = 7, 30,000 agents 7.5 / 6.5; k = 16, 10,000 6.5 / 11.3, 32,768
// 10.2 / about 9.5.  The avoidance passes and the walls carry more arithmetic
// per neighbour, and their line lies by the lanes in all (us a call of the main
// pass: k = 7, 50,000 agents 9.7 / 11.4, 65,536 11.5 / 11.7; k = 16, 20,000 7.9 /
// 12.0, 30,000 10.5 / 11.6, 65,536 19.1 / 16.0; k = 32, 10,000 9.2 / 11.5, 14,000
// 11.6 / 12.2, 20,000 15.5 / 13.0, 65,536 43 / 18; the close pass turns at two
// thirds of that).
bool lanes_calls(unsigned n, unsigned k, bool avoid) {
    const unsigned G = k <= 8 ? 8u : k <= 16 ? 16u : 32u;
    return k <= 32 && (avoid ? size_t(n) * G <= 450000 : n <= 20000u);
}

template <int G, int R>
static void launch_lanes_r(const FusedLaunch& L, const StepDev& p, unsigned nb, cudaStream_t st,
                           PhaseHook* hook) {
    if (!(p.need & NEED_WALLS)) {
        if (hook) hook->mark(2, true);
        if ((p.need & kNeedList) == (NEED_SEP | NEED_ALI | NEED_COH))
            launch_after(k_lanes_step<G, R, NEED_SEP | NEED_ALI | NEED_COH>, nb, kLaneBlock, 0, st, L, p);
        else
            launch_after(k_lanes_step<G, R, kNeedRuntime>, nb, kLaneBlock, 0, st, L, p);
        if (hook) hook->mark(2, false);
        return;
    }
    if (hook) hook->mark(2, true);
    launch_after(k_lanes_walls<G, R>, nb, kLaneBlock, 0, st, L, p);
    if (hook) hook->mark(2, false);
    if (hook) hook->mark(3, true);
    if ((p.need & kNeedList) == (NEED_SEP | NEED_AVOID))
        launch_after(k_lanes_rest<G, NEED_SEP | NEED_AVOID>, nb, kLaneBlock, 0, st, L, p);
    else
        launch_after(k_lanes_rest<G, kNeedRuntime>, nb, kLaneBlock, 0, st, L, p);
    if (hook) hook->mark(3, false);
}

template <int G>
static gs_status launch_lanes(const FusedLaunch& L, const StepDev& p, cudaStream_t st,
                              PhaseHook* hook) {
    const unsigned nb = blocks_for(L.n, kLaneBlock / G);
    if (p.r != 1) launch_lanes_r<G, 0>(L, p, nb, st, hook);
    else if (p.flat) launch_lanes_r<G, 3>(L, p, nb, st, hook);
    else launch_lanes_r<G, 9>(L, p, nb, st, hook);
    GS_LAUNCHED("fused_step_lanes");
    return GS_OK;
}

// One thread per agent costs about a quarter of the issue slots but takes its
// whole serial chain however few agents there are.  Measured per step
// (threads, lanes): flock k = 16, 4,096 agents 27.3 / 16.5 us, 16,384 29.5 /
// 28.8, 32,768 31.8 / 45.1; k = 7, 16,384 24.0 / 22.6, 32,768 25.2 / 30.8;
// k = 24, 4,096 29.3 / 20.6, 16,384 38.3 / 39.0; a crowd with walls (which
// also drops the exact lists' launch), 10,000 53.5 / 31.0, 20,000 59.9 / 47.9;
// eight of them, 20,219 agents together, 40.8 / 43.1.
bool lanes_preferred(unsigned n, bool walls) { return n <= (walls ? kLanesMost : 16384u); }

gs_status fused_step_lanes(const FusedLaunch& L, const StepDev& p, cudaStream_t st,
                           PhaseHook* hook) {
    if (L.n == 0) return GS_OK;
    if ((p.need & NEED_WALLS) && p.knw > 8)
        return fail(GS_ERR_UNSUPPORTED, "knw > 8 in the fused step");
    if (p.k <= 8) return launch_lanes<8>(L, p, st, hook);
    if (p.k <= 16) return launch_lanes<16>(L, p, st, hook);
    return launch_lanes<32>(L, p, st, hook);
}

}  // namespace gs
