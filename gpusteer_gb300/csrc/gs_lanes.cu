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

// The neighbour pass and the behaviours order[first..] of one agent: lane r
// holds neighbour r (ok: there is one) in b0 (position), b1 (heading | speed),
// br (radius) and its KNN distance kd.  Each lane evaluates its neighbour's
// terms with the reference's expressions; the sums run in list order.
template <int G>
__device__ __forceinline__ void lanes_behaviours(const StepDev& p, unsigned need, unsigned first,
                                                 const Self& me, unsigned lane, bool ok, V3 bpos,
                                                 V3 bdir, float bspeed, float br, float kd,
                                                 float* shared, unsigned& applied, V3& steer) {
    const V3 zero = v3(0.f, 0.f, 0.f);
    V3 r_sep = zero, r_ali = zero, r_coh = zero;
    if (need & (NEED_SEP | NEED_ALI | NEED_COH)) {
        LaneSums<G> sums{shared + (threadIdx.x / G) * LaneSums<G>::kWords};
        const V3 offset = sub(bpos, me.pos);
        const float dsq = dot(offset, offset), d = sqrtf(dsq);
        const float ahead = dot(me.dir, dvd(offset, d));
        auto member = [&](const float v[5]) {
            return ok && (d < v[0] || (!(d > v[1]) && ahead > v[2]));
        };
        unsigned n_sep = 0, n_ali = 0, n_coh = 0;
        if (need & NEED_SEP) {
            const bool in = member(p.sep);
            n_sep = __popc(lanes_ballot<G>(in));
            sums.put(0, lane, in ? dvd(offset, -dsq) : zero);
        }
        if (need & NEED_ALI) {
            const bool in = member(p.ali);
            n_ali = __popc(lanes_ballot<G>(in));
            sums.put(3, lane, in ? bdir : zero);
        }
        if (need & NEED_COH) {
            const bool in = member(p.coh);
            n_coh = __popc(lanes_ballot<G>(in));
            sums.put(6, lane, in ? bpos : zero);
        }
        sums.add_rows(lane);
        // lanes 0, 1, 2: the three behaviours' finish (flock_finish) side by side
        const unsigned kind = lane < 2 ? lane : 2u;
        const unsigned n = kind == 0 ? n_sep : kind == 1 ? n_ali : n_coh;
        const float w = kind == 0 ? p.sep[3] : kind == 1 ? p.ali[3] : p.coh[3];
        V3 r = n ? sums.sum(3 * kind) : zero;
        if (n) {
            const V3 mean = dvd(r, float(n));
            r = normalize(kind == 0 ? mean : sub(mean, kind == 1 ? me.dir : me.pos));
        }
        r = mul(r, w);
        if (need & NEED_SEP) r_sep = lanes_get<G>(r, 0);
        if (need & NEED_ALI) r_ali = lanes_get<G>(r, 1);
        if (need & NEED_COH) r_coh = lanes_get<G>(r, 2);
    }
    CloseAcc close;
    close_init(close);
    AvoidAcc avoid;
    avoid_init(avoid, p.min_time_col);
    if (need & NEED_CLOSE) {
        CloseAcc c;
        close_init(c);
        if (ok) close_add(c, me, p.min_sep, kd, bpos, br);
        const unsigned m = lanes_ballot<G>(c.found);
        const V3 s = lanes_get<G>(c.steer, m ? unsigned(__ffs(int(m)) - 1) : 0u);
        if (m) close.steer = s;
    }
    if (need & NEED_AVOID) {
        // every lane its neighbour's approach time and distance; then the
        // reference's pass over them in list order (avoid_add), whose window
        // [0, min_t) only narrows
        V3 at = zero;
        float t = __int_as_float(0x7f800000);
        bool danger = false;
        if (ok) {
            const float time =
                nearest_approach_time(me.pos, me.dir, me.speed, bpos, bdir, bspeed);
            if (time >= 0.f) t = time;
            danger = nearest_approach_positions(me.pos, me.dir, me.speed, bpos, bdir, bspeed, time,
                                                at) < me.radius + br;
        }
        const unsigned hits = lanes_ballot<G>(danger);
        unsigned last = UINT_MAX, threat = UINT_MAX;
        for (unsigned r = 0; r < p.k; ++r) {
            const float tr = __shfl_sync(kAllLanes, t, int(r), G);
            if (tr < avoid.min_t) {
                last = r;
                if ((hits >> r) & 1u) {
                    avoid.min_t = tr;
                    threat = r;
                }
            }
        }
        const unsigned lf = last == UINT_MAX ? 0u : last, tf = threat == UINT_MAX ? 0u : threat;
        const V3 la = lanes_get<G>(at, lf), tp = lanes_get<G>(bpos, tf), td = lanes_get<G>(bdir, tf);
        const float ts = __shfl_sync(kAllLanes, bspeed, int(tf), G);
        if (last != UINT_MAX) avoid.threat_at = la;
        if (threat != UINT_MAX) {
            avoid.threat = threat;
            avoid.threat_pos = tp;
            avoid.threat_dir = td;
            avoid.threat_speed = ts;
        }
    }
    auto flock = [&](V3 r, const float v[5], unsigned bit) {
        if (applied & __float_as_uint(v[4])) return;
        if (!is_zero(r)) applied |= bit;
        steer = add(r, steer);
    };
#pragma unroll 1
    for (unsigned o = first; o < p.n_order; ++o) {
        switch ((p.order_packed >> (3u * o)) & 7u) {
            case GS_B_SEPARATION:
                if (need & NEED_SEP) flock(r_sep, p.sep, SEPARATION_BIT);
                break;
            case GS_B_ALIGNMENT:
                if (need & NEED_ALI) flock(r_ali, p.ali, ALIGNMENT_BIT);
                break;
            case GS_B_COHESION:
                if (need & NEED_COH) flock(r_coh, p.coh, COHESION_BIT);
                break;
            case GS_B_SEEK:
                seek_finish(v3(p.seek_target[0], p.seek_target[1], p.seek_target[2]), p.w_seek,
                            p.mask_seek, me, applied, steer);
                break;
            case GS_B_AVOID_NEIGHBORS:
                if (need & NEED_AVOID) {
                    if (p.avoid_close) close_finish(close, p.w_avoid, p.mask_avoid, applied, steer);
                    avoid_finish(avoid, p.w_avoid, p.mask_avoid, me, applied, steer);
                }
                break;
            case GS_B_FOLLOW_PATH:
                follow_path_finish(p.path, p.path_time, p.w_path, p.mask_path, me, applied, steer);
                break;
            default: break;
        }
    }
}

// ---- whole step without walls -----------------------------------------------------------
template <int G, int R, unsigned NEEDC>
__global__ void __launch_bounds__(kLaneBlock) k_lanes_step(FusedLaunch L, StepDev p) {
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
                                            L.start, L.B.f[0]);
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
    lanes_behaviours<G>(p, need, 0, me, lane, ok, v3(b0), v3(b1), b1.w, br, key_dist(nb.key), sh,
                        applied, steer);
    integrate(me, steer, p.dt);
    if (act && lane == 0) store_next(L, s, me, id, scene, sc, p.wrap_mode);
}

// ---- wall phase ---------------------------------------------------------------------------
// The four tests of a wall line (touching, then the three feelers, walls_add)
// on lanes 0 to 3 of the group; the line's result is then taken in their order.
template <int G>
__device__ __forceinline__ void lanes_wall_line(WallAcc& wa, const Self& me, unsigned lane,
                                                unsigned line, bool on, V3 ls, V3 le, V3 ln) {
    const unsigned t = lane & 3u;
    const V3 end = t == 0 ? add(me.pos, mul(neg(ln), me.radius))
                          : t == 1 ? wa.feelers[0] : t == 2 ? wa.feelers[1] : wa.feelers[2];
    V3 ip = v3(0.f, 0.f, 0.f);
    const bool hit = on && lines_intersect(me.pos, end, ls, le, ip);
    const float d = distance(me.pos, ip);
    const unsigned hits = lanes_ballot<G>(hit) & 15u;
    unsigned from = 0;
#pragma unroll
    for (unsigned f = 0; f < 4; ++f) {
        const float df = __shfl_sync(kAllLanes, d, int(f), G);
        if (!((hits >> f) & 1u)) continue;
        if (f == 0) {
            wa.touching = true;
            wa.nearest_normal = ln;
            wa.nearest_d = df;
        } else if (df < wa.nearest_d) {
            wa.nearest_d = df;
            wa.nearest_line = line;
            wa.feeler_index = f - 1;
            wa.nearest_normal = ln;
            from = f;
        }
    }
    const V3 at = lanes_get<G>(ip, from);
    if (from) wa.nearest_ip = at;
}

template <int G, int R>
__global__ void __launch_bounds__(kLaneBlock) k_lanes_walls(FusedLaunch L, StepDev p) {
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
                                            L.start, L.B.f[0]);
    if (act && lane < p.k) {
        L.knn_slot[size_t(s) * p.k + lane] = nb.slot;
        // the KNN distance (before any wall correction moves agents), read by
        // avoid-close-neighbours only
        if (p.need & NEED_CLOSE) L.knn_dist[size_t(s) * p.k + lane] = key_dist(nb.key);
    }
    unsigned applied = p.clear_applied ? 0u : __float_as_uint(f4v.z);
    V3 steer = p.dirty ? v3(L.B.f[5][s]) : v3(0.f, 0.f, 0.f);
    const bool walls = sc.n_walls > 0 && L.w_pos_id != nullptr;
    if (__any_sync(kAllLanes, walls)) {
        Box wb = box;
        if (!walls) {  // a scene without walls searches an empty box
            wb.y0 = 1;
            wb.y1 = 0;
        }
        const LaneEntry<G> wl =
            lanes_knn<G, R>(p.knw, lane, me.pos, UINT_MAX, sc.grid, wb, sc.wall_cell_offset,
                            L.w_cell_start, L.w_pos_id);
        const unsigned found = lanes_ballot<G>(walls && lane < p.knw && wl.slot != UINT_MAX &&
                                               key_id(wl.key) < sc.n_walls);
        WallAcc wa;
        walls_init(wa, me, p.min_time_wall);
        const unsigned lines = __popc(found);  // the list is filled from rank 0
        const unsigned most = __reduce_max_sync(kAllLanes, lines);
        for (unsigned r = 0; r < most; ++r) {
            const unsigned line = unsigned(__shfl_sync(kAllLanes, wl.key, int(r), G));
            const bool on = r < lines;
            const unsigned g = on ? sc.wall_offset + line : 0u;
            lanes_wall_line<G>(wa, me, lane, line, on, v3(L.w_start[g]), v3(L.w_end[g]),
                               v3(L.w_normal[g]));
        }
        if (walls) walls_finish(wa, p.w_walls, p.mask_walls, me, applied, steer);
        else if (!(applied & p.mask_walls)) steer = add(mul(v3(0.f, 0.f, 0.f), p.w_walls), steer);
    } else if (!(applied & p.mask_walls)) {
        steer = add(mul(v3(0.f, 0.f, 0.f), p.w_walls), steer);
    }
    if (act && lane == 0) {
        L.w0[s] = make_float4(me.pos.x, me.pos.y, me.pos.z, me.radius);
        L.w1[s] = make_float4(me.dir.x, me.dir.y, me.dir.z, me.speed);
        L.w2[s] = make_float4(steer.x, steer.y, steer.z, __uint_as_float(applied));
    }
}

// ---- rest of the step after the wall phase -------------------------------------------------
template <int G, unsigned NEEDC>
__global__ void __launch_bounds__(kLaneBlock) k_lanes_rest(FusedLaunch L, StepDev p) {
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
    lanes_behaviours<G>(p, need, 1, me, lane, ok, v3(b0), v3(b1), b1.w, b0.w, kd, sh, applied,
                        steer);
    integrate(me, steer, p.dt);
    const Scene sc = L.scenes[scene];
    if (act && lane == 0) store_next(L, s, me, id, scene, sc, p.wrap_mode);
}

template <int G, int R>
static void launch_lanes_r(const FusedLaunch& L, const StepDev& p, unsigned nb, cudaStream_t st,
                           PhaseHook* hook) {
    if (!(p.need & NEED_WALLS)) {
        if (hook) hook->mark(2, true);
        if ((p.need & kNeedList) == (NEED_SEP | NEED_ALI | NEED_COH))
            k_lanes_step<G, R, NEED_SEP | NEED_ALI | NEED_COH><<<nb, kLaneBlock, 0, st>>>(L, p);
        else
            k_lanes_step<G, R, kNeedRuntime><<<nb, kLaneBlock, 0, st>>>(L, p);
        if (hook) hook->mark(2, false);
        return;
    }
    if (hook) hook->mark(2, true);
    k_lanes_walls<G, R><<<nb, kLaneBlock, 0, st>>>(L, p);
    if (hook) hook->mark(2, false);
    if (hook) hook->mark(3, true);
    if ((p.need & kNeedList) == (NEED_SEP | NEED_AVOID))
        k_lanes_rest<G, NEED_SEP | NEED_AVOID><<<nb, kLaneBlock, 0, st>>>(L, p);
    else
        k_lanes_rest<G, kNeedRuntime><<<nb, kLaneBlock, 0, st>>>(L, p);
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
bool lanes_preferred(unsigned n, bool walls) { return n <= (walls ? 20000u : 16384u); }

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
