// The fused step of a small group without a sort: one launch (two with walls)
// a step.
//
// The sorting step (gs_step.cu) is a chain of launches, scan, permute, step,
// whose latency is most of a small group's step.  Here agents keep their order
// and each cell has a fixed row of the table: the step's last act is to put
// (position, index) into the next table at its cell's count, and the next
// step's search reads the counts and rows of its box.  Two tables and three
// count arrays take turns: a step reads one, fills the next, and clears the
// third, which the step after fills.
//
// A cell that holds more than a row goes on in further rows, found by hashing
// (cell, row number): whoever puts an agent there claims the hashed slot's tag,
// or finds it claimed for the same row, and takes the next slot otherwise.
// Nothing is allocated and nobody waits, and a search reads what its box holds
// and no more, however crowded the rest of the world is.  (One overflow list
// for the whole world, which every agent scanned, took 8 steps of 16,384 boids
// in clumps of 60 to 3844 us instead of 279, and of a choke point's 10,000
// agents 1,200 steps on to 407 instead of 272; sorted, 276 and 290.)
//
// A group of lanes serves each agent (gs_lanes.cuh): lane by lane it loads the
// box's counts, lays the candidates' places end to end in shared memory, and
// takes them G at a time into an exact list.
#include "gs_lanes.cuh"
#include "gs_step.cuh"
#include "gs_table.cuh"

namespace gs {

constexpr unsigned kTableBlock = 128;
constexpr unsigned kTablePlaces = 128;  // candidates laid end to end per lane group

// Row `number` (from 1) of cell c, as its tag.  The tables' sizes keep both in
// their bits: at most 2^22 places in rows of 16 or more, and the lanes' groups
// have at most kLanesMost agents.
constexpr unsigned kTagCellBits = 18;
static_assert((kLanesMost >> 4) < 1u << (32 - kTagCellBits), "row numbers overflow a tag");
__device__ __forceinline__ unsigned row_tag(unsigned c, unsigned number) {
    return number << kTagCellBits | c;
}
__device__ __forceinline__ unsigned tag_slot(unsigned tag, unsigned ext_log2) {
    return (tag * 0x9e3779b1u) >> (32u - ext_log2);
}
// There are twice as many slots as further rows of n agents (table_reserve),
// so both loops end at their row.
__device__ __forceinline__ unsigned claim_row(const TableStep& T, unsigned c, unsigned number) {
    const unsigned tag = row_tag(c, number), last = (1u << T.ext_log2) - 1u;
    unsigned s = tag_slot(tag, T.ext_log2);
    for (unsigned i = 0; i < last; ++i, s = (s + 1u) & last) {
        const unsigned old = atomicCAS(T.tag_next + s, 0u, tag);
        if (old == 0u || old == tag) break;
    }
    return s;
}
__device__ __forceinline__ unsigned find_row(const TableStep& T, unsigned c, unsigned number) {
    const unsigned tag = row_tag(c, number), last = (1u << T.ext_log2) - 1u;
    unsigned s = tag_slot(tag, T.ext_log2);
    for (unsigned i = 0; i < last && T.tag[s] != tag; ++i) s = (s + 1u) & last;
    return s;
}
// Entry t of cell c.
__device__ __forceinline__ float4 table_entry(const TableStep& T, unsigned c, unsigned t) {
    const unsigned number = t >> T.row_log2;
    const unsigned row = number == 0 ? c : T.cells + find_row(T, c, number);
    return T.tab[(row << T.row_log2) + (t & ((1u << T.row_log2) - 1u))];
}

// Puts the agent in the next step's table.
__device__ __forceinline__ void table_put(const TableStep& T, V3 pos, int wrap_mode, unsigned id) {
    const V3 p = wrap_world(pos, T.sc.grid.ws, wrap_mode);
    const unsigned c = cell_of(T.sc.grid, p);
    const unsigned at = atomicAdd(T.cnt_next + c, 1u);
    const float4 e = make_float4(p.x, p.y, p.z, __uint_as_float(id));
    const unsigned number = at >> T.row_log2;
    const unsigned row = number == 0 ? c : T.cells + claim_row(T, c, number);
    T.tab_next[(row << T.row_log2) + (at & ((1u << T.row_log2) - 1u))] = e;
}

// Clears the counts and tags that the step after this one fills.
__device__ __forceinline__ void table_clear(const TableStep& T) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    for (unsigned i = t; i < T.cells; i += nt) T.cnt_clear[i] = 0u;
    for (unsigned i = t; i < 1u << T.ext_log2; i += nt) T.tag_clear[i] = 0u;
}

// The k nearest of the 27 (FLAT: 9) cells of box b, over the group's lanes.
template <int G, bool FLAT>
__device__ __forceinline__ LaneList<G, 1> table_knn(const TableStep& T, unsigned k, unsigned lane,
                                                    V3 p, unsigned self_id, const Box& b,
                                                    unsigned* places) {
    constexpr int CELLS = FLAT ? 9 : 27, Q = (CELLS + G - 1) / G;
    const Grid& g = T.sc.grid;
    LaneList<G, 1> list;
    list.e[0] = KEY_EMPTY;
    auto take = [&](float4 v, bool ok) {
        const unsigned id = __float_as_uint(v.w);
        const unsigned long long key = knn_key(distance(p, v3(v)), id);
        list.take(ok && id != self_id && key < KEY_EMPTY ? key : KEY_EMPTY, k, lane);
    };
    unsigned cell[Q], len[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const unsigned i = lane + unsigned(q * G);
        const unsigned x = b.x0 + i % 3u, z = b.z0 + (i / 3u) % 3u, y = b.y0 + i / 9u;
        cell[q] = len[q] = 0;
        if (i < unsigned(CELLS) && x <= b.x1 && y <= b.y1 && z <= b.z1) {
            cell[q] = cell_label(g, x, y, z);
            len[q] = T.cnt[cell[q]];
        }
    }
    unsigned total = 0, first[Q];
    bool rows = true;  // this lane's cells are within their rows
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        unsigned sum = len[q];
#pragma unroll
        for (int o = 1; o < G; o <<= 1) {
            const unsigned v = __shfl_up_sync(kAllLanes, sum, o, G);
            if (lane >= unsigned(o)) sum += v;
        }
        first[q] = total + sum - len[q];
        total += __shfl_sync(kAllLanes, sum, G - 1, G);
        rows = rows && len[q] <= 1u << T.row_log2;
    }
    const unsigned most = __reduce_max_sync(kAllLanes, total);
    if (most <= kTablePlaces && __all_sync(kAllLanes, rows)) {
#pragma unroll
        for (int q = 0; q < Q; ++q)
            for (unsigned t = 0; t < len[q]; ++t)
                places[first[q] + t] = (cell[q] << T.row_log2) + t;
        __syncwarp();
        // the next candidate is on its way while this one is taken
        auto load = [&](unsigned j) {
            return j < total ? T.tab[places[j]] : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        float4 v = load(lane);
        for (unsigned j = lane; j < most + lane; j += G) {
            const float4 next = load(j + G);
            take(v, j < total);
            v = next;
        }
    } else {  // crowded boxes: the cells end to end, a lane's cell found as it goes
        unsigned* cells = places;
        unsigned* pre = places + CELLS;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const unsigned i = lane + unsigned(q * G);
            if (i < unsigned(CELLS)) {
                cells[i] = cell[q];
                pre[i] = first[q];
            }
        }
        if (lane == 0) pre[CELLS] = total;
        __syncwarp();
        unsigned at = UINT_MAX, begin = 0, end = 0, c = 0;
        auto load = [&](unsigned j) {
            if (j >= total) return make_float4(0.f, 0.f, 0.f, 0.f);
            if (j >= end) {
                do end = pre[++at + 1];
                while (j >= end);
                begin = pre[at];
                c = cells[at];
            }
            return table_entry(T, c, j - begin);
        };
        float4 v = load(lane);
        for (unsigned j = lane; j < most + lane; j += G) {
            const float4 next = load(j + G);
            take(v, j < total);
            v = next;
        }
    }
    return list;
}

template <int G>
__device__ __forceinline__ bool table_agent(unsigned n, unsigned& i, unsigned& lane) {
    const unsigned a = (blockIdx.x * kTableBlock + threadIdx.x) / G;
    lane = threadIdx.x & unsigned(G - 1);
    i = a < n ? a : n - 1;
    return a < n;
}

__device__ __forceinline__ Self table_self(const TableStep& T, unsigned a, int wrap_mode,
                                           float4& f4v) {
    const float4 f0 = T.f0[a], f1 = T.f1[a], f2 = T.f2[a], f3 = T.f3[a];
    f4v = T.f4[a];
    Self me;
    me.pos = wrap_world(v3(f0), T.sc.grid.ws, wrap_mode);
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

// The agent's new state, in place but for the position and heading that other
// agents still read (f0_next, f1_next).
__device__ __forceinline__ void table_store(const TableStep& T, unsigned a, const Self& me,
                                            unsigned bits, int wrap_mode) {
    table_put(T, me.pos, wrap_mode, a);
    T.f0_next[a] = make_float4(me.pos.x, me.pos.y, me.pos.z, __uint_as_float(a));
    T.f1_next[a] = make_float4(me.dir.x, me.dir.y, me.dir.z, me.speed);
    // other agents may be reading the radius beside the side
    *reinterpret_cast<float2*>(T.f2 + a) = make_float2(me.side.x, me.side.y);
    reinterpret_cast<float*>(T.f2 + a)[2] = me.side.z;
    T.f3[a] = make_float4(me.up.x, me.up.y, me.up.z, me.mass);
    if (bits) T.f4[a] = make_float4(me.max_speed, me.max_force, 0.f, 0.f);  // the update clears them
}

// ---- whole step without walls -----------------------------------------------------------
template <int G, bool FLAT, unsigned NEEDC>
__global__ void __launch_bounds__(kTableBlock) k_table_step(const __grid_constant__ TableStep T,
                                                            const __grid_constant__ StepDev p) {
    after_previous();
    __shared__ __align__(16) float sh[kTableBlock / G * LaneSums<G>::kWords];
    __shared__ unsigned place_sh[kTableBlock / G * kTablePlaces];
    const unsigned need = NEEDC == kNeedRuntime ? p.need : NEEDC;
    unsigned a, lane;
    const bool act = table_agent<G>(T.n, a, lane);
    table_clear(T);
    float4 f4v;
    Self me = table_self(T, a, p.wrap_mode, f4v);
    unsigned ix, iy, iz;
    cell_coords(T.sc.grid, me.pos, ix, iy, iz);
    const LaneList<G, 1> list =
        table_knn<G, FLAT>(T, p.k, lane, me.pos, a, cell_box(T.sc.grid, ix, iy, iz, 1),
                           place_sh + threadIdx.x / G * kTablePlaces);
    const bool ok = lane < p.k && list.e[0] < KEY_EMPTY;
    const unsigned b = ok ? key_id(list.e[0]) : a;
    const float4 b0 = T.f0[b], b1 = T.f1[b];
    const float br = (need & (NEED_AVOID | NEED_CLOSE))
                         ? reinterpret_cast<const float*>(T.f2 + b)[3] : 0.f;
    const LaneNeighbour nb{ok, wrap_world(v3(b0), T.sc.grid.ws, p.wrap_mode), v3(b1), b1.w, br,
                           key_dist(list.e[0])};
    const unsigned bits = __float_as_uint(f4v.z);
    unsigned applied = p.clear_applied ? 0u : bits;
    V3 steer = p.dirty ? v3(T.f5[a]) : v3(0.f, 0.f, 0.f);
    lanes_behaviours<G, FLAT>(p, need, 0, me, lane, nb, LaneSums<G>::of(sh), applied, steer);
    integrate<FLAT>(me, steer, p.dt);
    if (act && lane == 0) table_store(T, a, me, bits, p.wrap_mode);
}

// ---- wall phase and the rest of the step -----------------------------------------------------
template <int G, bool FLAT>
__global__ void __launch_bounds__(kTableBlock) k_table_walls(const __grid_constant__ TableStep T,
                                                             const __grid_constant__ StepDev p) {
    after_previous();
    __shared__ unsigned place_sh[kTableBlock / G * kTablePlaces];
    unsigned a, lane;
    const bool act = table_agent<G>(T.n, a, lane);
    table_clear(T);
    float4 f4v;
    Self me = table_self(T, a, p.wrap_mode, f4v);
    unsigned ix, iy, iz;
    cell_coords(T.sc.grid, me.pos, ix, iy, iz);
    const Box box = cell_box(T.sc.grid, ix, iy, iz, 1);
    const LaneList<G, 1> list = table_knn<G, FLAT>(T, p.k, lane, me.pos, a, box,
                                                   place_sh + threadIdx.x / G * kTablePlaces);
    if (act && lane < p.k) {
        T.near[size_t(a) * p.k + lane] = key_id(list.e[0]);  // UINT_MAX for none
        if (p.need & NEED_CLOSE) T.near_dist[size_t(a) * p.k + lane] = key_dist(list.e[0]);
    }
    const unsigned bits = __float_as_uint(f4v.z);
    unsigned applied = p.clear_applied ? 0u : bits;
    V3 steer = p.dirty ? v3(T.f5[a]) : v3(0.f, 0.f, 0.f);
    lanes_walls<G, FLAT ? 3 : 9>(T.walls, T.sc, p, me, lane, box, applied, steer);
    if (act && lane == 0) {
        T.w0[a] = make_float4(me.pos.x, me.pos.y, me.pos.z, me.radius);
        T.w1[a] = make_float4(me.dir.x, me.dir.y, me.dir.z, me.speed);
        T.w2[a] = make_float4(steer.x, steer.y, steer.z, __uint_as_float(applied));
    }
}

template <int G, unsigned NEEDC>
__global__ void __launch_bounds__(kTableBlock) k_table_rest(const __grid_constant__ TableStep T,
                                                            const __grid_constant__ StepDev p) {
    after_previous();
    __shared__ __align__(16) float sh[kTableBlock / G * LaneSums<G>::kWords];
    const unsigned need = NEEDC == kNeedRuntime ? p.need : NEEDC;
    unsigned a, lane;
    const bool act = table_agent<G>(T.n, a, lane);
    const unsigned near = lane < p.k ? T.near[size_t(a) * p.k + lane] : UINT_MAX;
    const bool ok = near != UINT_MAX;
    const unsigned b = ok ? near : a;
    const float4 b0 = T.w0[b], b1 = T.w1[b];
    const float kd = (need & NEED_CLOSE) && lane < p.k ? T.near_dist[size_t(a) * p.k + lane] : 0.f;
    const float4 w0 = T.w0[a], w1 = T.w1[a], w2 = T.w2[a];
    float4 f4v;
    Self me = table_self(T, a, WRAP_NONE, f4v);
    me.pos = v3(w0);
    me.dir = v3(w1);
    me.speed = w1.w;
    const LaneNeighbour nb{ok, v3(b0), v3(b1), b1.w, b0.w, kd};
    unsigned applied = __float_as_uint(w2.w);
    V3 steer = v3(w2);
    lanes_behaviours<G, true>(p, need, 1, me, lane, nb, LaneSums<G>::of(sh), applied, steer);
    integrate<true>(me, steer, p.dt);
    if (act && lane == 0) table_store(T, a, me, __float_as_uint(f4v.z), p.wrap_mode);
}

// ---- from the reference layout -----------------------------------------------------------------
// A in agent order and the first table (T's `next` one; its counts are zero).
__global__ void k_table_init(GroupView g, const __grid_constant__ TableStep T, int wrap_mode,
                             int dirty, float4* f5, unsigned* redo_count) {
    after_previous();
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i == 0) *redo_count = 0u;
    if (i >= g.n) return;
    const float4 p = g.position[i], d = g.direction[i];
    const float3 sd = g.side[i], up = g.up[i];
    table_put(T, v3(p), wrap_mode, i);
    T.f0_next[i] = make_float4(p.x, p.y, p.z, __uint_as_float(i));
    T.f1_next[i] = make_float4(d.x, d.y, d.z, g.speed[i]);
    T.f2[i] = make_float4(sd.x, sd.y, sd.z, g.radius[i]);
    T.f3[i] = make_float4(up.x, up.y, up.z, g.mass[i]);
    T.f4[i] = make_float4(g.max_speed[i], g.max_force[i], __uint_as_float(g.applied[i]), 0.f);
    if (dirty) f5[i] = g.steering[i];
}

gs_status table_init(GroupView g, const TableStep& T, int wrap_mode, bool dirty, float4* f5,
                     unsigned* redo_count, cudaStream_t st) {
    launch_after(k_table_init, blocks_for(g.n, 64), 64, 0, st, g, T, wrap_mode, dirty ? 1 : 0, f5, redo_count);
    GS_LAUNCHED("table_init");
    return GS_OK;
}

template <int G, bool FLAT>
static void table_go(const TableStep& T, const StepDev& p, cudaStream_t st, PhaseHook* hook) {
    const unsigned nb = blocks_for(T.n, kTableBlock / G);
    if (hook) hook->mark(2, true);
    if (p.need & NEED_WALLS)
        launch_after(k_table_walls<G, FLAT>, nb, kTableBlock, 0, st, T, p);
    else if ((p.need & kNeedList) == (NEED_SEP | NEED_ALI | NEED_COH))
        launch_after(k_table_step<G, FLAT, NEED_SEP | NEED_ALI | NEED_COH>, nb, kTableBlock, 0, st, T, p);
    else
        launch_after(k_table_step<G, FLAT, kNeedRuntime>, nb, kTableBlock, 0, st, T, p);
    if (hook) hook->mark(2, false);
    if (!(p.need & NEED_WALLS)) return;
    if (hook) hook->mark(3, true);
    if ((p.need & kNeedList) == (NEED_SEP | NEED_AVOID))
        launch_after(k_table_rest<G, NEED_SEP | NEED_AVOID>, nb, kTableBlock, 0, st, T, p);
    else
        launch_after(k_table_rest<G, kNeedRuntime>, nb, kTableBlock, 0, st, T, p);
    if (hook) hook->mark(3, false);
}

gs_status table_step(const TableStep& T, const StepDev& p, cudaStream_t st, PhaseHook* hook) {
    if (T.n == 0) return GS_OK;
    if ((p.need & NEED_WALLS) && p.knw > 8)
        return fail(GS_ERR_UNSUPPORTED, "knw > 8 in the fused step");
    // k <= 8 on 16 lanes while the chip has room for them: the box's 27 counts
    // and its candidates take fewer rounds (4,096 boids 9.7 -> 9.2 us a step)
    const auto go = p.k <= 8 && T.n > 8192 ? (p.flat ? table_go<8, true> : table_go<8, false>)
                    : p.k <= 16            ? (p.flat ? table_go<16, true> : table_go<16, false>)
                                           : (p.flat ? table_go<32, true> : table_go<32, false>);
    go(T, p, st, hook);
    GS_LAUNCHED("table_step");
    return GS_OK;
}

// ---- frame diagnostics (ProcessData.cu:132-237) ----------------------------------------------------
// The counts are the density.  A cell's agents are added in ascending index,
// picked by increasing index.
__global__ void k_table_avg_velocity(const __grid_constant__ TableStep T, float3* __restrict__ out) {
    const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= T.cells) return;
    const unsigned n = T.cnt[c];
    V3 sum = v3(0.f, 0.f, 0.f);
    unsigned last = 0;
    for (unsigned t = 0; t < n; ++t) {
        unsigned next = UINT_MAX;
        for (unsigned s = 0; s < n; ++s) {
            const unsigned id = __float_as_uint(table_entry(T, c, s).w);
            if ((t == 0 || id > last) && id < next) next = id;
        }
        if (next == UINT_MAX) break;
        last = next;
        const float4 h = T.f1_next[next];
        sum = add(sum, mul(v3(h), h.w));
    }
    const V3 avg = n ? dvd(sum, float(n)) : v3(0.f, 0.f, 0.f);
    out[c] = make_float3(avg.x, avg.y, avg.z);
}

gs_status table_avg_velocity(const TableStep& T, float3* out, cudaStream_t st) {
    if (T.cells == 0) return GS_OK;
    k_table_avg_velocity<<<blocks_for(T.cells), kBlock, 0, st>>>(T, out);
    GS_LAUNCHED("cell_avg_velocity");
    return GS_OK;
}

}  // namespace gs
