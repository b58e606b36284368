// An agent's neighbour search and neighbour pass spread over a group of G
// lanes (8, 16 or 32; k <= G): lane r of the group ends up with the agent's
// r-th neighbour.
//
// With one thread per agent a small group leaves most SMs empty and its step
// takes as long as one thread's serial chain: the box's candidates one after
// another into a k-list, then k dependent neighbour gathers.  A lane group
// takes G candidates at a time and gathers all k neighbours at once, so the
// chain is a few rounds long and a few thousand agents fill the chip.  It
// costs more issue slots per agent (the list lives across lanes and every
// merge is shuffles), so large groups keep one thread per agent.
//
// Every key is exact, (distance bits, agent index), so no candidate order is
// left open and nothing is redone.  All lanes of a warp run the same number
// of rounds (the busiest group's), so every shuffle is warp-converged.
#pragma once

#include "gs_behaviours.cuh"
#include "gs_knn.cuh"
#include "gs_launch.h"

namespace gs {

constexpr unsigned kAllLanes = 0xffffffffu;

template <int G>
struct LaneEntry {
    unsigned long long key;  // (distance bits, agent index), KEY_EMPTY for none
    unsigned slot;           // the neighbour's slot, UINT_MAX for none

    // Keeps the smaller (keep_min) or larger of this entry and the one
    // `stride` lanes away.  Keys are unique but for KEY_EMPTY, whose slot is
    // the same everywhere.
    __device__ __forceinline__ void exchange(int stride, bool keep_min) {
        const unsigned long long ok = __shfl_xor_sync(kAllLanes, key, stride);
        const unsigned os = __shfl_xor_sync(kAllLanes, slot, stride);
        if ((ok < key) == keep_min) {
            key = ok;
            slot = os;
        }
    }
    // Ascending bitonic sort over the group's lanes.
    __device__ __forceinline__ void sort(unsigned lane) {
#pragma unroll
        for (int size = 2; size <= G; size <<= 1) {
#pragma unroll
            for (int stride = size >> 1; stride > 0; stride >>= 1)
                exchange(stride, ((lane & unsigned(stride)) == 0) == ((lane & unsigned(size)) == 0));
        }
    }
    // Merges the group's sorted chunk c into this sorted list, keeping the G
    // smallest: laid reversed against the list, the elementwise minima are
    // bitonic and hold them; log2(G) half-cleaners sort them again.
    __device__ __forceinline__ void merge(const LaneEntry& c, unsigned lane) {
        const unsigned long long rk = __shfl_xor_sync(kAllLanes, c.key, G - 1);
        const unsigned rs = __shfl_xor_sync(kAllLanes, c.slot, G - 1);
        if (rk < key) {
            key = rk;
            slot = rs;
        }
#pragma unroll
        for (int stride = G >> 1; stride > 0; stride >>= 1)
            exchange(stride, (lane & unsigned(stride)) == 0);
    }
};

// Takes one candidate per lane (c; KEY_EMPTY for none) into the list.
// `first`: the list is still empty.  Warp-converged; a chunk with nothing
// below any group's k-th key is dropped after one vote.
template <int G>
__device__ __forceinline__ void lanes_take(LaneEntry<G>& list, LaneEntry<G> c, bool first,
                                           unsigned k, unsigned lane) {
    if (first) {
        c.sort(lane);
        list = c;
        return;
    }
    const unsigned long long kth = __shfl_sync(kAllLanes, list.key, int(k) - 1, G);
    if (!__any_sync(kAllLanes, c.key < kth)) return;
    c.sort(lane);
    list.merge(c, lane);
}

template <int G>
__device__ __forceinline__ LaneEntry<G> lanes_candidate(V3 p, unsigned self_id, float4 q,
                                                        unsigned slot, bool ok) {
    LaneEntry<G> c{KEY_EMPTY, UINT_MAX};
    const unsigned id = __float_as_uint(q.w);
    const unsigned long long kk = knn_key(distance(p, v3(q)), id);
    if (ok && id != self_id && kk < KEY_EMPTY) {
        c.key = kk;
        c.slot = slot;
    }
    return c;
}

// Calls take(q, slot, ok, first) for the candidates of box b, one per lane of the
// group at a time, in warp-converged rounds (ok: this lane has one; first: the
// first round).
// R: rows of cells in the box at search radius 1 (9, or 3 on a grid one cell
// high in y); 0 for any radius.  The rows are laid end to end, so a group
// takes ceil(candidates / G) chunks whatever the rows' lengths; with R = 0
// their table is the group's kLaneRowWords words `rows` of shared memory, and
// a box of more than kLaneRows rows is taken row by row.
constexpr unsigned kLaneRows = 64, kLaneRowWords = 2 * kLaneRows + 1;
template <int G, int R, class Take>
__device__ __forceinline__ void lanes_box(unsigned lane, const Grid& g, const Box& b,
                                          unsigned cell_offset, const unsigned* start,
                                          const float4* pos_id, unsigned* rows, Take&& take) {
    const unsigned span = b.x1 - b.x0 + 1;
    if constexpr (R > 0) {
        constexpr int Q = (R + G - 1) / G;
        unsigned s0[Q], len[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const unsigned i = lane + unsigned(q * G);
            const unsigned cy = b.y0 + (R == 3 ? 0u : i / 3u), cz = b.z0 + (R == 3 ? i : i % 3u);
            s0[q] = len[q] = 0;
            if (i < unsigned(R) && cy <= b.y1 && cz <= b.z1) {
                const unsigned c0 = cell_offset + cell_label(g, b.x0, cy, cz);
                s0[q] = start[c0];
                len[q] = start[c0 + span] - s0[q];
            }
        }
        unsigned rs[R], pre[R + 1];
        pre[0] = 0;
#pragma unroll
        for (int i = 0; i < R; ++i) {
            rs[i] = __shfl_sync(kAllLanes, s0[i / G], i % G, G);
            pre[i + 1] = pre[i] + __shfl_sync(kAllLanes, len[i / G], i % G, G);
        }
        const unsigned total = pre[R], rounds = __reduce_max_sync(kAllLanes, total);
        auto at = [&](unsigned j) {
            unsigned s = rs[0] + j;
#pragma unroll
            for (int i = 1; i < R; ++i)
                if (j >= pre[i]) s = rs[i] + (j - pre[i]);
            return s;
        };
        // the next chunk's position is on its way while this one is sorted in
        unsigned sl = at(lane);
        float4 q = lane < total ? pos_id[sl] : make_float4(0.f, 0.f, 0.f, 0.f);
        for (unsigned j0 = 0; j0 < rounds; j0 += G) {
            const unsigned j = j0 + lane, jn = j + G;
            const unsigned sn = at(jn);
            const float4 qn = jn < total ? pos_id[sn] : make_float4(0.f, 0.f, 0.f, 0.f);
            take(q, sl, j < total, j0 == 0);
            sl = sn;
            q = qn;
        }
    } else {
        // (an empty box has y1 < y0)
        const unsigned nz = b.z1 - b.z0 + 1;
        const unsigned nr = b.y1 >= b.y0 ? (b.y1 - b.y0 + 1) * nz : 0u;
        const unsigned most = __reduce_max_sync(kAllLanes, nr);
        auto row = [&](unsigned i, unsigned& s0) {
            const unsigned c0 = cell_offset + cell_label(g, b.x0, b.y0 + i / nz, b.z0 + i % nz);
            s0 = start[c0];
            return start[c0 + span] - s0;
        };
        if (most <= kLaneRows) {
            unsigned* rs = rows;
            unsigned* pre = rows + kLaneRows;
            unsigned total = 0;
            for (unsigned i = lane; i < most + lane; i += G) {
                unsigned s0 = 0, len = i < nr ? row(i, s0) : 0u;
                unsigned sum = len;
#pragma unroll
                for (int o = 1; o < G; o <<= 1) {
                    const unsigned y = __shfl_up_sync(kAllLanes, sum, o, G);
                    if (lane >= unsigned(o)) sum += y;
                }
                if (i < nr) {
                    rs[i] = s0;
                    pre[i] = total + sum - len;
                }
                total += __shfl_sync(kAllLanes, sum, G - 1, G);
            }
            if (lane == 0) pre[nr] = total;
            __syncwarp();
            const unsigned rounds = __reduce_max_sync(kAllLanes, total);
            unsigned at = 0;
            for (unsigned j = lane; j < rounds + lane; j += G) {
                const bool ok = j < total;
                unsigned sl = 0;
                if (ok) {
                    while (j >= pre[at + 1]) ++at;
                    sl = rs[at] + (j - pre[at]);
                }
                const float4 q = ok ? pos_id[sl] : make_float4(0.f, 0.f, 0.f, 0.f);
                take(q, sl, ok, j < G);
            }
            __syncwarp();  // the rows may be written again
        } else {
            bool first = true;
            for (unsigned i = 0; i < most; ++i) {
                unsigned s0 = 0;
                const unsigned len = i < nr ? row(i, s0) : 0u;
                const unsigned rounds = __reduce_max_sync(kAllLanes, len);
                for (unsigned j = lane; j < rounds + lane; j += G) {
                    const float4 q =
                        j < len ? pos_id[s0 + j] : make_float4(0.f, 0.f, 0.f, 0.f);
                    take(q, s0 + j, j < len, first);
                    first = false;
                }
            }
        }
    }
}

// The k nearest of the box around cell (ix, iy, iz), in (distance, index)
// order over the group's lanes: lane r holds rank r (ranks past the last
// neighbour hold the empty entry; lanes r >= k hold leftovers).
template <int G, int R>
__device__ __forceinline__ LaneEntry<G> lanes_knn(unsigned k, unsigned lane, V3 p,
                                                  unsigned self_id, const Grid& g, const Box& b,
                                                  unsigned cell_offset,
                                                  const unsigned* start,
                                                  const float4* pos_id,
                                                  unsigned* rows = nullptr) {
    LaneEntry<G> list{KEY_EMPTY, UINT_MAX};
    lanes_box<G, R>(lane, g, b, cell_offset, start, pos_id, rows,
                    [&](float4 q, unsigned slot, bool ok, bool first) {
                        lanes_take(list, lanes_candidate<G>(p, self_id, q, slot, ok), first, k, lane);
                    });
    return list;
}

// This group's bits of a warp vote, lane 0 of the group in bit 0.
template <int G>
__device__ __forceinline__ unsigned lanes_ballot(bool pred) {
    const unsigned all = __ballot_sync(kAllLanes, pred);
    if (G == 32) return all;
    return (all >> (threadIdx.x & 31u & ~unsigned(G - 1))) & ((1u << (G & 31)) - 1u);
}
template <int G>
__device__ __forceinline__ V3 lanes_get(V3 v, unsigned from) {
    return v3(__shfl_sync(kAllLanes, v.x, int(from), G), __shfl_sync(kAllLanes, v.y, int(from), G),
              __shfl_sync(kAllLanes, v.z, int(from), G));
}

// A query's exact (distance, index) list over its group's lanes: lane r holds
// rank r in e[0] and, with L = 2 (32 < k <= 64, G = 32), rank 32 + r in e[1].
template <int G, int L>
struct LaneList {
    unsigned long long e[L];

    __device__ __forceinline__ unsigned long long kth(unsigned k) const {
        if (L == 1 || k <= 32) return __shfl_sync(kAllLanes, e[0], int(k) - 1, G);
        return __shfl_sync(kAllLanes, e[L - 1], int(k) - 33, G);
    }
    __device__ __forceinline__ static unsigned long long pick(unsigned long long a, int stride,
                                                              bool keep_min) {
        const unsigned long long b = __shfl_xor_sync(kAllLanes, a, stride);
        return (b < a) == keep_min ? b : a;
    }
    // One candidate key per lane (KEY_EMPTY for none).  A few that enter are
    // shifted in one after another; more are sorted and merged at once.
    __device__ __forceinline__ void take(unsigned long long c, unsigned k, unsigned lane) {
        const bool in = c < kth(k);
        if (!__any_sync(kAllLanes, in)) return;
        unsigned m = lanes_ballot<G>(in);
        unsigned most = __reduce_max_sync(kAllLanes, unsigned(__popc(m)));
        if (most <= 4) {
            for (; most; --most) {
                const int from = m ? __ffs(int(m)) - 1 : 0;
                unsigned long long key = __shfl_sync(kAllLanes, c, from, G);
                if (!m) key = KEY_EMPTY;
                m &= m - 1u;
                const unsigned long long up = __shfl_up_sync(kAllLanes, e[0], 1, G);
                if (L == 2) {
                    unsigned long long up1 = __shfl_up_sync(kAllLanes, e[L - 1], 1, G);
                    const unsigned long long last = __shfl_sync(kAllLanes, e[0], G - 1, G);
                    if (lane == 0) up1 = last;
                    if (key < e[L - 1]) e[L - 1] = up1 > key ? up1 : key;
                }
                if (key < e[0]) e[0] = (lane && up > key) ? up : key;
            }
            return;
        }
#pragma unroll
        for (int size = 2; size <= G; size <<= 1) {
#pragma unroll
            for (int stride = size >> 1; stride > 0; stride >>= 1)
                c = pick(c, stride,
                         ((lane & unsigned(stride)) == 0) == ((lane & unsigned(size)) == 0));
        }
        const unsigned long long r = __shfl_xor_sync(kAllLanes, c, G - 1);
        if (r < e[L - 1]) e[L - 1] = r;
        if (L == 2 && e[L - 1] < e[0]) {
            const unsigned long long x = e[0];
            e[0] = e[L - 1];
            e[L - 1] = x;
        }
#pragma unroll
        for (int h = 0; h < L; ++h)
#pragma unroll
            for (int stride = G >> 1; stride > 0; stride >>= 1)
                e[h] = pick(e[h], stride, (lane & unsigned(stride)) == 0);
    }
};

// One value per lane of a group summed in lane order, for up to 9 value
// columns at once: each column is a row of shared memory and one lane adds
// up one row from 0, as the reference's loop over the list does (a lane that
// is not in the sum holds +0, which changes no partial sum: those start at
// +0 and never become -0).  Rows are padded to G + 4 words, so eight lanes'
// 16-byte reads of eight rows meet no bank twice.
template <int G>
struct LaneSums {
    static constexpr unsigned kRow = G + 4;
    static constexpr unsigned kWords = 9 * kRow + 12;
    float* w;  // this group's kWords words, 16-byte aligned
    __device__ __forceinline__ static LaneSums of(float* shared) {
        return LaneSums{shared + threadIdx.x / G * kWords};
    }
    __device__ __forceinline__ void put(unsigned first, unsigned lane, V3 v) {
        w[first * kRow + lane] = v.x;
        w[(first + 1) * kRow + lane] = v.y;
        w[(first + 2) * kRow + lane] = v.z;
    }
    __device__ __forceinline__ void add_rows(unsigned lane) {
        __syncwarp();
        for (unsigned c = lane; c < 9; c += G) {
            const float4* row = reinterpret_cast<const float4*>(w + c * kRow);
            float s = 0.f;
#pragma unroll
            for (int i = 0; i < G / 4; ++i) {
                const float4 v = row[i];
                s = s + v.x;
                s = s + v.y;
                s = s + v.z;
                s = s + v.w;
            }
            w[9 * kRow + c] = s;
        }
        __syncwarp();
    }
    __device__ __forceinline__ V3 sum(unsigned first) const {
        return v3(w[9 * kRow + first], w[9 * kRow + first + 1], w[9 * kRow + first + 2]);
    }
};

// ---- the neighbour pass over lanes -----------------------------------------------------
// Lane r's neighbour (rank r of the list): ok when there is one; `dist` is its
// KNN distance.  Each lane evaluates its neighbour's terms with the
// reference's expressions; what the reference does in list order happens in
// lane order.
struct LaneNeighbour {
    bool ok;
    V3 pos, dir;
    float speed, radius, dist;
};

// The weighted separation, alignment and cohesion vectors (flock_finish up to
// its mask test) of the behaviours in `need`; the others' are left unset.
template <bool FLAT = false, int G = 32>
__device__ __forceinline__ void lanes_flock(unsigned need, const FlockParams& fs,
                                            const FlockParams& fa, const FlockParams& fc,
                                            const Self& me, unsigned lane,
                                            const LaneNeighbour& nb, LaneSums<G> sums, V3& r_sep,
                                            V3& r_ali, V3& r_coh) {
    if (!(need & (NEED_SEP | NEED_ALI | NEED_COH))) return;
    const V3 zero = v3(0.f, 0.f, 0.f);
    const V3 offset = sub(nb.pos, me.pos);
    const float dsq = dot(offset, offset), d = sqrtf(dsq);
    const float ahead = dot(me.dir, dvd<FLAT>(offset, d));
    auto member = [&](const FlockParams& f) {  // inBoidNeighborhood, FlockingCommon.cuh:4-30
        return nb.ok && (d < f.min_d || (!(d > f.max_d) && ahead > f.cos_max));
    };
    unsigned n_sep = 0, n_ali = 0, n_coh = 0;
    if (need & NEED_SEP) {
        const bool in = member(fs);
        n_sep = __popc(lanes_ballot<G>(in));
        sums.put(0, lane, in ? dvd<FLAT>(offset, -dsq) : zero);
    }
    if (need & NEED_ALI) {
        const bool in = member(fa);
        n_ali = __popc(lanes_ballot<G>(in));
        sums.put(3, lane, in ? nb.dir : zero);
    }
    if (need & NEED_COH) {
        const bool in = member(fc);
        n_coh = __popc(lanes_ballot<G>(in));
        sums.put(6, lane, in ? nb.pos : zero);
    }
    sums.add_rows(lane);
    // lanes 0, 1, 2: the three behaviours' finish side by side
    const unsigned kind = lane < 2 ? lane : 2u;
    const unsigned n = kind == 0 ? n_sep : kind == 1 ? n_ali : n_coh;
    const float w = kind == 0 ? fs.w : kind == 1 ? fa.w : fc.w;
    V3 r = zero;
    if (n) {
        const V3 mean = dvd<FLAT>(sums.sum(3 * kind), float(n));
        r = normalize<FLAT>(kind == 0 ? mean : sub(mean, kind == 1 ? me.dir : me.pos));
    }
    r = mul(r, w);
    if (need & NEED_SEP) r_sep = lanes_get<G>(r, 0);
    if (need & NEED_ALI) r_ali = lanes_get<G>(r, 1);
    if (need & NEED_COH) r_coh = lanes_get<G>(r, 2);
    __syncwarp();  // the sums may be written again
}
// The rest of flock_finish.
__device__ __forceinline__ void flock_apply(V3 r, const FlockParams& f, unsigned bit,
                                            unsigned& applied, V3& steer) {
    if (applied & f.mask) return;
    if (!is_zero(r)) applied |= bit;
    steer = add(r, steer);
}

// close_add over the list: its first hit.
template <int G>
__device__ __forceinline__ CloseAcc lanes_close(const Self& me, float min_sep,
                                                const LaneNeighbour& nb) {
    CloseAcc c;
    close_init(c);
    if (nb.ok) close_add(c, me, min_sep, nb.dist, nb.pos, nb.radius);
    const unsigned m = lanes_ballot<G>(c.found);
    const V3 s = lanes_get<G>(c.steer, m ? unsigned(__ffs(int(m)) - 1) : 0u);
    c.found = m != 0;
    c.steer = m ? s : v3(0.f, 0.f, 0.f);
    return c;
}

// avoid_add over the list: every lane its neighbour's approach time and
// distance, then the reference's pass over them, whose window [0, min_t) only
// narrows (`at` keeps the last neighbour in it, threat or not).
template <int G, bool FLAT = false>
__device__ __forceinline__ AvoidAcc lanes_avoid(const Self& me, float min_time, unsigned k,
                                                const LaneNeighbour& nb) {
    AvoidAcc a;
    avoid_init(a, min_time);
    V3 at = v3(0.f, 0.f, 0.f);
    float t = __int_as_float(0x7f800000);
    bool danger = false;
    if (nb.ok) {
        const float time =
            nearest_approach_time<FLAT>(me.pos, me.dir, me.speed, nb.pos, nb.dir, nb.speed);
        if (time >= 0.f) t = time;
        danger = nearest_approach_positions(me.pos, me.dir, me.speed, nb.pos, nb.dir, nb.speed,
                                            time, at) < me.radius + nb.radius;
    }
    const unsigned hits = lanes_ballot<G>(danger);
    unsigned last = UINT_MAX;
    for (unsigned r = 0; r < k; ++r) {
        const float tr = __shfl_sync(kAllLanes, t, int(r), G);
        if (tr < a.min_t) {
            last = r;
            if ((hits >> r) & 1u) {
                a.min_t = tr;
                a.threat = r;
            }
        }
    }
    const unsigned lf = last == UINT_MAX ? 0u : last, tf = a.threat == UINT_MAX ? 0u : a.threat;
    const V3 la = lanes_get<G>(at, lf), tp = lanes_get<G>(nb.pos, tf),
             td = lanes_get<G>(nb.dir, tf);
    const float ts = __shfl_sync(kAllLanes, nb.speed, int(tf), G);
    if (last != UINT_MAX) a.threat_at = la;
    if (a.threat != UINT_MAX) {
        a.threat_pos = tp;
        a.threat_dir = td;
        a.threat_speed = ts;
    }
    return a;
}

// The behaviours order[first..] of one agent over its lanes' neighbours.
template <int G, bool FLAT>
__device__ __forceinline__ void lanes_behaviours(const StepDev& p, unsigned need, unsigned first,
                                                 const Self& me, unsigned lane,
                                                 const LaneNeighbour& nb, LaneSums<G> sums,
                                                 unsigned& applied, V3& steer) {
    const FlockParams fs = flock_params(p.sep, p.sep_dsq), fa = flock_params(p.ali, p.ali_dsq),
                      fc = flock_params(p.coh, p.coh_dsq);
    V3 r_sep, r_ali, r_coh;
    lanes_flock<FLAT>(need, fs, fa, fc, me, lane, nb, sums, r_sep, r_ali, r_coh);
    CloseAcc close;
    AvoidAcc avoid;
    if (need & NEED_CLOSE) close = lanes_close<G>(me, p.min_sep, nb);
    if (need & NEED_AVOID) avoid = lanes_avoid<G, FLAT>(me, p.min_time_col, p.k, nb);
#pragma unroll 1
    for (unsigned o = first; o < p.n_order; ++o) {
        switch ((p.order_packed >> (3u * o)) & 7u) {
            case GS_B_SEPARATION:
                if (need & NEED_SEP) flock_apply(r_sep, fs, SEPARATION_BIT, applied, steer);
                break;
            case GS_B_ALIGNMENT:
                if (need & NEED_ALI) flock_apply(r_ali, fa, ALIGNMENT_BIT, applied, steer);
                break;
            case GS_B_COHESION:
                if (need & NEED_COH) flock_apply(r_coh, fc, COHESION_BIT, applied, steer);
                break;
            case GS_B_SEEK:
                seek_finish<FLAT>(v3(p.seek_target[0], p.seek_target[1], p.seek_target[2]), p.w_seek,
                                  p.mask_seek, me, applied, steer);
                break;
            case GS_B_AVOID_NEIGHBORS:
                if (need & NEED_AVOID) {
                    if (need & NEED_CLOSE)
                        close_finish<FLAT>(close, p.w_avoid, p.mask_avoid, applied, steer);
                    avoid_finish<FLAT>(avoid, p.w_avoid, p.mask_avoid, me, applied, steer);
                }
                break;
            case GS_B_FOLLOW_PATH:
                follow_path_finish(p.path, p.path_time, p.w_path, p.mask_path, me, applied, steer);
                break;
            default: break;
        }
    }
}

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

// Avoid-walls for one agent (its box: that of its KNN): the nearest walls'
// list, then their lines in order; may move the agent.
template <int G, int R>
__device__ __forceinline__ void lanes_walls(const WallRefs& W, const Scene& sc, const StepDev& p,
                                            Self& me, unsigned lane, const Box& box,
                                            unsigned& applied, V3& steer,
                                            unsigned* rows = nullptr) {
    const bool walls = sc.n_walls > 0 && W.pos_id != nullptr;
    if (__any_sync(kAllLanes, walls)) {
        Box wb = box;
        if (!walls) {  // a scene without walls searches an empty box
            wb.y0 = 1;
            wb.y1 = 0;
        }
        const LaneEntry<G> wl =
            lanes_knn<G, R>(p.knw, lane, me.pos, UINT_MAX, sc.grid, wb, sc.wall_cell_offset,
                            W.cell_start, W.pos_id, rows);
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
            lanes_wall_line<G>(wa, me, lane, line, on, v3(W.start[g]), v3(W.end[g]),
                               v3(W.normal[g]));
        }
        if (walls) walls_finish(wa, p.w_walls, p.mask_walls, me, applied, steer);
        else if (!(applied & p.mask_walls)) steer = add(mul(v3(0.f, 0.f, 0.f), p.w_walls), steer);
    } else if (!(applied & p.mask_walls)) {
        steer = add(mul(v3(0.f, 0.f, 0.f), p.w_walls), steer);
    }
}

}  // namespace gs
