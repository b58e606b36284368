// Brute-force KNN of large groups (KNNBruteForceCudaKernel.cu:207-283): the k
// nearest of all candidates, found in the cells that can hold them.
//
// One launch sorts the candidates into an automatic grid of about k / 8 a cell
// (gs_db.cu: a sample, the grid and the counting sort in one cluster, nothing
// read back by the host); one gives each query a group of G lanes.  A query
// first takes the 27 cells about its own (then 5^3, 9^3, ... while its list is
// not full), which bounds its k-th distance D.  Every candidate at a distance of
// at most D lies within D of the query on each axis, so in the cells from that
// of q - D to that of q + D: the rest of that box is scanned once more, and the
// list is that over all candidates.  The bound is exact: a distance's rounded
// square is no less than its largest component's, a cell's number grows with
// the coordinate (auto_coords), and D is widened by 1e-5 of itself before q - D
// is rounded down and q + D up.  A query or candidate that is not finite has no
// distance below the largest float to any other, so it is in no list and has
// none.
//
// Instead of every pair (or the 2 % of the bucketed chunks this replaced) a
// query meets about 90 candidates at k = 16.  Crowded cells come down to their
// candidates' squared distances against a rounded-up bound of the k-th distance,
// as k_knn_brute3's filter has it: 262,144 agents in two clusters, 131,000
// candidates a query, 41 ms (70 with every candidate's key made).
#include <cmath>

#include "gs_db.cuh"
#include "gs_lanes.cuh"
#include "gs_launch.h"

namespace gs {

constexpr unsigned kBruteBlock = 256;
constexpr unsigned kBruteSegs = 64;

struct BruteQuery {
    V3 p;
    unsigned self_id;
};

// Takes the candidates of box `out` but not of box `in` (any = false: of none)
// into the list; `on`: this group has a box to take.  segs: the group's
// 2 * kBruteSegs + 1 words of shared memory.  Returns the candidates met by
// this lane.
template <int G, int L>
__device__ __forceinline__ unsigned brute_region(LaneList<G, L>& list, const BruteQuery& q,
                                                 unsigned k, unsigned lane, bool on, const Box& out,
                                                 bool any, const Box& in, const Grid& g,
                                                 const unsigned* start,
                                                 const float4* pos_id,
                                                 unsigned* segs) {
    unsigned* s0s = segs;
    unsigned* pre = segs + kBruteSegs;
    const unsigned nz = out.z1 - out.z0 + 1, sides = any ? 1u : 0u;
    const unsigned ns = on ? ((out.y1 - out.y0 + 1) * nz) << sides : 0u;
    const unsigned most = __reduce_max_sync(kAllLanes, ns);
    unsigned met = 0;
    float bound = prefilter_bound(list.kth(k));
    for (unsigned base = 0; base < most; base += kBruteSegs) {
        // up to kBruteSegs runs of cells, laid end to end: a row each, or two
        // with an inner box, left and right of it where the row crosses it
        const unsigned slots = min(most - base, kBruteSegs);
        unsigned total = 0;
        for (unsigned i = lane; i < slots + lane; i += G) {
            unsigned s0 = 0, len = 0;
            if (base + i < ns && i < slots) {
                const unsigned row = (base + i) >> sides;
                const unsigned y = out.y0 + row / nz, z = out.z0 + row % nz;
                const bool cross = any && y >= in.y0 && y <= in.y1 && z >= in.z0 && z <= in.z1;
                unsigned x0 = out.x0, x1 = out.x1 + 1;  // [x0, x1)
                if ((base + i) & sides) x0 = cross ? in.x1 + 1 : x1;
                else if (cross) x1 = in.x0;
                if (x0 < x1) {
                    const unsigned c = cell_label(g, x0, y, z);
                    s0 = start[c];
                    len = start[c + (x1 - x0)] - s0;
                }
            }
            unsigned sum = len;
#pragma unroll
            for (int o = 1; o < G; o <<= 1) {
                const unsigned v = __shfl_up_sync(kAllLanes, sum, o, G);
                if (lane >= unsigned(o)) sum += v;
            }
            if (i < slots) {
                s0s[i] = s0;
                pre[i] = total + sum - len;
            }
            total += __shfl_sync(kAllLanes, sum, G - 1, G);
        }
        if (lane == 0) pre[slots] = total;
        __syncwarp();
        const unsigned rounds = __reduce_max_sync(kAllLanes, total);
        // the next candidate is on its way while this one is taken
        unsigned at = 0;
        auto load = [&](unsigned j) {
            if (j >= total) return make_float4(0.f, 0.f, 0.f, 0.f);
            while (j >= pre[at + 1]) ++at;
            return pos_id[s0s[at] + (j - pre[at])];
        };
        float4 v = load(lane);
        for (unsigned j = lane; j < rounds + lane; j += G) {
            const float4 next = load(j + G);
            const V3 o = sub(q.p, v3(v));
            const float dsq = dot(o, o);
            const unsigned id = __float_as_uint(v.w);
            const bool near = j < total && dsq <= bound && id != q.self_id;
            met += j < total;
            v = next;
            if (!__any_sync(kAllLanes, near)) continue;
            const unsigned long long key = knn_key(sqrtf(dsq), id);
            list.take(near && key < KEY_EMPTY ? key : KEY_EMPTY, k, lane);
            bound = prefilter_bound(list.kth(k));
        }
        __syncwarp();
    }
    return met;
}

// q_pos: the queries, position and (by_slot) agent index; the index is the
// query's place otherwise.
template <int G, int L>
__global__ void __launch_bounds__(kBruteBlock) k_brute_cells(
    const float4* q_pos, bool by_slot, unsigned nA, const float4* pos_id,
    const unsigned* start, const AutoGrid* grid, bool self, unsigned k,
    unsigned long long* evaluated, unsigned* idx,
    float* dist) {
    after_previous();
    __shared__ unsigned sh[kBruteBlock / G * (2 * kBruteSegs + 1)];
    __shared__ unsigned met_sh[kBruteBlock / 32];
    unsigned* segs = sh + threadIdx.x / G * (2 * kBruteSegs + 1);
    const unsigned lane = threadIdx.x & unsigned(G - 1);
    const unsigned s = (blockIdx.x * kBruteBlock + threadIdx.x) / G;
    const bool act = s < nA;  // spare groups run along with nothing to take
    const float4 v = q_pos[act ? s : nA - 1];
    const unsigned a = by_slot ? __float_as_uint(v.w) : s;
    const BruteQuery q{v3(v), self ? a : UINT_MAX};
    const AutoGrid ag = *grid;
    const Grid& g = ag.grid;
    const bool live = act && is_finite(q.p);
    LaneList<G, L> list;
#pragma unroll
    for (int h = 0; h < L; ++h) list.e[h] = KEY_EMPTY;
    unsigned ix, iy, iz;
    auto_coords(ag, q.p, ix, iy, iz);
    Box out = cell_box(g, ix, iy, iz, 1), done = out;  // to take now; taken so far
    bool any = false, on = live, last = false;
    unsigned met = 0;
    for (unsigned r = 2;; r = 2 * r) {
        met += brute_region(list, q, k, lane, on, out, any, done, g, start, pos_id, segs);
        if (last) break;
        any = true;
        if (on) done = out;
        const unsigned long long kth = list.kth(k);
        const bool whole = done.x0 == 0 && done.y0 == 0 && done.z0 == 0 &&
                           done.x1 == g.wc[0] - 1 && done.y1 == g.wc[1] - 1 &&
                           done.z1 == g.wc[2] - 1;
        on = live && !whole && kth >= KEY_EMPTY;
        if (__any_sync(kAllLanes, on)) {
            if (on) out = cell_box(g, ix, iy, iz, r);
            continue;
        }
        // the rest of the box that can hold a candidate at the k-th distance
        const float reach = __fadd_ru(__fmul_ru(key_dist(kth), 1.00001f), 1e-18f);
        unsigned lx, ly, lz, ux, uy, uz;
        auto_coords(ag, v3(__fsub_rd(q.p.x, reach), __fsub_rd(q.p.y, reach),
                           __fsub_rd(q.p.z, reach)), lx, ly, lz);
        auto_coords(ag, v3(__fadd_ru(q.p.x, reach), __fadd_ru(q.p.y, reach),
                           __fadd_ru(q.p.z, reach)), ux, uy, uz);
        out = Box{min(lx, done.x0), max(ux, done.x1), min(ly, done.y0),
                  max(uy, done.y1), min(lz, done.z0), max(uz, done.z1)};
        on = live;
        last = true;
    }
    if (act) {
#pragma unroll
        for (int h = 0; h < L; ++h) {
            const unsigned rank = 32u * h + lane;
            if (rank < k) {
                idx[a + size_t(rank) * nA] = key_id(list.e[h]);
                dist[a + size_t(rank) * nA] = key_dist(list.e[h]);
            }
        }
    }
    const unsigned w = __reduce_add_sync(kAllLanes, met);
    if ((threadIdx.x & 31u) == 0) met_sh[threadIdx.x >> 5] = w;
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long sum = 0;
        for (unsigned i = 0; i < kBruteBlock / 32; ++i) sum += met_sh[i];
        atomicAdd(evaluated, sum);
    }
}

template <int G, int L>
static void brute_go(const float4* q_pos, bool by_slot, unsigned nA, const Database& B,
                     const BruteWork& w, bool self, unsigned k, unsigned* idx, float* dist,
                     cudaStream_t st) {
    launch_after(k_brute_cells<G, L>, blocks_for(nA, kBruteBlock / G), kBruteBlock, 0, st, q_pos, by_slot, nA, B.pos_id, B.start, w.grid, self, k, w.evaluated, idx, dist);
}

// k / 8 candidates a cell: the 27 cells then hold about 3.4 k, 8 of them (a
// corner of the grid) about k.
unsigned brute_cells(unsigned n, unsigned k) {
    const double per = std::fmin(std::fmax(k / 8.0, 0.5), 5.0), c = n / per;
    return c > 1.0 ? unsigned(std::fmin(c, double(1u << 24))) : 1u;
}

gs_status launch_knn_brute_cells(const float4* posA, unsigned nA, const float4* posB, unsigned nB,
                                 bool self, unsigned k, Database& B, const BruteWork& w,
                                 unsigned* idx, float* dist, cudaStream_t st) {
    if (nA == 0) return GS_OK;
    if (k == 0 || k > 64 || nB == 0)
        return fail(GS_ERR_UNSUPPORTED, "brute force over cells needs 1 <= k <= 64");
    DbJobs J;
    J.job[0] = db_job(B, posB, nB, Grid{});
    // per axis, so that the cells are at most brute_cells(nB, k)
    const double most = double(brute_cells(nB, k));
    for (int a = 0; a < 3; ++a) {
        unsigned c = unsigned(std::floor(std::pow(most, 1.0 / (a + 1)) + 1e-9));
        while (c > 1 && std::pow(double(c), a + 1) > most) --c;
        J.job[0].auto_axis[a] = c ? c : 1u;
    }
    J.job[0].grid_out = w.grid;
    J.job[0].zero = w.evaluated;
    GS_TRY(db_build_clusters(J, 1, st));
    const float4* q = self ? B.pos_id : posA;
    if (k <= 8) brute_go<8, 1>(q, self, nA, B, w, self, k, idx, dist, st);
    else if (k <= 16) brute_go<16, 1>(q, self, nA, B, w, self, k, idx, dist, st);
    else if (k <= 32) brute_go<32, 1>(q, self, nA, B, w, self, k, idx, dist, st);
    else brute_go<32, 2>(q, self, nA, B, w, self, k, idx, dist, st);
    GS_LAUNCHED("knn_brute_cells");
    return GS_OK;
}

}  // namespace gs
