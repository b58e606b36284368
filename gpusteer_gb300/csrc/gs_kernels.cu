// Counting-sort binning and the per-function (drop-in) kernels.
//
// The bin rebuild replaces KNNBinningV2UpdateDBCUDA::run (KNNBinningV2.cu:87-162:
// BuildDB, a host synchronisation, thrust::sort_by_key, a memset of every cell
// and ReorderDB) with three passes that never leave the device: an atomic
// count per cell (which also hands each agent its rank inside the cell), an
// exclusive scan of the counts, and a scatter of (position, index) into
// bucketed order.  The order inside a cell follows the atomics and is not
// deterministic; nothing downstream depends on it because every KNN uses the
// total order (distance, agent index).
#include <algorithm>
#include <atomic>
#include <cstring>

#include "gs_behaviours.cuh"
#include "gs_db.cuh"
#include "gs_knn.cuh"
#include "gs_scan.cuh"

#include "gs_launch.h"

namespace gs {

unsigned sm_count() {
    static std::atomic<int> known[64];
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 1;
    if ((sms = known[dev].load(std::memory_order_relaxed)) > 0) return unsigned(sms);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return 1;
    known[dev].store(sms, std::memory_order_relaxed);
    return unsigned(sms);
}

// ---- exclusive scan (device code in gs_scan.cuh) ----------------------------------
unsigned scan_tile_count(unsigned C) { return (C + kScanTile - 1) / kScanTile; }

__global__ void __launch_bounds__(kBlock) k_scan_reduce(const unsigned* count,
                                                        unsigned C, unsigned* tile) {
    after_previous();
    __shared__ unsigned sh[kScanTile + kScanTile / 32];
    __shared__ unsigned ws[kBlock / 32];
    scan_reduce_tile(count, C, blockIdx.x, sh, ws, tile);
}

// One block scans the tile totals in place (exclusive) and writes start[C].
__global__ void __launch_bounds__(1024) k_scan_tiles(unsigned* tile, unsigned T,
                                                     unsigned* start, unsigned C) {
    after_previous();
    __shared__ unsigned ws[32];
    __shared__ unsigned carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (unsigned base = 0; base < T; base += 1024) {
        const unsigned i = base + threadIdx.x;
        const unsigned v = i < T ? tile[i] : 0u;
        const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        unsigned x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= unsigned(o)) x += y;
        }
        if (lane == 31) ws[warp] = x;
        __syncthreads();
        if (warp == 0) {
            unsigned w = ws[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const unsigned y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= unsigned(o)) w += y;
            }
            ws[lane] = w;
        }
        __syncthreads();
        const unsigned before = (warp ? ws[warp - 1] : 0u) + carry;
        if (i < T) tile[i] = before + x - v;
        __syncthreads();
        if (threadIdx.x == 1023) carry = before + x;
        __syncthreads();
    }
    if (threadIdx.x == 0) start[C] = carry;
}

__global__ void __launch_bounds__(kBlock) k_scan_apply(unsigned* count, unsigned C,
                                                       const unsigned* tile,
                                                       unsigned* start) {
    after_previous();
    __shared__ unsigned sh[kScanTile + kScanTile / 32];
    __shared__ unsigned ws[kBlock / 32];
    unsigned items[kScanItems];
    load_tile(count, C, blockIdx.x, sh, items);
    unsigned s = 0;
#pragma unroll
    for (unsigned j = 0; j < kScanItems; ++j) s += items[j];
    unsigned total;
    unsigned run = block_exclusive_sum(s, ws, total) + tile[blockIdx.x];
#pragma unroll
    for (unsigned j = 0; j < kScanItems; ++j) {
        const unsigned i = threadIdx.x * kScanItems + j;
        sh[i + i / 32] = run;
        run += items[j];
    }
    __syncthreads();
    const unsigned base = blockIdx.x * kScanTile;
#pragma unroll
    for (unsigned j = 0; j < kScanItems; ++j) {
        const unsigned i = j * kBlock + threadIdx.x;
        if (base + i < C) {
            start[base + i] = sh[i + i / 32];
            count[base + i] = 0u;
        }
    }
}

gs_status scan_counts(unsigned* count, unsigned* start, unsigned C, unsigned* tile,
                      cudaStream_t st) {
    const unsigned T = scan_tile_count(C);
    launch_after(k_scan_reduce, T, kBlock, 0, st, count, C, tile);
    launch_after(k_scan_tiles, 1, 1024, 0, st, tile, T, start, C);
    launch_after(k_scan_apply, T, kBlock, 0, st, count, C, tile, start);
    GS_LAUNCHED("scan");
    return GS_OK;
}

// ---- the fused engine's counting-sort scan: one launch, tiles near agents ---------
// The step's counting atomics add each tile's total as they go, so no reduce
// pass reads the counts (only a whole recount, from the reference layout or
// on a new grid, takes one); every block sums the totals of the tiles before its own (a
// few thousand words from L2) and writes its tile's starts, and no block
// waits on another (scan_apply_sparse_tile).
__global__ void __launch_bounds__(kBlock) k_scan_apply_sparse(unsigned* count,
                                                              unsigned C,
                                                              const unsigned* tile,
                                                              unsigned* start,
                                                              unsigned T, unsigned reach,
                                                              unsigned* live) {
    after_previous();
    __shared__ unsigned sh[kScanTile + kScanTile / 32];
    __shared__ unsigned ws[kBlock / 32];
    scan_apply_sparse_tile(count, C, tile, start, T, blockIdx.x, reach, live, sh, ws);
}

gs_status scan_tile_totals(const unsigned* count, unsigned C, unsigned* tile, cudaStream_t st) {
    const unsigned T = scan_tile_count(C);
    if (T == 0) return GS_OK;
    launch_after(k_scan_reduce, T, kBlock, 0, st, count, C, tile);
    GS_LAUNCHED("scan_tile_totals");
    return GS_OK;
}

gs_status scan_counts_sparse(unsigned* count, unsigned* start, unsigned C, const unsigned* tile,
                             unsigned* live, unsigned reach, cudaStream_t st) {
    const unsigned T = scan_tile_count(C);
    if (T == 0) return GS_OK;
    launch_after(k_scan_apply_sparse, T, kBlock, 0, st, count, C, tile, start, T, reach, live);
    GS_LAUNCHED("scan_sparse");
    return GS_OK;
}

unsigned scan_reach_tiles(const unsigned wc[3], unsigned r) {
    // labels are x + z wc0 + y wc0 wc2: a box of radius r reads starts at
    // most rx + rz wc0 + ry wc0 wc2 + 1 labels from its centre cell (the +1:
    // the start after a row's last cell)
    auto reach = [&](unsigned n) { return std::min<unsigned long long>(r, n ? n - 1 : 0); };
    const unsigned long long d = reach(wc[0]) + reach(wc[2]) * wc[0] +
                                 reach(wc[1]) * (unsigned long long)wc[0] * wc[2] + 1;
    const unsigned long long t = (d + kScanTile - 1) / kScanTile;
    return t > 0xffffffffull ? 0xffffffffu : unsigned(t);
}

// ---- database -----------------------------------------------------------------------
gs_status db_reserve(Database& db, unsigned n, unsigned C) {
    if (db.cells != C) {
        dfree(db.start);
        dfree(db.count);
        dfree(db.tile);
        dfree(db.live);
        GS_TRY(dalloc(&db.start, size_t(C) + 1));
        GS_TRY(dalloc(&db.count, C));
        GS_TRY(dalloc(&db.tile, scan_tile_count(C) + 1));
        GS_TRY(dalloc(&db.live, scan_tile_count(C) + 1));
        GS_CUDA(cudaMemset(db.count, 0, size_t(C) * sizeof(unsigned)));
        GS_CUDA(cudaMemset(db.tile, 0, (size_t(scan_tile_count(C)) + 1) * sizeof(unsigned)));
        GS_CUDA(cudaMemset(db.live, 0, (size_t(scan_tile_count(C)) + 1) * sizeof(unsigned)));
        // the counts are used next on a non-blocking stream
        GS_CUDA(cudaDeviceSynchronize());
        db.cells = C;
    }
    if (n > 0 && db.cell == nullptr) {
        GS_TRY(dalloc(&db.cell, n));
        GS_TRY(dalloc(&db.rank, n));
        GS_TRY(dalloc(&db.sorted, n));
        GS_TRY(dalloc(&db.pos_id, n));
    }
    db.valid = false;
    return GS_OK;
}

void db_release(Database& db) {
    dfree(db.cell);
    dfree(db.rank);
    dfree(db.sorted);
    dfree(db.pos_id);
    dfree(db.start);
    dfree(db.count);
    dfree(db.tile);
    dfree(db.live);
    db.cells = 0;
    db.agent_cap = 0;
    db.valid = false;
}

__global__ void k_db_count(const float4* pos, unsigned n, Grid g,
                           unsigned* cell, unsigned* rank,
                           unsigned* count) {
    after_previous();
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned c = cell_of(g, v3(pos[i]));
    cell[i] = c;
    rank[i] = atomicAdd(count + c, 1u);
}

__global__ void k_db_scatter(const float4* pos, unsigned n,
                             const unsigned* cell, const unsigned* rank,
                             const unsigned* start, unsigned* sorted,
                             float4* pos_id) {
    after_previous();
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const unsigned dst = start[cell[i]] + rank[i];
    if (dst >= n) return;
    const float4 p = pos[i];
    sorted[dst] = i;
    pos_id[dst] = make_float4(p.x, p.y, p.z, __uint_as_float(i));
}

gs_status db_build(Database& db, const float4* pos, unsigned n, const Grid& grid,
                   cudaStream_t st) {
    const unsigned C = grid.wc[0] * grid.wc[1] * grid.wc[2];
    if (db.cells != C || (n > 0 && db.cell == nullptr))
        return fail(GS_ERR_STATE, "database not reserved for this grid");
    if (n > 0 && db_on_cluster(n, C)) {
        DbJobs J;
        J.job[0] = db_job(db, pos, n, grid);
        GS_TRY(db_build_clusters(J, 1, st));
    } else {
        if (n > 0)
            launch_after(k_db_count, blocks_for(n), kBlock, 0, st, pos, n, grid, db.cell, db.rank, db.count);
        GS_TRY(scan_counts(db.count, db.start, C, db.tile, st));
        if (n > 0)
            launch_after(k_db_scatter, blocks_for(n), kBlock, 0, st, pos, n, db.cell, db.rank, db.start, db.sorted, db.pos_id);
        GS_LAUNCHED("db_build");
    }
    db.grid = grid;
    db.valid = true;
    return GS_OK;
}

// ---- brute-force KNN (KNNBruteForceCudaKernel.cu:207-283) ---------------------------
// ---- brute force, FP32-pipe form (k <= 64) ----------------------------------------------
// One warp serves kBruteQW queries and keeps each query's exact (distance,
// index) top-k list spread over its lanes: lane r holds entry r (and entry
// 32 + r for k > 32), so the list is sorted across the warp and its k-th key
// is one shuffle away.  The
// block stages kBruteTile candidates in shared memory as x / y / z arrays;
// each lane takes two neighbouring candidates per step and computes their
// squared distances to every query of its warp with packed f32x2 subtract,
// multiply and fused multiply-add.  Those squared distances only filter:
// the warp votes on "within the rounded-up bound of a list's k-th distance"
// and, when any lane says yes, every lane recomputes the candidate's distance
// with the reference's unfused binary32 operations (KNNBruteForceCudaKernel.cu
// :245-271) and the list takes it with one shuffle-and-select insertion.  The
// packed d^2 differs from the unfused one by a few units in the last place,
// far inside the bound's 4e-6 relative margin, so no candidate that belongs
// in a list is filtered out; insertion is by the exact key, so the lists are
// the reference's (distance, lower index) order.  After the first few
// hundred candidates almost no step has a vote, so the warp runs the packed
// arithmetic without divergence.
constexpr unsigned kBruteWarps = 8;
constexpr unsigned kBruteQW = 4;      // queries per warp
constexpr unsigned kBruteTile = 2048; // candidates staged per block step

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// A query's exact (distance, index) top-k list spread over the warp: lane r
// holds rank r in e[0] and, with L = 2 (32 < k <= 64), rank 32 + r in e[1].
// Ranks at or past k hold the empty key.
template <int L>
struct WarpList {
    unsigned long long e[L];
    __device__ __forceinline__ void init() {
#pragma unroll
        for (int h = 0; h < L; ++h) e[h] = KEY_EMPTY;
    }
    // the k-th key, on every lane (k is warp-uniform)
    __device__ __forceinline__ unsigned long long kth(unsigned k) const {
        if (L == 1 || k <= 32) return __shfl_sync(0xffffffffu, e[0], int(k) - 1);
        return __shfl_sync(0xffffffffu, e[L - 1], int(k) - 33);
    }
};

// Inserts candidate (x, y, z, id) into the lane-distributed list if its
// exact key is below the k-th: each rank below k whose key is larger takes
// the larger of the candidate and the rank before it (all from the old
// list); updates the filter bound.  Every lane runs it with the same
// candidate.
template <int L>
__device__ __forceinline__ void warp_list_insert(WarpList<L>& w, float& bound, V3 q, float x, float y, float z, unsigned id, unsigned k,
                                                 unsigned lane) {
    const unsigned long long key = knn_key(distance(q, v3(x, y, z)), id);
    if (!(key < w.kth(k))) return;  // warp-uniform
    const unsigned long long left0 = __shfl_up_sync(0xffffffffu, w.e[0], 1);
    if (L == 2) {
        unsigned long long left1 = __shfl_up_sync(0xffffffffu, w.e[L - 1], 1);
        const unsigned long long last0 = __shfl_sync(0xffffffffu, w.e[0], 31);
        if (lane == 0) left1 = last0;  // rank 32 follows rank 31
        if (32 + lane < k && key < w.e[L - 1]) w.e[L - 1] = key > left1 ? key : left1;
    }
    if (lane < k && key < w.e[0]) w.e[0] = (lane == 0 || key > left0) ? key : left0;
    bound = prefilter_bound(w.kth(k));
}

// Writes a warp list to idx / dist[a + rank * nA], ranks below k.
template <int L>
__device__ __forceinline__ void warp_list_store(const WarpList<L>& w, unsigned a, unsigned nA,
                                                unsigned k, unsigned lane,
                                                unsigned* __restrict__ idx,
                                                float* __restrict__ dist) {
#pragma unroll
    for (int h = 0; h < L; ++h) {
        const unsigned rank = 32u * h + lane;
        if (rank < k) {
            idx[a + size_t(rank) * nA] = key_id(w.e[h]);
            dist[a + size_t(rank) * nA] = key_dist(w.e[h]);
        }
    }
}

// The warp's step over the staged candidates t0 .. t0 + 63 (each lane the
// pair t0 + 2 lane, t0 + 2 lane + 1): the packed filter against every query
// of the warp, then the exact insertion of the candidates that passed.
template <int L>
__device__ __forceinline__ void brute_chunk(
    const float* sx, const float* sy, const float* sz, unsigned base, unsigned t0, unsigned cnt,
    unsigned lane, bool self, unsigned k, const V3 (&q)[kBruteQW],
    const unsigned (&qid)[kBruteQW], const unsigned long long (&px)[kBruteQW],
    const unsigned long long (&py)[kBruteQW], const unsigned long long (&pz)[kBruteQW],
    WarpList<L> (&entry)[kBruteQW], float (&bound)[kBruteQW]) {
    const unsigned t = t0 + 2 * lane;
    const unsigned long long x2 = *reinterpret_cast<const unsigned long long*>(sx + t);
    const unsigned long long y2 = *reinterpret_cast<const unsigned long long*>(sy + t);
    const unsigned long long z2 = *reinterpret_cast<const unsigned long long*>(sz + t);
    bool hit0[kBruteQW], hit1[kBruteQW];
    bool any = false;
#pragma unroll
    for (unsigned j = 0; j < kBruteQW; ++j) {
        const unsigned long long dx = sub2(px[j], x2), dy = sub2(py[j], y2), dz = sub2(pz[j], z2);
        float e0, e1;
        unpack2(fma2(dz, dz, fma2(dy, dy, mul2(dx, dx))), e0, e1);
        hit0[j] = e0 <= bound[j];
        hit1[j] = e1 <= bound[j];
        any |= hit0[j] | hit1[j];
    }
    if (!__any_sync(0xffffffffu, any)) return;
    // only the candidates that passed: the lane's first (h = 0) and second
    // (h = 1) candidate have separate votes
#pragma unroll
    for (unsigned j = 0; j < kBruteQW; ++j) {
#pragma unroll
        for (unsigned h = 0; h < 2; ++h) {
            unsigned m = __ballot_sync(0xffffffffu, h ? hit1[j] : hit0[j]);
            while (m) {
                const unsigned src = unsigned(__ffs(m)) - 1u;
                m &= m - 1u;
                const unsigned c = t0 + 2 * src + h;
                if (c >= cnt) continue;
                const unsigned id = base + c;
                if (self && id == qid[j]) continue;
                warp_list_insert(entry[j], bound[j], q[j], sx[c], sy[c], sz[c], id, k, lane);
            }
        }
    }
}

template <int L>
__global__ void __launch_bounds__(kBruteWarps * 32) k_knn_brute3(
    const float4* __restrict__ posA, unsigned nA, const float4* __restrict__ posB, unsigned nB,
    bool self, unsigned k, unsigned* __restrict__ idx, float* __restrict__ dist) {
    __shared__ __align__(16) float sx[kBruteTile], sy[kBruteTile], sz[kBruteTile];
    const unsigned warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned q0 = (blockIdx.x * kBruteWarps + warp) * kBruteQW;
    V3 q[kBruteQW];
    unsigned qid[kBruteQW];
    unsigned long long px[kBruteQW], py[kBruteQW], pz[kBruteQW];
    WarpList<L> entry[kBruteQW];
    float bound[kBruteQW];
#pragma unroll
    for (unsigned j = 0; j < kBruteQW; ++j) {
        const bool act = q0 + j < nA;
        qid[j] = q0 + j;
        q[j] = act ? v3(posA[q0 + j]) : v3(0.f, 0.f, 0.f);
        px[j] = pack2(q[j].x, q[j].x);
        py[j] = pack2(q[j].y, q[j].y);
        pz[j] = pack2(q[j].z, q[j].z);
        entry[j].init();
        bound[j] = act ? prefilter_bound(KEY_EMPTY) : -1.f;
    }
    const float inf = __int_as_float(0x7f800000);
    for (unsigned base = 0; base < nB; base += kBruteTile) {
        __syncthreads();
        for (unsigned c = threadIdx.x; c < kBruteTile; c += blockDim.x) {
            const float4 v = base + c < nB ? posB[base + c] : make_float4(inf, inf, inf, 0.f);
            sx[c] = v.x;
            sy[c] = v.y;
            sz[c] = v.z;
        }
        __syncthreads();
        const unsigned cnt = min(kBruteTile, nB - base);
        for (unsigned t0 = 0; t0 < cnt; t0 += 64)
            brute_chunk(sx, sy, sz, base, t0, cnt, lane, self, k, q, qid, px, py, pz, entry, bound);
    }
#pragma unroll
    for (unsigned j = 0; j < kBruteQW; ++j)
        if (q0 + j < nA) warp_list_store(entry[j], q0 + j, nA, k, lane, idx, dist);
}

gs_status launch_knn_brute(const float4* posA, unsigned nA, const float4* posB, unsigned nB,
                           bool self, unsigned k, unsigned* idx, float* dist, cudaStream_t st) {
    if (nA == 0) return GS_OK;
    if (k == 0 || k > 64) return fail(GS_ERR_UNSUPPORTED, "brute force needs 1 <= k <= 64");
    const unsigned per_block = kBruteWarps * kBruteQW, blocks = (nA + per_block - 1) / per_block;
    if (k <= 32)
        k_knn_brute3<1><<<blocks, kBruteWarps * 32, 0, st>>>(posA, nA, posB, nB, self, k, idx,
                                                             dist);
    else
        k_knn_brute3<2><<<blocks, kBruteWarps * 32, 0, st>>>(posA, nA, posB, nB, self, k, idx,
                                                             dist);
    GS_LAUNCHED("knn_brute");
    return GS_OK;
}

// ---- ExtractData diagnostics (ProcessData.cu:132-237) -------------------------------------
// live (the fused engine's frame, may be null): tiles whose starts the last
// scan wrote; a cell of another tile is empty.
__device__ __forceinline__ bool frame_cell_live(const unsigned* live, unsigned c) {
    return live == nullptr || live[c / kScanTile] != 0u;
}

__global__ void k_cell_density(const unsigned* __restrict__ start, unsigned C,
                               const unsigned* __restrict__ live, unsigned* __restrict__ out) {
    const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c < C) out[c] = frame_cell_live(live, c) ? start[c + 1] - start[c] : 0u;
}

// A cell's agents are added in ascending index, the order the reference's
// stable sort leaves them in; this database's counting sort orders a cell's
// slots arbitrarily, so the cell's thread picks its agents by increasing
// index (quadratic in the cell's count: a diagnostic, not a step kernel).
__global__ void k_cell_avg_velocity(const unsigned* __restrict__ start,
                                    const unsigned* __restrict__ sorted, unsigned C,
                                    const float4* __restrict__ dir,
                                    const float* __restrict__ speed, float3* __restrict__ out) {
    const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const unsigned s0 = start[c], s1 = start[c + 1];
    V3 sum = v3(0.f, 0.f, 0.f);
    unsigned last = 0;
    for (unsigned t = 0; t < s1 - s0; ++t) {
        unsigned next = UINT_MAX;
        for (unsigned s = s0; s < s1; ++s) {
            const unsigned id = sorted[s];
            if ((t == 0 || id > last) && id < next) next = id;
        }
        last = next;
        sum = add(sum, mul(v3(dir[next]), speed[next]));
    }
    const V3 avg = s1 > s0 ? dvd(sum, float(s1 - s0)) : v3(0.f, 0.f, 0.f);
    out[c] = make_float3(avg.x, avg.y, avg.z);
}

// The same average over the fused step's frame: slot s of the start-of-step
// buckets holds the agent whose new state the step wrote to A[s] (its index
// in f0.w, heading and speed in f1).  A cell's agents belong to one scene, so
// ascending index is the reference's order here too.
__global__ void k_cell_avg_velocity_frame(const unsigned* __restrict__ start, unsigned C,
                                          const unsigned* __restrict__ live,
                                          const float4* __restrict__ f0,
                                          const float4* __restrict__ f1,
                                          float3* __restrict__ out) {
    const unsigned c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const bool on = frame_cell_live(live, c);
    const unsigned s0 = on ? start[c] : 0u, s1 = on ? start[c + 1] : 0u;
    V3 sum = v3(0.f, 0.f, 0.f);
    unsigned last = 0;
    for (unsigned t = 0; t < s1 - s0; ++t) {
        unsigned next = UINT_MAX, at = s0;
        for (unsigned s = s0; s < s1; ++s) {
            const unsigned id = __float_as_uint(f0[s].w);
            if ((t == 0 || id > last) && id < next) {
                next = id;
                at = s;
            }
        }
        last = next;
        const float4 h = f1[at];
        sum = add(sum, mul(v3(h), h.w));
    }
    const V3 avg = s1 > s0 ? dvd(sum, float(s1 - s0)) : v3(0.f, 0.f, 0.f);
    out[c] = make_float3(avg.x, avg.y, avg.z);
}

gs_status launch_frame_cell_density(const unsigned* start, const unsigned* live, unsigned C,
                                    unsigned* out, cudaStream_t st) {
    if (C == 0) return GS_OK;
    k_cell_density<<<blocks_for(C), kBlock, 0, st>>>(start, C, live, out);
    GS_LAUNCHED("cell_density");
    return GS_OK;
}

gs_status launch_frame_cell_avg_velocity(const unsigned* start, const unsigned* live,
                                         unsigned C, const float4* f0, const float4* f1,
                                         float3* out, cudaStream_t st) {
    if (C == 0) return GS_OK;
    k_cell_avg_velocity_frame<<<blocks_for(C), kBlock, 0, st>>>(start, C, live, f0, f1, out);
    GS_LAUNCHED("cell_avg_velocity");
    return GS_OK;
}

gs_status launch_cell_density(const Database& db, unsigned* out, cudaStream_t st) {
    if (db.cells == 0) return GS_OK;
    k_cell_density<<<blocks_for(db.cells), kBlock, 0, st>>>(db.start, db.cells, nullptr, out);
    GS_LAUNCHED("cell_density");
    return GS_OK;
}

gs_status launch_cell_avg_velocity(const Database& db, const float4* dir, const float* speed,
                                   float3* out, cudaStream_t st) {
    if (db.cells == 0) return GS_OK;
    k_cell_avg_velocity<<<blocks_for(db.cells), kBlock, 0, st>>>(db.start, db.sorted, db.cells,
                                                                  dir, speed, out);
    GS_LAUNCHED("cell_avg_velocity");
    return GS_OK;
}

// Threads per block of the per-function launches: small groups in small
// blocks, so that their few warps spread over all SMs.
static unsigned call_block(unsigned n) { return n <= 64u * 8u * sm_count() ? 64u : unsigned(kBlock); }

// ---- WrapWorldCUDAKernel.cu:11-48 ---------------------------------------------------
__global__ void k_wrap(float4* pos, unsigned n, float wx, float wy, float wz, int mode) {
    after_previous();
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float ws[3] = {wx, wy, wz};
    pos[i] = f4(wrap_world(v3(pos[i]), ws, mode), 0.f);
}

gs_status launch_wrap(float4* pos, unsigned n, const float ws[3], int mode, cudaStream_t st) {
    if (n == 0) return GS_OK;
    const unsigned bs = call_block(n);
    launch_after(k_wrap, blocks_for(n, bs), bs, 0, st, pos, n, ws[0], ws[1], ws[2], mode);
    GS_LAUNCHED("wrap_world");
    return GS_OK;
}

// ---- one behaviour per launch ----------------------------------------------------------
__device__ __forceinline__ Self load_self(const GroupView& g, unsigned i) {
    Self s;
    s.pos = v3(g.position[i]);
    s.dir = v3(g.direction[i]);
    const float3 sd = g.side[i], u = g.up[i];
    s.side = v3(sd.x, sd.y, sd.z);
    s.up = v3(u.x, u.y, u.z);
    s.speed = g.speed[i];
    s.radius = g.radius[i];
    s.max_speed = g.max_speed[i];
    s.max_force = g.max_force[i];
    s.mass = g.mass[i];
    return s;
}

// A behaviour over a KNN list, one thread per agent.  The list's entries are
// taken kCallChunk at a time: their indices, then their neighbours' state, are
// loaded together, so a chunk costs two load latencies instead of two per
// entry (the loop over single entries was one dependent chain: 11.1 us at
// 30,011 agents, k = 7, and 23 us at 10,000, k = 16).  An index past the
// other group ends the list, as in the reference's kernels.
constexpr unsigned kCallChunk = 8;

// Calls body(s0, b, ok) for each chunk: ok[j]: entry s0 + j holds neighbour b[j]
// (b[j] is 0 where there is none, a safe index to load).
template <unsigned CHUNK = kCallChunk, class Body>
__device__ __forceinline__ void for_each_chunk(const unsigned* knn, unsigned i,
                                               unsigned n, unsigned k, unsigned n_other,
                                               Body&& body) {
    bool more = true;
    for (unsigned s0 = 0; s0 < k && more; s0 += CHUNK) {
        unsigned b[CHUNK];
        bool ok[CHUNK];
#pragma unroll
        for (unsigned j = 0; j < CHUNK; ++j)
            b[j] = s0 + j < k ? knn[i + size_t(s0 + j) * n] : UINT_MAX;
#pragma unroll
        for (unsigned j = 0; j < CHUNK; ++j) {
            more = more && b[j] < n_other;
            ok[j] = more;
            b[j] = ok[j] ? b[j] : 0u;
        }
        if (!ok[0]) return;
        more = body(s0, b, ok) && more;
    }
}

// KIND: 0 separation, 1 alignment, 2 cohesion
// (SteerFor{Separation,Alignment,Cohesion}CUDAKernel.cu:85-134)
template <int KIND>
__global__ void k_flock(GroupView g, const unsigned* knn, unsigned k, OtherView o,
                        FlockParams fp) {
    after_previous();
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    unsigned applied = g.applied[i];
    const V3 pos = v3(g.position[i]), dir = v3(g.direction[i]);
    V3 steer = v3(g.steering[i]);
    if (applied & fp.mask) return;
    const AngleGate gate = angle_gate(dir, fp.cos_max);
    FlockAcc acc;
    flock_init(acc);
    for_each_chunk(knn, i, g.n, k, o.n, [&](unsigned, const unsigned* b, const bool* ok) {
        float4 bp[kCallChunk], bd[kCallChunk];
#pragma unroll
        for (unsigned j = 0; j < kCallChunk; ++j) {
            bp[j] = o.position[b[j]];
            if (KIND == 1) bd[j] = o.direction[b[j]];
        }
#pragma unroll
        for (unsigned j = 0; j < kCallChunk; ++j) {
            const V3 offset = sub(v3(bp[j]), pos);
            const float dsq = dot(offset, offset), d = sqrtf(dsq);
            // inBoidNeighborhood (FlockingCommon.cuh:4-30); its angle test
            // without the divisions wherever the gate decides it
            bool in = ok[j] && d < fp.min_d;
            if (ok[j] && !in && !(d > fp.max_d)) {
                const float de = (dsq >= 0x1p-60f && dsq <= 0x1p60f) ? d : __int_as_float(0x7fffffff);
                const int ahead = angle_decide(dot(dir, offset), de, fp.cos_max, gate);
                in = ahead < 0 ? forward_component(dir, offset, dsq) > fp.cos_max : ahead > 0;
            }
            if (!in) continue;
            acc.sum = add(acc.sum, KIND == 0 ? dvd<true>(offset, -dsq) : KIND == 1 ? v3(bd[j]) : v3(bp[j]));
            acc.n++;
        }
        return true;
    });
    Self me;
    me.pos = pos;
    me.dir = dir;
    flock_finish<true>(KIND, acc, fp, me, applied, steer);
    g.steering[i] = f4(steer, 0.f);
    g.applied[i] = applied;
}

gs_status launch_flock(int kind, GroupView g, const unsigned* knn, unsigned k, OtherView o,
                       float min_d, float max_d, float cos_max, float w, unsigned mask,
                       cudaStream_t st) {
    if (g.n == 0) return GS_OK;
    const FlockParams fp{min_d, max_d, cos_max, w, mask};
    if (lanes_calls(g.n, k, false)) {
        launch_flock_lanes(kind, g, knn, k, o, fp, st);
        GS_LAUNCHED("steer_flock");
        return GS_OK;
    }
    const unsigned bs = call_block(g.n), nb = blocks_for(g.n, bs);
    if (kind == 0) launch_after(k_flock<0>, nb, bs, 0, st, g, knn, k, o, fp);
    else if (kind == 1) launch_after(k_flock<1>, nb, bs, 0, st, g, knn, k, o, fp);
    else launch_after(k_flock<2>, nb, bs, 0, st, g, knn, k, o, fp);
    GS_LAUNCHED("steer_flock");
    return GS_OK;
}

__global__ void k_seek(GroupView g, float tx, float ty, float tz, float w, unsigned mask) {
    after_previous();
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    unsigned applied = g.applied[i];
    if (applied & mask) return;
    Self me;
    me.pos = v3(g.position[i]);
    me.dir = v3(g.direction[i]);
    V3 steer = v3(g.steering[i]);
    seek_finish<true>(v3(tx, ty, tz), w, mask, me, applied, steer);
    g.steering[i] = f4(steer, 0.f);
    g.applied[i] = applied;
}

gs_status launch_seek(GroupView g, const float target[3], float w, unsigned mask,
                      cudaStream_t st) {
    if (g.n == 0) return GS_OK;
    const unsigned bs = call_block(g.n);
    launch_after(k_seek, blocks_for(g.n, bs), bs, 0, st, g, target[0], target[1], target[2], w, mask);
    GS_LAUNCHED("steer_seek");
    return GS_OK;
}

__global__ void k_follow_path(GroupView g, PathDev path, float prediction_time, float w,
                              unsigned mask) {
    after_previous();
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    unsigned applied = g.applied[i];
    if (applied & mask) return;
    Self me;
    me.pos = v3(g.position[i]);
    me.dir = v3(g.direction[i]);
    me.speed = g.speed[i];
    V3 steer = v3(g.steering[i]);
    follow_path_finish(path, prediction_time, w, mask, me, applied, steer);
    g.steering[i] = f4(steer, 0.f);
    g.applied[i] = applied;
}

gs_status launch_follow_path(GroupView g, const PathDev& path, float prediction_time, float w,
                             unsigned mask, cudaStream_t st) {
    if (g.n == 0) return GS_OK;
    launch_after(k_follow_path, blocks_for(g.n), kBlock, 0, st, g, path, prediction_time, w, mask);
    GS_LAUNCHED("steer_follow_path");
    return GS_OK;
}

template <unsigned CHUNK>
__global__ void k_avoid_close(GroupView g, const unsigned* knn,
                              const float* knn_dist, unsigned k, OtherView o,
                              float min_sep, float w, unsigned mask) {
    after_previous();
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    unsigned applied = g.applied[i];
    const Self me = load_self(g, i);
    V3 steer = v3(g.steering[i]);
    if (applied & mask) return;
    CloseAcc acc;
    close_init(acc);
    for_each_chunk<CHUNK>(knn, i, g.n, k, o.n, [&](unsigned s0, const unsigned* b, const bool* ok) {
        float4 bp[CHUNK];
        float br[CHUNK], kd[CHUNK];
#pragma unroll
        for (unsigned j = 0; j < CHUNK; ++j) {
            bp[j] = o.position[b[j]];
            br[j] = o.radius[b[j]];
            kd[j] = ok[j] ? knn_dist[i + size_t(s0 + j) * g.n] : 0.f;
        }
#pragma unroll
        for (unsigned j = 0; j < CHUNK; ++j)
            if (ok[j]) close_add(acc, me, min_sep, kd[j], v3(bp[j]), br[j]);
        return !acc.found;
    });
    close_finish(acc, w, mask, applied, steer);
    g.steering[i] = f4(steer, 0.f);
    g.applied[i] = applied;
}

// False only where the neighbour's approach time is provably outside [0, min_t)
// (avoid_time_window_test), so that avoid_add would change nothing.
__device__ __forceinline__ bool avoid_time_may_fall_in(const Self& me, float min_t, V3 bpos, V3 bdir,
                                                       float bspeed) {
    const V3 rv = sub(mul(bdir, bspeed), mul(me.dir, me.speed)), rp = sub(me.pos, bpos);
    const V3 h = v3(rv.x * rp.x, rv.y * rp.y, rv.z * rp.z);
    return avoid_time_window_test(dot(rv, rv), (h.x + h.y) + h.z,
                                  (fabsf(h.x) + fabsf(h.y)) + fabsf(h.z), min_t);
}

template <unsigned CHUNK, int BLOCKS>
__global__ void __launch_bounds__(kBlock, BLOCKS) k_avoid(GroupView g, const unsigned* knn, unsigned k, OtherView o,
                        float min_time, float w, unsigned mask) {
    after_previous();
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    unsigned applied = g.applied[i];
    const Self me = load_self(g, i);
    V3 steer = v3(g.steering[i]);
    if (applied & (mask | AVOID_CLOSE_NEIGHBORS_BIT)) return;
    AvoidAcc acc;
    avoid_init(acc, min_time);
    for_each_chunk<CHUNK>(knn, i, g.n, k, o.n, [&](unsigned, const unsigned* b, const bool* ok) {
        float4 bp[CHUNK], bd[CHUNK];
        float bv[CHUNK], br[CHUNK];
#pragma unroll
        for (unsigned j = 0; j < CHUNK; ++j) {
            bp[j] = o.position[b[j]];
            bd[j] = o.direction[b[j]];
            bv[j] = o.speed[b[j]];
            br[j] = o.radius[b[j]];
        }
#pragma unroll
        for (unsigned j = 0; j < CHUNK; ++j)
            if (ok[j] && avoid_time_may_fall_in(me, min_time, v3(bp[j]), v3(bd[j]), bv[j]))
                avoid_add<true>(acc, me, b[j], v3(bp[j]), v3(bd[j]), bv[j], br[j]);
        return true;
    });
    if (acc.threat == UINT_MAX) return;
    avoid_finish<true>(acc, w, mask, me, applied, steer);
    g.steering[i] = f4(steer, 0.f);
    g.applied[i] = applied;
}

gs_status launch_avoid_neighbors(GroupView g, const unsigned* knn, const float* knn_dist,
                                 unsigned k, OtherView o, float min_time, float min_sep,
                                 bool avoid_close, float w, unsigned mask, cudaStream_t st) {
    if (g.n == 0) return GS_OK;
    if (lanes_calls(g.n, k, true)) {
        launch_avoid_lanes(g, knn, knn_dist, k, o, min_time, min_sep, avoid_close, w, mask, st);
        GS_LAUNCHED("steer_avoid_neighbors");
        return GS_OK;
    }
    const unsigned bs = call_block(g.n), nb = blocks_for(g.n, bs);
    // Groups that pass the blocks that fit at two to an SM have warps enough to
    // hide the loads' latency, and gain by more blocks instead (us a call, a chunk
    // of 8 / 1: 200,000 agents, k = 7 32.2 / 24.7, k = 16 44.6 / 41.1, 400,000,
    // k = 16 79 / 64; with the close pass, 8 / 2: 36.1 / 27.7 and 42.2 / 33.6).
    const bool many = g.n > 2 * kBlock * sm_count();
    if (avoid_close) {
        const auto close = many ? k_avoid_close<2> : k_avoid_close<kCallChunk>;
        launch_after(close, nb, bs, 0, st, g, knn, knn_dist, k, o, min_sep, w, mask);
    }
    const auto avoid = many ? k_avoid<1, 4> : k_avoid<kCallChunk, 2>;
    launch_after(avoid, nb, bs, 0, st, g, knn, k, o, min_time, w, mask);
    GS_LAUNCHED("steer_avoid_neighbors");
    return GS_OK;
}

__global__ void k_avoid_walls(GroupView g, const unsigned* knw, unsigned kw,
                              const float4* ls, const float4* le,
                              const float4* ln, unsigned n_lines, float min_time,
                              float w, unsigned mask) {
    after_previous();
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    unsigned applied = g.applied[i];
    if (applied & mask) return;
    Self me = load_self(g, i);
    WallAcc acc;
    walls_init(acc, me, min_time);
    for (unsigned s = 0; s < kw; ++s) {
        const unsigned line = knw[i + size_t(s) * g.n];
        if (line >= n_lines) break;
        walls_add(acc, me, line, v3(ls[line]), v3(le[line]), v3(ln[line]));
    }
    V3 steer = v3(g.steering[i]);
    walls_finish(acc, w, mask, me, applied, steer);
    g.steering[i] = f4(steer, 0.f);
    g.position[i] = f4(me.pos, 0.f);
    g.direction[i] = f4(me.dir, 0.f);
    g.applied[i] = applied;
}

gs_status launch_avoid_walls(GroupView g, const unsigned* knw, unsigned kw, const float4* start,
                             const float4* end, const float4* normal, unsigned n_lines,
                             float min_time, float w, unsigned mask, cudaStream_t st) {
    if (g.n == 0) return GS_OK;
    if (kw <= 8 && lanes_calls(g.n, kw, true)) {
        launch_avoid_walls_lanes(g, knw, kw, start, end, normal, n_lines, min_time, w, mask, st);
        GS_LAUNCHED("steer_avoid_walls");
        return GS_OK;
    }
    const unsigned bs = call_block(g.n);
    launch_after(k_avoid_walls, blocks_for(g.n, bs), bs, 0, st, g, knw, kw, start, end, normal, n_lines, min_time, w, mask);
    GS_LAUNCHED("steer_avoid_walls");
    return GS_OK;
}

__global__ void k_update(GroupView g, float dt) {
    after_previous();
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    Self me = load_self(g, i);
    integrate<true>(me, v3(g.steering[i]), dt);
    g.side[i] = make_float3(me.side.x, me.side.y, me.side.z);
    g.up[i] = make_float3(me.up.x, me.up.y, me.up.z);
    g.direction[i] = f4(me.dir, 0.f);
    g.position[i] = f4(me.pos, 0.f);
    g.steering[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    g.speed[i] = me.speed;
    g.applied[i] = 0u;
}

gs_status launch_update(GroupView g, float dt, cudaStream_t st) {
    if (g.n == 0) return GS_OK;
    const unsigned bs = call_block(g.n);
    launch_after(k_update, blocks_for(g.n, bs), bs, 0, st, g, dt);
    GS_LAUNCHED("update_group");
    return GS_OK;
}

// updateGroupWithAntiPenetration (UpdateCUDAKernelNew.cu:95-268): the update
// with the walls' anti-penetration.  Behaviour kept from the reference kernel:
// the wall list is read row-major, knl[i*k + s] (:149-150), although
// findKNearestNeighbors writes it column-major; the overlap test measures the
// distance to lineStart + (lineEnd - lineStart), the segment's end, because
// ClosestPointOnLine's clamp(0.f, 1.f, t) returns 1 (:67-80); the last listed
// line within the radius pushes the agent out (:215-229); the nearest crossing
// of the move turns the velocity parallel to that wall (:201-237); applied
// bits are kept.  An agent whose new speed is 0 keeps its side vector.
__global__ void k_update_antipen_wall(GroupView g, const unsigned* __restrict__ knl, unsigned k,
                                      const float4* __restrict__ start,
                                      const float4* __restrict__ end,
                                      const float4* __restrict__ normal, unsigned n_lines,
                                      float dt) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    Self me = load_self(g, i);
    const V3 steer = truncate_length(v3(g.steering[i]), me.max_force);
    const V3 acc = dvd(steer, me.mass);
    V3 vel = add(mul(me.dir, me.speed), mul(acc, dt));
    vel = truncate_length(vel, me.max_speed);
    const V3 future = add(me.pos, mul(vel, dt));
    const float r = me.radius;
    float line_d = FLT_MAX, hit_d = FLT_MAX;
    unsigned line = UINT_MAX, hit = UINT_MAX;
    V3 line_n = v3(0.f, 0.f, 0.f), hit_n = v3(0.f, 0.f, 0.f);
    for (unsigned s = 0; s < k; ++s) {
        const unsigned li = knl[size_t(i) * k + s];
        if (li >= n_lines) break;
        const V3 ls = v3(start[li]), le = v3(end[li]), ln = v3(normal[li]);
        V3 ip;
        if (lines_intersect(me.pos, future, ls, le, ip)) {
            const float d = distance(me.pos, ip);
            if (d < hit_d) {
                hit_d = d;
                hit = li;
                hit_n = ln;
            }
        }
        const V3 o = sub(add(ls, sub(le, ls)), me.pos);
        const float dsq = dot(o, o);
        if (dsq < r * r) {
            line_d = sqrtf(dsq);
            line = li;
            line_n = ln;
        }
    }
    unsigned applied = g.applied[i];
    if (line != UINT_MAX) {
        me.pos = add(me.pos, mul(neg(line_n), line_d - r));
        applied |= ANTI_PENETRATION_WALL;
    }
    if (hit != UINT_MAX) {
        vel = perpendicular_component(vel, hit_n);
        applied |= ANTI_PENETRATION_WALL;
    }
    me.speed = length(vel);
    if (me.speed > 0.f) {
        me.dir = dvd(vel, me.speed);
        me.side = normalize(cross(me.dir, me.up));
        me.up = cross(me.side, me.dir);
    }
    me.pos = add(me.pos, mul(vel, dt));
    g.side[i] = make_float3(me.side.x, me.side.y, me.side.z);
    g.up[i] = make_float3(me.up.x, me.up.y, me.up.z);
    g.direction[i] = f4(me.dir, 0.f);
    g.position[i] = f4(me.pos, 0.f);
    g.steering[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    g.speed[i] = me.speed;
    g.applied[i] = applied;
}

gs_status launch_update_antipen_wall(GroupView g, const unsigned* knl, unsigned k,
                                     const float4* start, const float4* end,
                                     const float4* normal, unsigned n_lines, float dt,
                                     cudaStream_t st) {
    if (g.n == 0) return GS_OK;
    k_update_antipen_wall<<<blocks_for(g.n), kBlock, 0, st>>>(g, knl, k, start, end, normal,
                                                              n_lines, dt);
    GS_LAUNCHED("update_group_with_antipenetration");
    return GS_OK;
}

// antiPenetrationWall (AntiPenetrationWallCUDAKernel.cu:52-134): an agent
// whose move velocity * dt crosses a listed wall turns its heading parallel
// to the nearest crossed wall.  As the reference kernel: every agent is
// tested (its early-out `! applied & KERNEL_AVOID_WALLS_BIT`, :73, is never
// true), the wall list is read row-major (:88-91), every direction is
// rewritten with w = 0 (:133).
__global__ void k_antipen_wall(GroupView g, const unsigned* __restrict__ knl, unsigned k,
                               const float4* __restrict__ start, const float4* __restrict__ end,
                               const float4* __restrict__ normal, unsigned n_lines, float dt) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    const V3 pos = v3(g.position[i]);
    V3 dir = v3(g.direction[i]);
    const V3 future = add(pos, mul(mul(dir, g.speed[i]), dt));
    float hit_d = FLT_MAX;
    unsigned hit = UINT_MAX;
    for (unsigned s = 0; s < k; ++s) {
        const unsigned li = knl[size_t(i) * k + s];
        if (li >= n_lines) break;
        V3 ip;
        if (lines_intersect(pos, future, v3(start[li]), v3(end[li]), ip)) {
            const float d = distance(pos, ip);
            if (d < hit_d) {
                hit_d = d;
                hit = li;
            }
        }
    }
    if (hit != UINT_MAX) {
        dir = normalize(perpendicular_component(dir, v3(normal[hit])));
        g.applied[i] |= ANTI_PENETRATION_WALL;
    }
    g.direction[i] = f4(dir, 0.f);
}

gs_status launch_antipen_wall(GroupView g, const unsigned* knl, unsigned k, const float4* start,
                              const float4* end, const float4* normal, unsigned n_lines,
                              float dt, cudaStream_t st) {
    if (g.n == 0) return GS_OK;
    k_antipen_wall<<<blocks_for(g.n), kBlock, 0, st>>>(g, knl, k, start, end, normal, n_lines,
                                                       dt);
    GS_LAUNCHED("anti_penetration_wall");
    return GS_OK;
}

// One group's behaviour calls of a MultiGroup frame (Group::update,
// plugins/MultiGroup.cpp:558-601), per agent in the calls' order: avoid the
// neighbours of every other group (close pass, then main pass, per group,
// :573-580), separation from every group (:583-588), alignment and cohesion
// with this group (:590-591), then path following and seek of the path's
// second point when the group has a path (:593-597).  Each call keeps its own
// mask test and normalisation, and the applied bits accumulate from call to
// call, as the per-call kernels do.  Only steering and applied bits are
// written (positions move in the update that follows), so every read of a
// group's state sees the state the per-call kernels see.
__global__ void k_multigroup_steer(MultiSteer M) {
    const unsigned a = blockIdx.x * blockDim.x + threadIdx.x;
    const GroupView& g = M.g;
    if (a >= g.n) return;
    const unsigned n = g.n;
    unsigned applied = g.applied[a];
    V3 steer = v3(g.steering[a]);
    const Self me = load_self(g, a);
    for (unsigned j = 0; j < M.n_groups; ++j) {
        if (j == M.self) continue;
        const OtherView& o = M.o[j];
        const unsigned* idx = M.idx[j];
        if (M.avoid_close && !(applied & M.mask_avoid)) {
            CloseAcc acc;
            close_init(acc);
            for (unsigned s = 0; s < M.k[j]; ++s) {
                const unsigned b = idx[a + size_t(s) * n];
                if (b >= o.n) break;
                close_add(acc, me, M.min_sep, M.dist[j][a + size_t(s) * n], v3(o.position[b]),
                          o.radius[b]);
                if (acc.found) break;
            }
            close_finish(acc, M.w_avoid, M.mask_avoid, applied, steer);
        }
        if (!(applied & (M.mask_avoid | AVOID_CLOSE_NEIGHBORS_BIT))) {
            AvoidAcc acc;
            avoid_init(acc, M.min_time);
            for (unsigned s = 0; s < M.k[j]; ++s) {
                const unsigned b = idx[a + size_t(s) * n];
                if (b >= o.n) break;
                avoid_add(acc, me, b, v3(o.position[b]), v3(o.direction[b]), o.speed[b],
                          o.radius[b]);
            }
            if (acc.threat != UINT_MAX) avoid_finish(acc, M.w_avoid, M.mask_avoid, me, applied, steer);
        }
    }
    for (unsigned j = 0; j < M.n_groups; ++j) {
        if (applied & M.sep.mask) continue;
        const OtherView& o = M.o[j];
        FlockAcc acc;
        flock_init(acc);
        for (unsigned s = 0; s < M.k[j]; ++s) {
            const unsigned b = M.idx[j][a + size_t(s) * n];
            if (b >= o.n) break;
            const V3 offset = sub(v3(o.position[b]), me.pos);
            const float dsq = dot(offset, offset);
            separation_add(acc, M.sep, me.dir, offset, dsq, sqrtf(dsq));
        }
        flock_finish(0, acc, M.sep, me, applied, steer);
    }
    for (int kind = 1; kind <= 2; ++kind) {
        const FlockParams& fp = kind == 1 ? M.ali : M.coh;
        if (applied & fp.mask) continue;
        const OtherView& o = M.o[M.self];
        FlockAcc acc;
        flock_init(acc);
        for (unsigned s = 0; s < M.k[M.self]; ++s) {
            const unsigned b = M.idx[M.self][a + size_t(s) * n];
            if (b >= o.n) break;
            const V3 bp = v3(o.position[b]);
            const V3 offset = sub(bp, me.pos);
            const float d = sqrtf(dot(offset, offset));
            if (kind == 1) alignment_add(acc, fp, me.dir, offset, d, v3(o.direction[b]));
            else cohesion_add(acc, fp, me.dir, offset, d, bp);
        }
        flock_finish(kind, acc, fp, me, applied, steer);
    }
    if (M.has_path) {
        if (!(applied & M.mask_path))
            follow_path_finish(M.path, M.path_time, M.w_path, M.mask_path, me, applied, steer);
        if (!(applied & M.mask_seek))
            seek_finish(v3(M.seek_target[0], M.seek_target[1], M.seek_target[2]), M.w_seek,
                        M.mask_seek, me, applied, steer);
    }
    g.steering[a] = f4(steer, 0.f);
    g.applied[a] = applied;
}

gs_status launch_multigroup_steer(const MultiSteer& M, cudaStream_t st) {
    if (M.g.n == 0) return GS_OK;
    k_multigroup_steer<<<blocks_for(M.g.n), kBlock, 0, st>>>(M);
    GS_LAUNCHED("multigroup_steer");
    return GS_OK;
}

// AntiPenetrationAgentsCUDAKernel.cu:72-108.  Positions are read from the
// group and written to pos_out (the reference's m_pdPositionNew); the other
// group's applied bits are read from a snapshot taken before the launch (the
// reference reads them while this kernel sets bit 13 on the same array).
__global__ void k_antipen(GroupView g, const unsigned* __restrict__ knn,
                          const float* __restrict__ knn_dist, OtherView o,
                          const unsigned* __restrict__ applied_b, float4* __restrict__ out,
                          unsigned mask) {
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= g.n) return;
    const float4 p4 = g.position[i];
    out[i] = p4;
    unsigned applied = g.applied[i];
    if (applied & mask) return;
    const unsigned b = knn[i];
    if (b >= o.n) return;
    const float sum_radii = g.radius[i] + o.radius[b];
    const float overlap = sum_radii - knn_dist[i];
    if (overlap < 0.f) return;
    const V3 pos = v3(p4);
    const V3 offset = sub(pos, v3(o.position[b]));
    const V3 unit = normalize(offset);
    const float move = (applied_b[b] & mask) ? overlap : 0.5f * overlap;
    out[i] = f4(add(pos, mul(unit, move)), 0.f);
    g.applied[i] = applied | ANTI_PENETRATION_AGENT;
}

gs_status launch_antipenetration(GroupView g, const unsigned* knn, const float* knn_dist,
                                 unsigned k, OtherView o, const unsigned* applied_snapshot,
                                 float4* pos_out, unsigned mask, cudaStream_t st) {
    (void)k;
    if (g.n == 0) return GS_OK;
    k_antipen<<<blocks_for(g.n), kBlock, 0, st>>>(g, knn, knn_dist, o, applied_snapshot,
                                                  pos_out, mask);
    GS_LAUNCHED("anti_penetration_agents");
    GS_CUDA(cudaMemcpyAsync(g.position, pos_out, size_t(g.n) * sizeof(float4),
                            cudaMemcpyDeviceToDevice, st));
    return GS_OK;
}

}  // namespace gs
