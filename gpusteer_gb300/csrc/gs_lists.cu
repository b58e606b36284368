// Binned KNN with the reference's output layout (KNNBinningV2Kernel.cu:417-528):
// findKNearestNeighbors of one pair of groups, and every pair of a MultiGroup
// frame in one launch.  Queries are taken in bucketed order (neighbouring
// threads scan the same cells); results go to idx / dist[a + rank * nA].
//
// Two forms up to k = 32, and a warp per query beyond.  Few queries: a group of
// lanes per query (gs_lanes.cuh), whose serial chain is a few chunks of
// candidates.  Many: one thread per query on the streaming scan, whose list is in
// registers and whose candidates take no shared memory, so many warps stay
// resident; a query that scan cannot vouch for (ties, more than 256 candidates)
// is searched again by its whole warp, or, where a warp has many of them, by its
// own thread.
#include <algorithm>

#include "gs_lanes.cuh"
#include "gs_launch.h"

namespace gs {

constexpr unsigned kListBlock = 128;

__device__ __forceinline__ void put_entry(const KnnPair& pr, unsigned a, unsigned r, unsigned id,
                                          float d) {
    pr.idx[a + size_t(r) * pr.nA] = id;
    pr.dist[a + size_t(r) * pr.nA] = d;
}

// ---- a group of lanes per query ------------------------------------------------------------
template <int G, int R>
__device__ __forceinline__ void lists_lanes(const KnnPair& pr, const Grid& grid, unsigned r,
                                            unsigned thread, unsigned* rows) {
    const unsigned lane = threadIdx.x & unsigned(G - 1), q = thread / G;
    const bool act = q < pr.nA;  // spare groups run along and store nothing
    const float4 v = pr.a_pos_id[act ? q : pr.nA - 1];
    const unsigned a = __float_as_uint(v.w);
    unsigned ix, iy, iz;
    cell_coords(grid, v3(v), ix, iy, iz);
    const Box box = cell_box(grid, ix, iy, iz, r);
    const LaneEntry<G> e = lanes_knn<G, R>(pr.k, lane, v3(v), pr.self ? a : UINT_MAX, grid, box, 0u,
                                           pr.b_start, pr.b_pos_id, rows);
    // the empty entry is (FLT_MAX, UINT_MAX)
    if (act && lane < pr.k) put_entry(pr, a, lane, key_id(e.key), key_dist(e.key));
}

template <int G, int R>
__global__ void __launch_bounds__(kListBlock) k_lists_lanes(KnnPair pr, Grid grid, unsigned r) {
    after_previous();
    __shared__ unsigned row_sh[R ? 1 : kListBlock / G * kLaneRowWords];
    lists_lanes<G, R>(pr, grid, r, blockIdx.x * kListBlock + threadIdx.x,
                      row_sh + (R ? 0u : threadIdx.x / G * kLaneRowWords));
}

// The pair table rides in the kernel parameters; each pair owns a run of
// blocks, and a block finds its pair by a scan of the (few) block offsets.
__device__ __forceinline__ unsigned pair_of_block(const KnnPairs& P) {
    unsigned q = 0;
    while (q + 1 < P.n_pairs && blockIdx.x >= P.pair[q + 1].block_begin) ++q;
    return q;
}

template <int G, int R>
__global__ void __launch_bounds__(kListBlock) k_lists_lanes_pairs(const __grid_constant__ KnnPairs P) {
    after_previous();
    __shared__ unsigned row_sh[R ? 1 : kListBlock / G * kLaneRowWords];
    const KnnPair& pr = P.pair[pair_of_block(P)];
    lists_lanes<G, R>(pr, P.grid, P.r, (blockIdx.x - pr.block_begin) * kListBlock + threadIdx.x,
                      row_sh + (R ? 0u : threadIdx.x / G * kLaneRowWords));
}

// ---- one thread per query --------------------------------------------------------------------
template <int KMAX>
static __device__ __noinline__ void lists_exact(int k, V3 p, unsigned self_id, const Grid& g, Box b,
                                                const unsigned* start,
                                                const float4* pos_id, unsigned* col) {
    knn_neighbours_exact<KMAX>(k, p, self_id, g, b, 0u, start, pos_id, col, kListBlock);
}

// A warp with this many queries to search again lets each thread search its
// own (a whole warp per query costs about 150 of its instructions a chunk of
// 32 candidates; one thread about 130 a candidate, all lanes at once).
constexpr unsigned kListsRedoThreads = 12;

template <int KMAX, bool FLAT>
__device__ __forceinline__ void lists_thread(const KnnPair& pr, const Grid& grid, unsigned s,
                                             unsigned* sh) {
    const bool act = s < pr.nA;
    const float4 v = pr.a_pos_id[act ? s : pr.nA - 1];
    const V3 p = v3(v);
    const unsigned a = __float_as_uint(v.w), self_id = pr.self ? a : UINT_MAX;
    unsigned ix, iy, iz;
    cell_coords(grid, p, ix, iy, iz);
    const Box box = cell_box(grid, ix, iy, iz, 1);
    unsigned* col = sh + threadIdx.x;
    bool ok = true;
    if (act) {
        if constexpr (FLAT)
            ok = knn_neighbours_flat<KMAX, 8>(int(pr.k), p, self_id, grid, box, 0u, pr.b_start,
                                              pr.b_pos_id, col, kListBlock);
        else
            ok = knn_neighbours_stream<KMAX, 8>(int(pr.k), p, self_id, grid, box, 0u, pr.b_start,
                                                pr.b_pos_id, col, kListBlock);
    }
    __syncwarp();
    unsigned redo = __ballot_sync(kAllLanes, !ok);
    if (__popc(redo) >= int(kListsRedoThreads)) {
        if (!ok) lists_exact<KMAX>(int(pr.k), p, self_id, grid, box, pr.b_start, pr.b_pos_id, col);
    } else {
        const unsigned lane = threadIdx.x & 31u;
        for (; redo; redo &= redo - 1u) {
            const int from = __ffs(int(redo)) - 1;
            const V3 rp = lanes_get<32>(p, unsigned(from));
            const unsigned id = __shfl_sync(kAllLanes, self_id, from);
            cell_coords(grid, rp, ix, iy, iz);
            const LaneEntry<32> e =
                lanes_knn<32, FLAT ? 3 : 9>(pr.k, lane, rp, id, grid, cell_box(grid, ix, iy, iz, 1),
                                            0u, pr.b_start, pr.b_pos_id);
            if (lane < pr.k) sh[(threadIdx.x & ~31u) + unsigned(from) + lane * kListBlock] = e.slot;
            __syncwarp();
        }
    }
    if (!act) return;
    for (unsigned r = 0; r < pr.k; ++r) {
        const unsigned bs = col[r * kListBlock];
        const float4 q = bs == UINT_MAX ? make_float4(0.f, 0.f, 0.f, 0.f) : pr.b_pos_id[bs];
        put_entry(pr, a, r, bs == UINT_MAX ? UINT_MAX : __float_as_uint(q.w),
                  bs == UINT_MAX ? FLT_MAX : distance(p, v3(q)));
    }
}

template <int KMAX, bool FLAT>
__global__ void __launch_bounds__(kListBlock) k_lists_thread(KnnPair pr, Grid grid) {
    after_previous();
    __shared__ unsigned sh[KMAX * kListBlock];
    lists_thread<KMAX, FLAT>(pr, grid, blockIdx.x * kListBlock + threadIdx.x, sh);
}

template <int KMAX, bool FLAT>
__global__ void __launch_bounds__(kListBlock) k_lists_thread_pairs(const __grid_constant__ KnnPairs P) {
    after_previous();
    __shared__ unsigned sh[KMAX * kListBlock];
    const KnnPair& pr = P.pair[pair_of_block(P)];
    lists_thread<KMAX, FLAT>(pr, P.grid, (blockIdx.x - pr.block_begin) * kListBlock + threadIdx.x,
                             sh);
}

// 32 < k <= 64: a warp per query, two ranks a lane.  One thread per query on a
// register list of 64 keys was one long chain whatever its box held (k = 40, 13
// candidates to a box: 3,000 queries 76.5 us, 131,072 231).
template <int R>
__device__ __forceinline__ void lists_wide(const KnnPair& pr, const Grid& grid, unsigned r,
                                           unsigned thread, unsigned* rows) {
    const unsigned lane = threadIdx.x & 31u, q = thread / 32u;
    const bool act = q < pr.nA;  // (whole warps)
    const float4 v = pr.a_pos_id[act ? q : pr.nA - 1];
    const V3 p = v3(v);
    const unsigned a = __float_as_uint(v.w), self_id = pr.self ? a : UINT_MAX;
    unsigned ix, iy, iz;
    cell_coords(grid, p, ix, iy, iz);
    LaneList<32, 2> list;
    list.e[0] = list.e[1] = KEY_EMPTY;
    lanes_box<32, R>(lane, grid, cell_box(grid, ix, iy, iz, r), 0u, pr.b_start, pr.b_pos_id, rows,
                     [&](float4 c, unsigned, bool ok, bool) {
                         const unsigned id = __float_as_uint(c.w);
                         const unsigned long long key = knn_key(distance(p, v3(c)), id);
                         list.take(ok && id != self_id && key < KEY_EMPTY ? key : KEY_EMPTY, pr.k,
                                   lane);
                     });
    if (!act) return;
#pragma unroll
    for (unsigned h = 0; h < 2; ++h) {
        const unsigned rank = 32u * h + lane;
        if (rank < pr.k) put_entry(pr, a, rank, key_id(list.e[h]), key_dist(list.e[h]));
    }
}

template <int R>
__global__ void __launch_bounds__(kListBlock) k_lists_wide(KnnPair pr, Grid grid, unsigned r) {
    after_previous();
    __shared__ unsigned row_sh[R ? 1 : kListBlock / 32 * kLaneRowWords];
    lists_wide<R>(pr, grid, r, blockIdx.x * kListBlock + threadIdx.x,
                  row_sh + (R ? 0u : threadIdx.x / 32u * kLaneRowWords));
}
template <int R>
__global__ void __launch_bounds__(kListBlock) k_lists_wide_pairs(const __grid_constant__ KnnPairs P) {
    after_previous();
    __shared__ unsigned row_sh[R ? 1 : kListBlock / 32 * kLaneRowWords];
    const KnnPair& pr = P.pair[pair_of_block(P)];
    lists_wide<R>(pr, P.grid, P.r, (blockIdx.x - pr.block_begin) * kListBlock + threadIdx.x,
                  row_sh + (R ? 0u : threadIdx.x / 32u * kLaneRowWords));
}

// ---- dispatch ----------------------------------------------------------------------------------
// Measured per call, start of the lists kernel / lanes / threads, boxes with
// about the neighbours asked for (us): k = 7, 4,096 queries 12.4 / 6.2 / 12.4,
// 65,536 25 / 14.5 / 16.5, 131,072 39 / 24.7 / 22.6, 262,144 68 / 43 / 37;
// k = 16, 65,536 41 / 26.7 / 28.8, 131,072 73 / 46.9 / 45.1, 262,144 115 / 91 /
// 74; k = 32, 4,096 61 / 8.3 / 30, 262,144 481 / 182 / 192 (the start: a
// 128 KB candidate table per block, one block on an SM).  Radius 2 boxes, up
// to 25 rows, have only the lanes: k = 16, 131,072 401 / 115.
static bool lists_on_lanes(size_t queries, unsigned k, unsigned r) {
    return r != 1 || k > 16 || queries <= 98304;
}

template <int G>
static void lists_lanes_go(const KnnPair& pr, const Grid& grid, unsigned r, cudaStream_t st) {
    const unsigned nb = blocks_for(pr.nA, kListBlock / G);
    if (r != 1) launch_after(k_lists_lanes<G, 0>, nb, kListBlock, 0, st, pr, grid, r);
    else if (grid.wc[1] == 1) launch_after(k_lists_lanes<G, 3>, nb, kListBlock, 0, st, pr, grid, r);
    else launch_after(k_lists_lanes<G, 9>, nb, kListBlock, 0, st, pr, grid, r);
}
template <int KMAX>
static void lists_thread_go(const KnnPair& pr, const Grid& grid, cudaStream_t st) {
    const unsigned nb = blocks_for(pr.nA, kListBlock);
    if (grid.wc[1] == 1) launch_after(k_lists_thread<KMAX, true>, nb, kListBlock, 0, st, pr, grid);
    else launch_after(k_lists_thread<KMAX, false>, nb, kListBlock, 0, st, pr, grid);
}

gs_status launch_knn_binned(const Database& A, unsigned nA, const Database& B, bool self,
                            unsigned r, unsigned k, unsigned* idx, float* dist, cudaStream_t st) {
    if (nA == 0) return GS_OK;
    const KnnPair pr{A.pos_id, B.start, B.pos_id, idx, dist, nA, k, 0u, self};
    if (k > 32) {
        const unsigned nb = blocks_for(nA, kListBlock / 32);
        if (r != 1) launch_after(k_lists_wide<0>, nb, kListBlock, 0, st, pr, B.grid, r);
        else if (B.grid.wc[1] == 1) launch_after(k_lists_wide<3>, nb, kListBlock, 0, st, pr, B.grid, r);
        else launch_after(k_lists_wide<9>, nb, kListBlock, 0, st, pr, B.grid, r);
    } else if (lists_on_lanes(nA, k, r)) {
        if (k <= 8) lists_lanes_go<8>(pr, B.grid, r, st);
        else if (k <= 16) lists_lanes_go<16>(pr, B.grid, r, st);
        else lists_lanes_go<32>(pr, B.grid, r, st);
    } else {
        if (k <= 8) lists_thread_go<8>(pr, B.grid, st);
        else lists_thread_go<16>(pr, B.grid, st);
    }
    GS_LAUNCHED("knn_binned");
    return GS_OK;
}

static_assert(sizeof(KnnPairs) <= 4096, "batched KNN parameters exceed 4 KiB");

template <int G>
static void pairs_lanes_go(const KnnPairs& P, unsigned nb, cudaStream_t st) {
    if (P.r != 1) launch_after(k_lists_lanes_pairs<G, 0>, nb, kListBlock, 0, st, P);
    else if (P.grid.wc[1] == 1) launch_after(k_lists_lanes_pairs<G, 3>, nb, kListBlock, 0, st, P);
    else launch_after(k_lists_lanes_pairs<G, 9>, nb, kListBlock, 0, st, P);
}
template <int KMAX>
static void pairs_thread_go(const KnnPairs& P, unsigned nb, cudaStream_t st) {
    if (P.grid.wc[1] == 1) launch_after(k_lists_thread_pairs<KMAX, true>, nb, kListBlock, 0, st, P);
    else launch_after(k_lists_thread_pairs<KMAX, false>, nb, kListBlock, 0, st, P);
}

gs_status launch_knn_binned_pairs(KnnPairs& P, cudaStream_t st) {
    if (P.n_pairs == 0 || P.n_pairs > kMaxKnnPairs)
        return fail(GS_ERR_INVALID_ARG, "between 1 and 49 group pairs per batched KNN");
    unsigned kmax = 0;
    size_t queries = 0;
    for (unsigned q = 0; q < P.n_pairs; ++q) {
        kmax = std::max(kmax, P.pair[q].k);
        queries += P.pair[q].nA;
    }
    const unsigned G = kmax <= 8 ? 8 : kmax <= 16 ? 16 : 32;
    // (beyond k = 32 a warp per query)
    const bool lanes = kmax > 32 || lists_on_lanes(queries, kmax, P.r);
    unsigned blocks = 0;
    for (unsigned q = 0; q < P.n_pairs; ++q) {
        P.pair[q].block_begin = blocks;
        blocks += blocks_for(P.pair[q].nA, lanes ? kListBlock / G : kListBlock);
    }
    if (blocks == 0) return GS_OK;
    if (kmax > 32) {
        if (P.r != 1) launch_after(k_lists_wide_pairs<0>, blocks, kListBlock, 0, st, P);
        else if (P.grid.wc[1] == 1) launch_after(k_lists_wide_pairs<3>, blocks, kListBlock, 0, st, P);
        else launch_after(k_lists_wide_pairs<9>, blocks, kListBlock, 0, st, P);
    } else if (lanes) {
        if (G == 8) pairs_lanes_go<8>(P, blocks, st);
        else if (G == 16) pairs_lanes_go<16>(P, blocks, st);
        else pairs_lanes_go<32>(P, blocks, st);
    } else {
        if (G == 8) pairs_thread_go<8>(P, blocks, st);
        else pairs_thread_go<16>(P, blocks, st);
    }
    GS_LAUNCHED("knn_binned_pairs");
    return GS_OK;
}

}  // namespace gs
