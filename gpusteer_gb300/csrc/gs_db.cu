// updateKNNDatabase for small groups: the whole counting sort in one launch.
//
// The rebuild's three passes (count, exclusive scan, scatter) each depend on
// all of the one before, so over the whole chip they are five launches, about
// 20 us whatever the size of a small group.  A cluster of 16 blocks on one GPC
// runs them with hardware barriers between (no block waits on one that may not
// be running: a cluster's blocks are resident together), and several groups'
// databases are several clusters of one launch.
#include <cooperative_groups.h>

#include "gs_db.cuh"
#include "gs_launch.h"

namespace cg = cooperative_groups;

namespace gs {

constexpr unsigned kDbThreads = 1024;
constexpr unsigned kDbCluster = 16;

// Counts and starts are written by other SMs during the launch: read past L1.
__device__ __forceinline__ uint4 load_counts(const unsigned* count, unsigned i, unsigned end) {
    if (i + 4 <= end) return __ldcg(reinterpret_cast<const uint4*>(count + i));
    uint4 v = make_uint4(0u, 0u, 0u, 0u);
    if (i < end) v.x = __ldcg(count + i);
    if (i + 1 < end) v.y = __ldcg(count + i + 1);
    if (i + 2 < end) v.z = __ldcg(count + i + 2);
    return v;
}

// Exclusive prefix of v over the block, and the block's total.
__device__ __forceinline__ unsigned block_scan(unsigned v, unsigned* warp_sums, unsigned& total) {
    const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= unsigned(o)) x += y;
    }
    if (lane == 31) warp_sums[warp] = x;
    __syncthreads();
    if (warp == 0) {
        unsigned w = warp_sums[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const unsigned y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= unsigned(o)) w += y;
        }
        warp_sums[lane] = w;
    }
    __syncthreads();
    total = warp_sums[31];
    const unsigned before = warp ? warp_sums[warp - 1] : 0u;
    __syncthreads();
    return before + x - v;
}

// The grid of a sample of kSample positions spread evenly over the agents, by
// one block; every block of a cluster computes the same.  Per axis, a centre and
// a reach start from all of the sample; each round takes the mean and four times
// the mean distance from the centre of what lies within the reach, so that a few
// positions far off, at whatever distance, drop out and a box or a cloud keeps
// everything.  The sample's extent within the last reach, a little widened, is
// the axis' (a grid over the extent of all positions, about the origin, lost
// most of its cells to one far position, to one that is not finite, or to a
// crowd far from the origin: 65,536 agents, k = 16, 9.2 ms for each of these
// and 0.1 ms for a cube about the origin).
constexpr unsigned kSample = 256;
constexpr int kSampleRounds = 4;
struct Sample {
    float x[3][kSample];                   // NaN: not a finite position
    float low[3], high[3], count[3];
};
template <class Op>
__device__ __forceinline__ float warp_all(float v, Op op) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ AutoGrid automatic_grid(const float4* pos, unsigned n,
                                                   const unsigned axis_cells[3], Sample& sh) {
    const unsigned t = threadIdx.x, lane = t & 31u, warp = t >> 5, take = min(n, kSample);
    constexpr float kScale = 0x1p-12f;  // sums of the largest floats stay finite
    if (t < kSample) {
        const V3 p = v3(pos[t < take ? size_t(t) * n / take : 0]);
        const bool ok = t < take && is_finite(p);
        const float none = __int_as_float(0x7fffffff);
        sh.x[0][t] = ok ? p.x * kScale : none;
        sh.x[1][t] = ok ? p.y * kScale : none;
        sh.x[2][t] = ok ? p.z * kScale : none;
    }
    __syncthreads();
    if (warp < 3) {  // a warp an axis
        const auto sum = [](float u, float v) { return u + v; };
        const auto least = [](float u, float v) { return fminf(u, v); };
        const auto most = [](float u, float v) { return fmaxf(u, v); };
        float x[kSample / 32];
#pragma unroll
        for (unsigned i = 0; i < kSample / 32; ++i) x[i] = sh.x[warp][32 * i + lane];
        float centre = 0.f, reach = FLT_MAX;
        for (int round = 0; round < kSampleRounds; ++round) {
            float m = 0.f, u = 0.f, v = 0.f;
#pragma unroll
            for (unsigned i = 0; i < kSample / 32; ++i) {
                const float d = x[i] - centre;
                const bool in = fabsf(d) <= reach;
                m += in ? 1.f : 0.f;
                u += in ? d : 0.f;
                v += in ? fabsf(d) : 0.f;
            }
            m = warp_all(m, sum);
            u = warp_all(u, sum);
            v = warp_all(v, sum);
            if (m > 0.f) {
                centre += u / m;
                reach = 4.f * (v / m);
            }
        }
        float m = 0.f, low = FLT_MAX, high = -FLT_MAX;
#pragma unroll
        for (unsigned i = 0; i < kSample / 32; ++i) {
            const bool in = fabsf(x[i] - centre) <= reach;
            m += in ? 1.f : 0.f;
            low = in ? fminf(low, x[i]) : low;
            high = in ? fmaxf(high, x[i]) : high;
        }
        m = warp_all(m, sum);
        low = warp_all(low, least);
        high = warp_all(high, most);
        if (lane == 0) {
            sh.low[warp] = m > 0.f ? low : 0.f;
            sh.high[warp] = m > 0.f ? high : 0.f;
            sh.count[warp] = m;
        }
    }
    __syncthreads();
    AutoGrid g;
    float width[3], most = 0.f;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        width[a] = (sh.high[a] - sh.low[a]) * (1.f + 2.f / fmaxf(sh.count[a], 2.f));
        most = fmaxf(most, width[a]);
    }
    int dims = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a) dims += width[a] > 1e-3f * most;
    const unsigned cells = dims == 1 ? axis_cells[0] : dims == 2 ? axis_cells[1] : axis_cells[2];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        g.grid.wc[a] = width[a] > 1e-3f * most ? cells : 1u;
        g.grid.ws[a] = fminf(fmaxf(width[a], 1e-30f), FLT_MAX * kScale * 0.25f) * (1.f / kScale);
        g.mid[a] = (0.5f * sh.low[a] + 0.5f * sh.high[a]) * (1.f / kScale);
    }
    return g;
}

__global__ void __launch_bounds__(kDbThreads) k_db_cluster(const __grid_constant__ DbJobs J) {
    after_previous();
    __shared__ unsigned ws[32];
    __shared__ unsigned totals[kDbCluster];
    __shared__ Sample sample;
    cg::cluster_group cluster = cg::this_cluster();
    const unsigned R = cluster.num_blocks(), rank = cluster.block_rank(), t = threadIdx.x;
    const DbJob& j = J.job[blockIdx.x / R];
    const unsigned first = rank * kDbThreads + t, step = R * kDbThreads, n = j.n;
    const bool automatic = j.auto_axis[0] != 0;
    AutoGrid a{j.grid, {0.f, 0.f, 0.f}};
    if (first == 0 && j.zero) *j.zero = 0ull;
    if (automatic) {
        a = automatic_grid(j.pos, n, j.auto_axis, sample);
        if (first == 0) *j.grid_out = a;
    }
    const unsigned cells = a.grid.wc[0] * a.grid.wc[1] * a.grid.wc[2];
    const unsigned C = cells + (automatic ? 1u : 0u);
    for (unsigned i = first; i < n; i += step) {
        V3 p = v3(j.pos[i]);
        if (j.wrap_mode >= 0) {
            p = wrap_world(p, j.wrap_ws, j.wrap_mode);
            j.pos[i] = f4(p, 0.f);
        }
        unsigned c;
        if (automatic) {
            unsigned x, y, z;
            auto_coords(a, p, x, y, z);
            c = is_finite(p) ? cell_label(a.grid, x, y, z) : cells;
        } else {
            c = cell_of(a.grid, p);
        }
        j.cell[i] = c;
        j.rank[i] = atomicAdd(j.count + c, 1u);
        if (j.applied) j.applied[i] = 0u;
    }
    cluster.sync();
    // this block's run of cells: its total, then its starts
    const unsigned per = ((C + R - 1) / R + 3u) & ~3u;
    const unsigned c0 = min(rank * per, C), c1 = min(c0 + per, C);
    unsigned sum = 0;
    for (unsigned i = c0 + 4 * t; i < c1; i += 4 * kDbThreads) {
        const uint4 v = load_counts(j.count, i, c1);
        sum += v.x + v.y + v.z + v.w;
    }
    unsigned total;
    block_scan(sum, ws, total);
    if (t < R) cluster.map_shared_rank(totals, t)[rank] = total;
    cluster.sync();
    unsigned base = 0;
    for (unsigned q = 0; q < rank; ++q) base += totals[q];
    for (unsigned b = c0; b < c1; b += 4 * kDbThreads) {
        const unsigned i = b + 4 * t;
        const uint4 v = load_counts(j.count, i, c1);
        unsigned run = base + block_scan(v.x + v.y + v.z + v.w, ws, total);
        const uint4 s = make_uint4(run, run + v.x, run + v.x + v.y, run + v.x + v.y + v.z);
        if (i + 4 <= c1) {
            *reinterpret_cast<uint4*>(j.start + i) = s;
            *reinterpret_cast<uint4*>(j.count + i) = make_uint4(0u, 0u, 0u, 0u);
        } else {
            if (i < c1) {
                j.start[i] = s.x;
                j.count[i] = 0u;
            }
            if (i + 1 < c1) {
                j.start[i + 1] = s.y;
                j.count[i + 1] = 0u;
            }
            if (i + 2 < c1) {
                j.start[i + 2] = s.z;
                j.count[i + 2] = 0u;
            }
        }
        base += total;
    }
    if (first == 0) j.start[C] = n;
    cluster.sync();
    for (unsigned i = first; i < n; i += step) {
        const unsigned dst = __ldcg(j.start + j.cell[i]) + j.rank[i];
        if (dst >= n) continue;
        const float4 p = j.pos[i];
        if (j.sorted) j.sorted[dst] = i;
        j.pos_id[dst] = make_float4(p.x, p.y, p.z, __uint_as_float(i));
    }
}

DbJob db_job(Database& db, const float4* pos, unsigned n, const Grid& grid) {
    DbJob j;
    std::memset(static_cast<void*>(&j), 0, sizeof(j));
    j.pos = const_cast<float4*>(pos);  // written only when wrap_mode >= 0
    j.n = n;
    j.grid = grid;
    j.wrap_mode = -1;
    j.cell = db.cell;
    j.rank = db.rank;
    j.sorted = db.sorted;
    j.start = db.start;
    j.count = db.count;
    j.pos_id = db.pos_id;
    return j;
}

// Rebuild, cluster / five launches (us): 16,384 agents on 32,768 cells 10.6 /
// 20.6, 32,768 on 64,000 14.4 / 20.6, 65,536 on 132,651 22.6 / 20.6.
bool db_on_cluster(unsigned n, unsigned C) { return n <= 32768 && C <= 131072; }

gs_status db_build_clusters(const DbJobs& J, unsigned count, cudaStream_t st) {
    if (count == 0) return GS_OK;
    if (count > kMaxDbJobs) return fail(GS_ERR_INVALID_ARG, "too many databases in one launch");
    // 16 blocks a cluster is past the portable 8: allowed per kernel and device
    GS_CUDA(cudaFuncSetAttribute(k_db_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kDbCluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;  // as launch_after
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kDbCluster * count);
    cfg.blockDim = dim3(kDbThreads);
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    GS_CUDA(cudaLaunchKernelEx(&cfg, k_db_cluster, J));
    return GS_OK;
}

}  // namespace gs
