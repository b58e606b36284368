// Counting-sort databases built by one thread-block cluster each.
#pragma once

#include <cfloat>

#include "gs_internal.cuh"

namespace gs {

// An automatic grid: even cells about `mid` over where most positions lie; what
// lies outside is in the cells at its edges, as everywhere.
struct AutoGrid {
    Grid grid;
    float mid[3];
};
// Grows with every coordinate over all floats: so do the difference, rounded,
// and cell_coord.
GS_HD void auto_coords(const AutoGrid& a, V3 p, unsigned& ix, unsigned& iy, unsigned& iz) {
    cell_coords(a.grid, sub(p, v3(a.mid[0], a.mid[1], a.mid[2])), ix, iy, iz);
}
GS_HD bool is_finite(V3 p) {
    return fabsf(p.x) <= FLT_MAX && fabsf(p.y) <= FLT_MAX && fabsf(p.z) <= FLT_MAX;
}

// One database to build: count cells (wrapping the positions first when
// wrap_mode >= 0, and clearing `applied` when given), scan, scatter.
struct DbJob {
    float4* pos;
    unsigned n;
    Grid grid;            // or chosen by the kernel: auto_axis[0] != 0
    unsigned auto_axis[3];  // cells per axis when 1, 2 or 3 axes have extent
    AutoGrid* grid_out;   // the chosen grid; positions that are not finite are
                          // in a cell past its last
    unsigned long long* zero;  // a word to clear (may be null)
    int wrap_mode;        // -1: positions stay as they are
    float wrap_ws[3];
    unsigned* applied;    // may be null
    unsigned *cell, *rank, *sorted, *start, *count;
    float4* pos_id;
};
constexpr unsigned kMaxDbJobs = 7;
struct DbJobs {
    DbJob job[kMaxDbJobs];
};

DbJob db_job(Database& db, const float4* pos, unsigned n, const Grid& grid);
// Builds `count` databases in one launch, a cluster each.
gs_status db_build_clusters(const DbJobs& J, unsigned count, cudaStream_t st);
// Sizes at which one cluster is faster than a launch over the whole chip per pass.
bool db_on_cluster(unsigned n, unsigned C);

}  // namespace gs
