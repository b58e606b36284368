// Counting-sort databases built by one thread-block cluster each.
#pragma once

#include "gs_internal.cuh"

namespace gs {

// One database to build: count cells (wrapping the positions first when
// wrap_mode >= 0, and clearing `applied` when given), scan, scatter.
struct DbJob {
    float4* pos;
    unsigned n;
    Grid grid;            // or chosen by the kernel: auto_axis[0] != 0
    unsigned auto_axis[3];  // cells per axis when 1, 2 or 3 axes have extent
    Grid* grid_out;       // the chosen grid
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
