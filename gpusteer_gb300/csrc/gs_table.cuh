// The fused step on cell tables (gs_table.cu).
#pragma once

#include "gs_launch.h"

namespace gs {

// One step's buffers.  tab / cnt / over: this step's table, counts and
// overflow list; *_next the ones it fills, *_clear the counts it clears.
struct TableStep {
    const float4 *f0, *f1;
    float4 *f0_next, *f1_next, *f2, *f3, *f4;
    const float4* f5;
    const float4* tab;
    const unsigned* cnt;
    const float4* over;
    const unsigned* over_n;
    float4* tab_next;
    unsigned* cnt_next;
    float4* over_next;
    unsigned* over_n_next;
    unsigned *cnt_clear, *over_n_clear;
    WallRefs walls;
    float4 *w0, *w1, *w2;
    unsigned* near;    // [n * k] neighbour lists, agent by agent (walls)
    float* near_dist;
    unsigned n, cells, row_log2;
    Scene sc;
};

gs_status table_init(GroupView g, const TableStep& T, int wrap_mode, bool dirty, float4* f5,
                     unsigned* redo_count, cudaStream_t st);
gs_status table_step(const TableStep& T, const StepDev& p, cudaStream_t st);
// Mean velocity per cell of the step that T described (its f1_next holds the
// agents' new state).
gs_status table_avg_velocity(const TableStep& T, float3* out, cudaStream_t st);

}  // namespace gs
