// The fused step on cell tables (gs_table.cu).
#pragma once

#include "gs_launch.h"

namespace gs {

// One step's buffers.  tab / cnt: this step's rows, one a cell and then the
// further ones, and the cells' counts; tag: what each further row is; *_next
// the ones it fills, *_clear the counts and tags it clears.
struct TableStep {
    const float4 *f0, *f1;
    float4 *f0_next, *f1_next, *f2, *f3, *f4;
    const float4* f5;
    const float4* tab;
    const unsigned* cnt;
    const unsigned* tag;
    float4* tab_next;
    unsigned* cnt_next;
    unsigned* tag_next;
    unsigned *cnt_clear, *tag_clear;
    WallRefs walls;
    float4 *w0, *w1, *w2;
    unsigned* near;    // [n * k] neighbour lists, agent by agent (walls)
    float* near_dist;
    unsigned n, cells, row_log2, ext_log2;
    Scene sc;
};

gs_status table_init(GroupView g, const TableStep& T, int wrap_mode, bool dirty, float4* f5,
                     unsigned* redo_count, cudaStream_t st);
// hook (may be null) brackets the launches as phases 2 and 3.
gs_status table_step(const TableStep& T, const StepDev& p, cudaStream_t st, PhaseHook* hook);
// Mean velocity per cell of the step that T described (its f1_next holds the
// agents' new state).
gs_status table_avg_velocity(const TableStep& T, float3* out, cudaStream_t st);

}  // namespace gs
