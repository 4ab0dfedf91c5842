// emv_resident.h -- the one-launch solver of small instances (host side).
#pragma once

#include "emv_common.cuh"
#include "emv_solver.h"

constexpr int32_t RESIDENT_SMEM = 224 * 1024;

struct ResidentPlan {
    int blocks;              // CTAs
    int32_t rows;            // rows of the widest level's largest share
    int32_t mw;              // vertices of a merge block
};

// Rows of the widest level of kt terminals' subsets.
int64_t resident_max_rows(int32_t kt);
// Whether the device functions of emv_resident.cuh can take the instance.
bool resident_fits(int32_t n, int32_t kt);
// Vertices of a merge block when `ctas` CTAs share the instance: as few waves
// of blocks as the shared memory allows, and within them the narrowest blocks,
// so that every CTA has some; cap > 0 bounds it.
int32_t resident_merge_width(int32_t n, int32_t kt, int32_t ctas, int32_t cap);
uint32_t res_inv_slices(int32_t n);
int32_t res_hub_min(int32_t n, int64_t arcs, int32_t kt);
// Polls after which a CTA gives up on the others of its team: CTAs without rows
// of a level wait for those that close `rows` of them.
uint32_t res_spin_limit(int32_t n, int64_t arcs, int64_t rows);
// crowded: the graph is known to have vertices of far more arcs than most.
bool resident_plan(const emv_ctx *c, int32_t n, int64_t arcs, int32_t kt, bool host_table, bool crowded, ResidentPlan &p);
// Enqueues the whole DP over the first kt of the k terminals, CSR check
// included, and the copy of its result words; fills the table's 2^kt rows
// (stride ld) and c->adj.
int resident_launch(emv_ctx *c, const ResidentPlan &p, int32_t n, int64_t arcs, const int32_t *row_ptr,
                    const int32_t *col, const int32_t *w, const int32_t *terms, int32_t k, int32_t kt, int32_t *table,
                    int64_t ld, bool check, cudaStream_t st);
// Status, cost and times once the stream has been waited for (with spanned
// set, a vertex that no terminal reaches is EMV_ERR_DISCONNECTED).
int resident_finish(emv_ctx *c, int32_t n, int32_t k, bool check, bool spanned, int64_t *cost_out, emv_timing *tm);
// Device words of the launch: the terminals, and two that are 0 where the table
// has been filled (the error word, and whether the CSR check refused the graph).
struct ResidentWords {
    const int32_t *terms;
    const uint32_t *err, *refused;
};
ResidentWords resident_words(const emv_ctx *c);
// Status of a device CSR check (emv_device.cu).
int scan_status(const emv::GraphScan &s, int32_t n);
