// emv_batch_host.h -- host helpers of the batched launch, shared with the server.
#pragma once

#include <chrono>
#include <functional>
#include <vector>

#include "emv_batch_types.h"
#include "emv_solver.h"

struct BatchPack {
    int32_t lane = 0;                  // emv_ctx::blane
    std::vector<emv::BatchInst> desc;  // in launch order
    std::vector<int64_t> row_off, arc_off, term_off, table_off;  // into the packed device buffers
    int64_t rows = 0, arcs = 0, terms = 0, table_words = 0;
    int32_t count = 0;
    int32_t blocks = 0;                // CTAs of the launch
    int32_t end[emv::BATCH_SIZES] = {};  // classes (BatchArgs::end)
    int64_t arc_bytes = 0;             // largest sliced arcs
    int32_t rcap_used = 0;
    int64_t cost_slots = 0;            // entries the device cost array needs (max orig + 1)
    int32_t *h_row = nullptr;          // views into the pinned staging buffer
    int2 *h_adj = nullptr;
    int32_t *h_term = nullptr;
    emv::BatchInst *h_desc = nullptr;
    std::chrono::steady_clock::time_point t_upload_end;
};

int32_t batch_class_of(int32_t n, int32_t k);
bool batch_fits(int32_t n, int32_t k);
// What the kernel needs to know of a host graph beyond its sizes.
struct BatchGraph {
    bool narrow = false;      // every weight fits a packed arc
    int64_t arc_bytes = 0;    // sliced arcs
};
BatchGraph batch_graph(const int32_t *row_ptr, int32_t n, uint32_t largest_weight, int32_t hub_min);
// Packs the arcs; returns their largest weight.
uint32_t pack_arcs(const emv_graph &g, int2 *adj);
// Estimated time (us) of levels lo..hi on one CTA.
double batch_work(int32_t n, int32_t kt, int64_t arcs, int32_t lo, int32_t hi);
// Team sizes (at most max_size) for a grid of `blocks` CTAs and the order by
// class (then largest first): order[j] is the input's index, size[] by input index.
void batch_plan(const std::vector<double> &work, const std::vector<int64_t> &states, int32_t blocks, int32_t max_size,
                std::vector<int32_t> &order, std::vector<int32_t> &size);
// Fills the fields that follow from n, k, kt, the arcs and the team size.
void batch_shape(const emv_ctx *c, int64_t arcs, emv::BatchInst &d);
int prepare_batch_subsets(emv_ctx *c, cudaStream_t st);
int batch_kernel_setup(emv_ctx *c);
// Team sizes and launch order of the instances ids[] (blocks > 0: single-CTA
// teams in the given order, for a launch of that many CTAs).  whole: solve the
// subsets of all terminals (the tables are wanted), else those the costs need.
struct BatchOrder {
    std::vector<int32_t> ids, size;  // in launch order
    std::vector<double> work;
};
BatchOrder batch_order(const emv_ctx *c, const emv_instance *inst, const std::vector<int32_t> &ids, bool whole,
                       int32_t blocks);
// Lays out entries [from, to) of an order for one launch, and reserves staging.
int batch_layout(emv_ctx *c, const emv_instance *inst, const BatchOrder &ord, int32_t from, int32_t to, bool whole,
                 int32_t blocks, BatchPack &pk);
// Fills the staging from the instances; check(i) is called for each before it
// is read and says whether to.
int batch_fill(emv_ctx *c, const emv_instance *inst, BatchPack &pk, const std::function<bool(int32_t)> &check);
// spare: buffers that grow take a quarter more where it is free.
int batch_upload(emv_ctx *c, BatchPack &pk, bool spare, cudaStream_t st);
emv::BatchArgs batch_args(emv_ctx *c, const BatchPack &pk);
// lines: control lines to reset, batch_ctl_lines(blocks) or more.
int launch_batch(emv_ctx *c, const emv::BatchArgs &a, int32_t blocks, int32_t lines, cudaStream_t st);
int batch_graph_launch(emv_ctx *c, int32_t lane, const emv::BatchArgs &a, int32_t blocks, cudaStream_t st);
// Bytes of BatchArgs::scratch for every CTA, from the largest sliced arcs.
int64_t batch_arc_stride(int64_t arc_bytes);
// CTAs for instances whose team sizes sum to ctas.
int32_t batch_blocks(const emv_ctx *c, int64_t ctas, int32_t cap);
