// emv_solver.h -- the solver context and the host-side helpers of the GPU DP.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "emv_internal.h"
#include "emv_plan.h"

#define CUDA_TRY(x)                                                                                        \
    do {                                                                                                   \
        cudaError_t e_ = (x);                                                                              \
        if (e_ != cudaSuccess) {                                                                           \
            cudaGetLastError();                                                                            \
            return emv_fail(EMV_ERR_CUDA, "%s: %s (%s:%d)", #x, cudaGetErrorString(e_), __FILE__, __LINE__); \
        }                                                                                                  \
    } while (0)

// A device allocation that only grows (freed on context destruction).
struct DevBuf {
    void *ptr = nullptr;
    size_t bytes = 0;
};

int dev_reserve(DevBuf &b, size_t bytes);
void dev_release(DevBuf &b);

constexpr int MAX_EVENTS = 64;
// emv_ctx::pinned: scalars of run_dp, then the one-launch solver's and the traceback's results
constexpr size_t PINNED_RES = 2048, PINNED_TB = 4096, PINNED_BYTES = 32768;
constexpr int NARROW_VARIANTS = 4;  // narrow-record kernels by width (narrow_fns)
constexpr int RELAX_VARIANTS = 20;  // relaxation kernels by record width and hubs (relax_fns)
constexpr int BATCH_CLASSES = 12;  // (n bucket 0..3) x (k bucket 0..2)

// One launch of the streamed merge: subsets [x0, x0 + cnt) of a level, its
// phases and its dynamic shared memory.
struct StreamGroup {
    int64_t x0, cnt, phase_off, nphase, smem;
};

// The block merge of a level.
struct BlockLevel {
    int64_t phase_off = 0, nphase = 0, rows = 0;
    bool split = false;
};

// Everything the DP needs per k, built once per k and context: the subsets by
// level, the pair and override slots of the staged-all-rows merge and the
// streamed merge's groups and phases.
struct KPlan {
    std::vector<uint32_t> xs_host;
    std::vector<int64_t> xs_off;   // level m occupies xs[off[m], off[m+1])
    DevBuf xs;                     // subsets by level
    DevBuf mpairs, movr;           // merge pair slots and override slots, all levels
    std::vector<int64_t> mpair_base, movr_base;  // per level
    DevBuf mstream_data, mstream_phases;
    std::vector<std::vector<StreamGroup>> mstream_groups;  // per level (none = not streamed)
    DevBuf mblock_data, mblock_phases;
    std::vector<BlockLevel> mblock_levels;                 // per level (nphase 0 = no block merge)
};

// A captured launch of the batched kernel, and the node its arguments go into.
struct BatchGraphExec {
    cudaGraph_t graph = nullptr;
    cudaGraphNode_t node = nullptr;
    cudaGraphExec_t exec = nullptr;
    const void *ctl = nullptr;     // the control words it resets
};
void batch_graph_release(BatchGraphExec &G);

// Buffers of one launch of the batched kernel.  A large batch runs as two
// launches, so that the host packs the second while the first is on the GPU.
constexpr int BATCH_LANES = 2;
struct BatchLane {
    DevBuf row, adj, term, desc, table, ctrl, arcs;
    void *stage = nullptr;         // pinned staging of the packed instances
    size_t stage_bytes = 0;
    BatchGraphExec graph[2];       // single-CTA teams; teams (a cooperative launch)
};

struct emv_ctx {
    int device = 0;
    int sms = 0;
    int relax_blocks_max[RELAX_VARIANTS] = {};  // cooperative grid of each relaxation kernel
    int narrow_blocks_max[NARROW_VARIANTS] = {};  // and of each narrow-record kernel
    int relax_sm_cap = 0;          // > 0: relaxation grids sized for this many SMs (the server's large solves)
    int64_t l2_bytes = 0;
    int64_t sweep_limit = 0;       // relaxation sweeps per chunk, 0 = n + 1
    int32_t value_bits = 0;        // 0: 16-bit merge staging / relaxation records where bounded, 32: never
    bool merge16_last = false;     // the last launch_merge took the 16-bit kernel
    int64_t relax_arcs = 0;       // arcs of the graph being relaxed (dense-sweep threshold)
    DevBuf ctrl, stat;             // relaxation barrier words, solve status
    DevBuf lvlmax;                 // per level: largest value its merge (level 1: relaxation) wrote
    DevBuf shadow;                 // 16-bit copy of the relaxed rows (the 16-bit merge's staging source)
    cudaEvent_t evmax[EMV_MAX_K + 1] = {};  // level m's maximum has reached the pinned buffer
    DevBuf scratch, act;           // vertex-major chunk buffer, active flags
    DevBuf hubs;                   // vertices of many arcs of the graph being relaxed
    int32_t relax_nhubs = 0;       // and their number
    DevBuf mark;                   // per vertex: last sweep in which it changed, lowest and highest excess
    DevBuf adj;                    // packed (col, w) arcs
    DevBuf gscan;                  // GraphScan of the last packed graph (device admission check)
    DevBuf terms;                  // terminals
    DevBuf g_all;                  // device copy of a host CSR (row_ptr, col, w)
    void *g_stage = nullptr;       // pinned staging of small host CSRs
    DevBuf table;                  // DP table of emv_solve
    DevBuf tb_edges, tb_out, tb_work;
    std::vector<int32_t> forest;   // union-find of the tree's edges, -1 between calls
    int32_t *h_dist = nullptr;     // pinned distances of emv_sssp, h_dist_n of them
    int32_t h_dist_n = 0;
    void *pinned = nullptr;        // small pinned host buffer for scalar reads, PINNED_BYTES
    cudaEvent_t ev[MAX_EVENTS] = {};
    int32_t xs_k = -1;             // k of the current plan
    KPlan *kp = nullptr;           // plan of xs_k
    KPlan *kplans[EMV_MAX_K + 1] = {};  // plans of every k used so far
    bool merge_attr = false;
    DevBuf res_arcs, res_out;        // one-launch solver: sliced arcs, control and result words
    bool res_attr = false;
    int64_t launches = 0;
    // batched launch
    DevBuf bxs, bxs_off;           // subset lists of every k <= BATCH_KMAX
    bool bxs_ready = false;
    int batch_blocks = 0;
    BatchLane blane[BATCH_LANES];
    DevBuf b_costs;                // by the caller's instance index
    cudaStream_t bstream = nullptr;  // of the second lane
    cudaEvent_t bev[2] = {};       // the caller's stream reached, the second lane done
    int32_t tune_rcap[BATCH_CLASSES] = {};  // most rows of a closure per class (0: a CTA's share of the widest level)
    int32_t tune_mw[BATCH_CLASSES] = {};  // most vertices of a merge block per class, in 32s (0: what fits)
};

int prepare_subsets(emv_ctx *c, int32_t k, cudaStream_t st);
int reserve_relax(emv_ctx *c, int32_t n);
constexpr int32_t SWEEP_RATE = 3;  // sweeps of narrow records, or rounds in one launch, for one of k_relax
int32_t max_sweeps(const emv_ctx *c, int32_t n, int32_t rate);
int32_t relax_chunk_rows_level(const emv_ctx *c, int32_t n, bool u16, int64_t cnt);
