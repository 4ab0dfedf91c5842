// emv_batch_types.h -- descriptors of the batched solver (host and device).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace emv {

constexpr int BATCH_KMAX = 12;
constexpr int32_t BATCH_SMEM_BYTES = 200 * 1024;  // admission: 2^k rows of 32 vertices and two rows of n
constexpr int32_t BATCH_MW_MAX = 8;      // widest merge vertex block that it tries: 8 columns of 32 vertices
constexpr int BATCH_SIZES = 8;           // team sizes 128, 64, .. 1

// Table stride of an instance: whole 16-byte quads.
__host__ __device__ constexpr int32_t batch_ld(int32_t n) { return (n + 3) / 4 * 4; }

struct BatchInst {
    const int32_t *row_ptr;  // n + 1 entries, arcs of this instance from 0
    const int2 *adj;         // packed (col, w) arcs
    const int32_t *terms;    // k terminals
    int32_t *table;          // 2^kt rows of batch_ld(n) int32
    int32_t n;
    int32_t k;
    int32_t kt;              // terminals whose subsets are solved: k, or table_terminals(k) when only the cost is wanted
    int32_t size;            // CTAs of its team (1 << a class)
    int32_t rows;            // most rows of a closure
    int32_t mw;              // vertices of a merge block
    int32_t narrow;          // every weight fits a packed arc
    uint32_t inv_slices;     // ResInst::inv_slices
    int32_t orig;            // slot of the cost in BatchArgs::costs
    int32_t lo;              // first level to run (1..kt)
    int32_t hi;              // last level to run (lo..kt)
    uint32_t spin_limit;     // ResTeam::limit
    int32_t hub_min;         // ResInst::hub_min
    int32_t pad;
    char *slices;            // its sliced arcs, or null: in BatchArgs::scratch
};

struct BatchArgs {
    const BatchInst *inst;   // by class
    const uint32_t *xs;      // subsets by level for k = 1..BATCH_KMAX, concatenated
    const int32_t *xs_off;   // xs_off[k * (BATCH_KMAX + 2) + m]: start of level m of k
    int64_t *costs;          // by orig; written when hi == kt
    uint32_t *ctl;           // lines of 32 words: status, a queue per class, a barrier per team; zero at launch
    char *scratch;           // sliced arcs, scratch_stride bytes for every CTA (a team uses its first CTA's)
    int64_t scratch_stride;
    int32_t smem;            // dynamic shared memory
    int32_t end[BATCH_SIZES];  // class c: instances [end[c - 1], end[c])
    int32_t pad;
};

// Lines of BatchArgs::ctl for a grid of at most `blocks` CTAs.
constexpr int32_t batch_ctl_lines(int32_t blocks) { return 1 + BATCH_SIZES + 2 * blocks; }

}  // namespace emv
