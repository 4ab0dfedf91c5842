// emv_batch.cuh -- the persistent kernel of batching and serving.
//
// Many independent instances of uneven n and k share one launch of a CTA per
// SM.  Every instance is solved by a team of CTAs with the device functions of
// emv_resident.cuh (rows of a level dealt out to the team, closures in shared
// memory; reader/reader-el.c:2033-2131).  The host sorts the instances into
// classes of team size 128, 64, .. 1: an instance that alone would take longer
// than its share of the whole batch gets a larger team, so that no CTA is left
// with one long instance at the end.  A CTA goes through the classes from the
// largest team size on; its teams are nested (CTAs [t * size, (t + 1) * size)),
// every class has a queue, and a class whose queue is empty is left for the
// next.  One team CTA solves n = 4096, k = 10 in 10 ms, sixteen in 0.8 ms.
// The table of an instance is int32 row-major with a stride of whole quads.
#pragma once

#include "emv_batch_types.h"
#include "emv_common.cuh"
#include "emv_resident.cuh"

namespace emv {

// Solves instances [beg, end) of class c with this CTA's team until the queue
// is empty; returns false when the team failed.  xs_kt: kt of the subset list
// in shared memory.
__device__ __forceinline__ bool batch_class(const BatchArgs &a, int32_t c, int32_t beg, int32_t end, ResTeam &tm, ResShared &sh,
                            ResInst &I, int32_t &s_idx, int32_t &xs_kt)
{
    for (;;) {
        if (tm.rank == 0 && threadIdx.x == 0) {
            const int32_t idx = beg + (int32_t)atomicAdd(a.ctl + 32 * (1 + c), 1u);
            if (tm.size > 1) __stcg(reinterpret_cast<int32_t *>(tm.bar) + 16, idx);
            else s_idx = idx;
        }
        if (tm.size > 1) {
            // the next index is written only after the team's next barriers
            if (!res_barrier(tm, sh)) return false;
            if (threadIdx.x == 0) s_idx = __ldcg(reinterpret_cast<const int32_t *>(tm.bar) + 16);
        }
        __syncthreads();
        const int32_t idx = s_idx;
        __syncthreads();
        if (idx >= end) return true;
        const BatchInst *B = a.inst + idx;
        const int32_t kt = B->kt, *lvl = a.xs_off + kt * (BATCH_KMAX + 2);
        const int32_t n = B->n, k = B->k;
        int32_t *table = B->table;
        if (threadIdx.x == 0) {
            I.row_ptr = B->row_ptr;
            I.adj = B->adj;
            I.slices = B->slices ? B->slices : a.scratch + (int64_t)(blockIdx.x - tm.rank) * a.scratch_stride;
            I.table = table;
            I.cost = a.costs + B->orig;
            I.unreached = nullptr;
            I.rounds = nullptr;
            I.ns = nullptr;
            I.ld = batch_ld(n);
            I.n = n;
            I.k = k;
            I.kt = kt;
            I.vec = 1;
            I.want_rows = B->rows;
            I.mw = B->mw;
            I.max_rounds = n + 1;
            I.inv_slices = B->inv_slices;
            I.hub_min = B->hub_min;
        }
        tm.limit = B->spin_limit;  // also of the barrier behind the instance
        const int32_t lo = B->lo, hi = B->hi;
        const int32_t base = __ldg(lvl + 1);
        if (threadIdx.x < k) sh.terms[threadIdx.x] = __ldg(B->terms + threadIdx.x);
        if (threadIdx.x < kt + 2) sh.lvl[threadIdx.x] = threadIdx.x == 0 ? 0 : __ldg(lvl + threadIdx.x) - base;
        const ResSmem sm = res_layout(n, kt, a.smem, a.xs + base, xs_kt == kt ? 0 : (1 << kt) - 1);
        xs_kt = kt;
        if (lo == 1)  // row 0 (R:2243-2259)
            for (int32_t v = tm.rank * RES_THREADS + threadIdx.x; v < n; v += tm.size * RES_THREADS) table[v] = INF;
        if (k == 1 && hi == kt && tm.rank == 0 && threadIdx.x == 0) a.costs[B->orig] = INT64_MAX;
        __syncthreads();
        res_solve(I, tm, sm, sh, B->narrow != 0, lo, hi);
        __syncthreads();
        if (*(volatile int *)&sh.ok == 0) return false;
    }
}

__global__ void __launch_bounds__(RES_THREADS, 1) k_batch(BatchArgs a)
{
    __shared__ ResShared sh;
    __shared__ ResInst s_inst;
    __shared__ int32_t s_idx;
    if (threadIdx.x == 0) sh.ok = 1;
    __syncthreads();
    int32_t line = 1 + BATCH_SIZES, beg = 0, xs_kt = -1;
    for (int32_t c = 0; c < BATCH_SIZES; c++) {
        const int32_t size = 1 << (BATCH_SIZES - 1 - c), teams = (int32_t)gridDim.x / size;
        const int32_t team = (int32_t)blockIdx.x / size, end = a.end[c];
        if (end > beg && team < teams) {
            ResTeam tm{a.ctl + 32 * (line + team), a.ctl, (int32_t)blockIdx.x % size, size, 0, RES_SPIN_LIMIT};
            if (!batch_class(a, c, beg, end, tm, sh, s_inst, s_idx, xs_kt)) return;
        }
        line += teams;
        beg = end;
    }
}

// Closes the gaps between the rows of every table whose stride is padded, so that
// it is copied to the host in one piece: a 2D copy into host pages that were
// never written takes six times as long (100 tables of 2^8 x 1002 118 ms, 20 so).
// In place, a CTA an instance: a word moves down only, and a chunk is read
// before it is written.
__global__ void __launch_bounds__(RES_THREADS) k_close_rows(const BatchInst *inst)
{
    const uint32_t n = (uint32_t)inst[blockIdx.x].n, ld = (uint32_t)batch_ld((int32_t)n), words = n << inst[blockIdx.x].kt;
    int32_t *table = inst[blockIdx.x].table;
    constexpr uint32_t PER = 16;
    if (ld == n) return;
    for (uint32_t base = threadIdx.x; base - threadIdx.x < words; base += PER * RES_THREADS) {
        int32_t x[PER];
#pragma unroll
        for (uint32_t j = 0; j < PER; j++) {
            const uint32_t i = base + j * RES_THREADS;
            if (i < words) x[j] = __ldcg(table + i / n * ld + i % n);
        }
        __syncthreads();
#pragma unroll
        for (uint32_t j = 0; j < PER; j++)
            if (base + j * RES_THREADS < words) __stcg(table + base + j * RES_THREADS, x[j]);
        __syncthreads();
    }
}

}  // namespace emv
