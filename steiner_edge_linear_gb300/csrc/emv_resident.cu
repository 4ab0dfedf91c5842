// emv_resident.cu -- host side of the one-launch solver (emv_resident.cuh).
#include "emv_resident.cuh"

#include <algorithm>
#include <cstring>

#include "emv_resident.h"

using namespace emv;

// Whether a solve of n vertices over kt terminals' subsets runs as one
// launch, and its shape.  The closure of a row needs about 7.4 bytes a vertex
// of shared memory (distance, list entry, two marks, arc count), so n is at
// most about 30 000.  Levels of more rows than SMs (kt >= 10) take turns on
// them, and the record kernels, which read an arc once for 256 rows, are
// faster from a few thousand vertices on.
bool resident_plan(const emv_ctx *c, int32_t n, int64_t arcs, int32_t kt, ResidentPlan &p)
{
    (void)arcs;
    if (kt > RES_KMAX || (kt > 9 && n > 4096)) return false;
    const int sms = c->relax_sm_cap > 0 && c->relax_sm_cap < c->sms ? c->relax_sm_cap : c->sms;
    int64_t maxcnt = 1;
    for (int32_t m = 1, x = 1; m <= kt; m++) {
        x = (int32_t)((int64_t)x * (kt - m + 1) / m);
        maxcnt = std::max<int64_t>(maxcnt, x);
    }
    // a CTA for every 1024 states of the widest level
    p.blocks = (int)std::max<int64_t>(1, std::min<int64_t>(sms, (maxcnt * n + RES_THREADS - 1) / RES_THREADS));
    p.rows = (int32_t)((maxcnt + p.blocks - 1) / p.blocks);
    const int64_t big = RESIDENT_SMEM - res_fixed_smem(n, kt);
    const int64_t merge_min = ((int64_t)16 << kt) + 4 * RES_ACC_WORDS;  // blocks of 4 vertices
    if (n > 32 * RES_THREADS || res_state_bytes(n, 1) > big || merge_min > big) return false;
    // merge blocks: as few waves of blocks as the shared memory allows, and
    // within them the narrowest blocks, so that every CTA has some
    const int64_t wmax = std::min<int64_t>((big - 4 * RES_ACC_WORDS) / ((int64_t)16 << kt) * 4, (int64_t)(n + 3) / 4 * 4);
    const int64_t waves = (n + p.blocks * wmax - 1) / (p.blocks * wmax);
    p.mw = (int32_t)std::min<int64_t>(wmax, ((n + p.blocks * waves - 1) / (p.blocks * waves) + 3) / 4 * 4);
    return true;
}

const int32_t *resident_terms(const emv_ctx *c) { return ((const ResOut *)c->res_out.ptr)->terms; }

int run_resident(emv_ctx *c, const ResidentPlan &p, int32_t n, int64_t arcs, const int32_t *row_ptr, const int32_t *col,
                 const int32_t *w, const int32_t *terms, int32_t k, int32_t kt, int32_t *table, int64_t ld, bool check,
                 cudaStream_t st, int64_t *cost_out, emv_timing *tm)
{
    int r = prepare_subsets(c, kt, st);
    if (!r) r = dev_reserve(c->adj, sizeof(int2) * (size_t)std::max<int64_t>(arcs, 1));
    if (!r) r = dev_reserve(c->res_arcs, sizeof(int4) * (RES_HUB / 2) * 32 * (((size_t)n + 31) / 32));
    if (!r) r = dev_reserve(c->res_out, sizeof(ResOut));
    if (r) return r;
    if (!c->res_attr) {
        CUDA_TRY(cudaFuncSetAttribute((const void *)k_resident, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      RESIDENT_SMEM));
        c->res_attr = true;
    }
    ResArgs a;
    std::memset(&a, 0, sizeof(a));
    a.row_ptr = row_ptr;
    a.col = col;
    a.w = w;
    a.adj = (int2 *)c->adj.ptr;
    a.slices = c->res_arcs.ptr;
    a.table = table;
    a.xs = (const uint32_t *)c->kp->xs.ptr;
    a.out = (ResOut *)c->res_out.ptr;
    a.ld = ld;
    a.arcs = arcs;
    a.n = n;
    a.k = k;
    a.kt = kt;
    a.check = check;
    a.vec = ld % 4 == 0 && ((uintptr_t)table & 15) == 0;
    a.want_rows = p.rows;
    a.mw = p.mw;
    a.smem = RESIDENT_SMEM;
    a.max_rounds = (c->sweep_limit > 0 && c->sweep_limit < (int64_t)n + 1) ? (int32_t)c->sweep_limit : n + 1;
    const uint64_t slices = ((uint64_t)n + 31) / 32;
    a.inv_slices = slices == 1 ? 0u : (uint32_t)((((uint64_t)1 << 32) + slices - 1) / slices);
    for (int32_t m = 0; m <= kt + 1; m++) a.xs_off[m] = (int32_t)c->kp->xs_off[(size_t)m];
    for (int32_t t = 0; t < k; t++) a.terms[t] = terms[t];
    CUDA_TRY(cudaMemsetAsync(a.out, 0, sizeof(ResOut), st));
    CUDA_TRY(cudaEventRecord(c->ev[0], st));
    void *args[] = {&a};
    if (p.blocks > 1)
        CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_resident, dim3(p.blocks), dim3(RES_THREADS), args, (size_t)RESIDENT_SMEM,
                                             st));
    else
        CUDA_TRY(cudaLaunchKernel((const void *)k_resident, dim3(1), dim3(RES_THREADS), args, (size_t)RESIDENT_SMEM, st));
    c->launches++;
    CUDA_TRY(cudaEventRecord(c->ev[1], st));
    ResOut *h = (ResOut *)((char *)c->pinned + 2048);
    static_assert(sizeof(ResOut) <= 2048, "result words fit the pinned buffer");
    CUDA_TRY(cudaMemcpyAsync(h, a.out, sizeof(ResOut), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    if (check) {
        r = scan_status(h->scan, n);
        if (r) return r;
    }
    if (h->err) return emv_dev_status_to_emv(h->err);
    if (check && h->unreached)
        return emv_fail(EMV_ERR_DISCONNECTED, "graph: not connected (a vertex is unreachable from terminal 1)");
    *cost_out = (k >= 2 && h->cost < INF) ? (int64_t)h->cost : INT64_MAX;
    if (tm) {
        float ms = 0;
        cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]);
        tm->kernel_ms = ms;
        tm->level1_ms = (float)(h->ns[0] * 1e-6);
        tm->merge_ms = (float)(h->ns[1] * 1e-6);
        tm->relax_ms = (float)(h->ns[2] * 1e-6);
        tm->relax_sweeps = h->rounds;
        tm->relax_launches = 1;
    }
    return EMV_OK;
}
