// emv_resident.cu -- host side of the one-launch solver (emv_resident.cuh).
#include "emv_resident.cuh"

#include <algorithm>
#include <cstring>

#include "emv_resident.h"

using namespace emv;

namespace emv {

// The whole solve: CSR check, arc slices, levels 1..kt.
__global__ void __launch_bounds__(RES_THREADS, 1) k_resident(ResArgs a)
{
    __shared__ ResShared sh;
    ResTeam tm{a.out->bar, &a.out->err, (int32_t)blockIdx.x, (int32_t)gridDim.x, 0, a.spin_limit};
    const int64_t first = (int64_t)blockIdx.x * RES_THREADS + threadIdx.x, stride = (int64_t)gridDim.x * RES_THREADS;
    const ResSmem sm = res_layout(a.inst.n, a.inst.kt, a.smem, a.xs, a.lvl[a.inst.kt + 1]);
    if (threadIdx.x == 0) sh.ok = 1;  // before the barrier that first reads it
    if (threadIdx.x < EMV_MAX_K) sh.terms[threadIdx.x] = a.terms[threadIdx.x];
    if (threadIdx.x < RES_KMAX + 2) sh.lvl[threadIdx.x] = a.lvl[threadIdx.x];
    if (blockIdx.x == 0 && threadIdx.x < EMV_MAX_K) a.out->terms[threadIdx.x] = a.terms[threadIdx.x];
    scan_csr(a.inst.row_ptr, a.inst.n, a.col, a.w, a.adj, a.arcs, &a.out->scan);
    if (!res_barrier(tm, sh)) return;
    const uint32_t bad = __ldcg(&a.out->scan.bad), maxw = __ldcg(&a.out->scan.maxw);
    if (a.check) {  // the host reads the same words and names the fault
        const long long bound =
            min((long long)(a.inst.n - 1) * (long long)maxw, (long long)(__ldcg(&a.out->scan.sumw) / 2));
        if (bad || bound >= INF) {
            if (blockIdx.x == 0 && threadIdx.x == 0) a.out->refused = 1;
            return;
        }
    }
    // row 0 (R:2243-2259), which no level reads; after the check: a refused call leaves the caller's table as it is
    for (int64_t v = first; v < a.inst.n; v += stride) a.inst.table[v] = INF;
    res_solve(a.inst, tm, sm, sh, maxw < RES_MAX_W && !(bad & SCAN_BAD_WEIGHT), 1, a.inst.kt);
}

}  // namespace emv

int64_t resident_max_rows(int32_t kt)
{
    int64_t most = 1;
    for (int32_t m = 1, x = 1; m <= kt; m++) {
        x = (int32_t)((int64_t)x * (kt - m + 1) / m);
        most = std::max<int64_t>(most, x);
    }
    return most;
}

bool resident_fits(int32_t n, int32_t kt)
{
    if (kt > RES_KMAX || n > 32 * RES_THREADS) return false;
    const int64_t big = RESIDENT_SMEM - res_fixed_smem(n, kt);
    return res_state_bytes(n, 1) <= big && ((int64_t)16 << kt) + 4 * RES_ACC_WORDS <= big;  // a merge block of 4 vertices
}

int32_t resident_merge_width(int32_t n, int32_t kt, int32_t ctas, int32_t cap)
{
    const int64_t big = RESIDENT_SMEM - res_fixed_smem(n, kt);
    int64_t wmax = std::min<int64_t>((big - 4 * RES_ACC_WORDS) / ((int64_t)16 << kt) * 4, (int64_t)(n + 3) / 4 * 4);
    if (cap > 0) wmax = std::min<int64_t>(wmax, std::max<int64_t>(4, cap / 4 * 4));
    const int64_t waves = (n + ctas * wmax - 1) / (ctas * wmax);
    return (int32_t)std::min<int64_t>(wmax, ((n + ctas * waves - 1) / (ctas * waves) + 3) / 4 * 4);
}

uint32_t res_inv_slices(int32_t n)
{
    const uint64_t slices = ((uint64_t)n + 31) / 32;
    return slices == 1 ? 0u : (uint32_t)((((uint64_t)1 << 32) + slices - 1) / slices);
}

// Arcs of a vertex up to which it has its place in a slice; more make it a hub.
// A slice is as wide as its widest vertex, so 64, but in dense graphs twice the
// mean degree as far as arc counts of pairs fit 8 bits: with every vertex a
// hub, read from adj by a warp, one launch lost to the record kernels and a
// batch to a CTA an instance.  Before and so: 900 cliques of 100, k = 7 5.6 and
// 2.1 ms on the device, 237 of 497, k = 9 58 and 17, n = 4000, degree 70, k = 8 3.80
// and 1.15 ms.  Past a mean degree of 254 few rows take longer so (clique of 400,
// k = 4 0.43 and 0.47 ms, k = 6 0.81 and 0.62).  With one row or two a level the
// slices' latency counts, and a warp a vertex is faster (clique of 200, one source
// 0.10 and 0.14 ms; n = 517, degree 235, k = 3 0.22 and 0.31).
int32_t res_hub_min(int32_t n, int64_t arcs, int32_t kt)
{
    const int64_t mean = arcs / n;
    return kt > 2 && mean > 48 && mean <= (kt > 4 ? 508 : 254) ? (int32_t)std::min<int64_t>(508, 2 * mean) : 64;
}

// A closure takes up to n + 1 rounds of at most about a nanosecond an arc and
// 5 us, a poll at least 0.3 us: the band of the longest closures (n = 25 600, 64
// arcs a vertex, rounds of 0.1 ms as 25 000 vertices have to change one after
// another) takes 2.5 s a row, while RES_SPIN_LIMIT polls are about 1.5 s.
uint32_t res_spin_limit(int32_t n, int64_t arcs, int64_t rows)
{
    const double polls = (double)rows * n * ((double)arcs / 256 + 16);
    return RES_SPIN_LIMIT + (uint32_t)std::min(polls, 2e9);
}

// Whether a solve of n vertices over kt terminals' subsets runs as one
// launch, and its shape.  The closure of a row needs about 7.3 bytes a vertex
// of shared memory (distance, list entry, mark, arc count), so n is at most
// about 31 000.  A row is closed by one CTA, and arcs that do not fit shared
// memory are read again in every round, while the record kernels read an arc
// once for 256 rows and have the whole GPU for a level of few rows; the more
// rows a level has, the more CTAs close some.  Whole calls into a device table,
// one launch and record kernels in ms, k = 3 and k = 9:
//   n = 8000, degree 36     0.49  0.48    1.36  1.62
//   n = 20 000, degree 8    0.43  0.48    1.30  1.68
//   n = 20 000, degree 12   0.49  0.43    1.47  1.65
//   n = 30 000, degree 4    0.51  0.53    1.56  1.75
//   n = 30 000, degree 8    0.60  0.48    1.86  1.83
// and with irregular degrees and weights past the packed arcs (twice the bytes)
//   n = 30 000, degree 8    0.94  0.47    2.91  2.14
// Levels of more rows than SMs (kt >= 10) take turns on them and read the arcs
// again each time: kernel times here and there, degree 8, kt = 10: n = 5800 0.62
// and 1.57 ms, 12 000 1.15 and 1.83, 20 011 1.86 and 2.07; kt = 11, n = 12 000 2.05
// and 2.84; calls with irregular degrees, kt = 10: n = 12 000, degree 16 2.15 and
// 2.01, 16 000, degree 16 2.69 and 2.04; kt = 11: n = 12 000, degree 16 3.51 and 3.08,
// 16 000, degree 10 3.95 and 3.27, degree 5 2.77 and 2.93 (regular; with weights past
// 16 bits 2.92 and 4.35, with weights of 100 to 120 2.17 and 1.96).
// The line does not hold for graphs with hubs, which narrow records leave to a
// warp each: n = 14 414, 288 000 arcs, half of them at a hundred vertices, k = 3 1.5
// and 6.6 ms.
// host_table: the call copies the table to the host.  Past 2^22 cells that copy
// outweighs the solve, and such calls keep the kernels whose value widths
// emv_timing reports.
constexpr int64_t RESIDENT_MAX_ARCS = 300000;
bool resident_plan(const emv_ctx *c, int32_t n, int64_t arcs, int32_t kt, bool host_table, bool crowded, ResidentPlan &p)
{
    const int64_t most = kt <= 9 ? 270000 + 9000 * kt : kt == 10 ? 260000 : 200000;
    if (!resident_fits(n, kt) || arcs > RESIDENT_MAX_ARCS || (!crowded && arcs + 5 * (int64_t)n > most)) return false;
    if (kt > 9 && n > 4096 && (n > 16384 || (host_table && (int64_t)n << kt > 1 << 22))) return false;
    const int sms = c->relax_sm_cap > 0 && c->relax_sm_cap < c->sms ? c->relax_sm_cap : c->sms;
    const int64_t maxcnt = resident_max_rows(kt);
    // a CTA for every 1024 states of the widest level
    p.blocks = (int)std::max<int64_t>(1, std::min<int64_t>(sms, (maxcnt * n + RES_THREADS - 1) / RES_THREADS));
    p.rows = (int32_t)((maxcnt + p.blocks - 1) / p.blocks);
    p.mw = resident_merge_width(n, kt, p.blocks, 0);
    return true;
}

ResidentWords resident_words(const emv_ctx *c)
{
    const ResOut *o = (const ResOut *)c->res_out.ptr;
    return {o->terms, &o->err, &o->refused};
}

int resident_launch(emv_ctx *c, const ResidentPlan &p, int32_t n, int64_t arcs, const int32_t *row_ptr,
                    const int32_t *col, const int32_t *w, const int32_t *terms, int32_t k, int32_t kt, int32_t *table,
                    int64_t ld, bool check, cudaStream_t st)
{
    int r = prepare_subsets(c, kt, st);
    if (!r) r = dev_reserve(c->adj, sizeof(int2) * (size_t)std::max<int64_t>(arcs, 1));
    const int32_t hub_min = res_hub_min(n, arcs, kt);
    if (!r) r = dev_reserve(c->res_arcs, sizeof(int4) * (size_t)(hub_min / 2) * 32 * (((size_t)n + 31) / 32));
    if (!r) r = dev_reserve(c->res_out, sizeof(ResOut));
    if (r) return r;
    if (!c->res_attr) {
        CUDA_TRY(cudaFuncSetAttribute((const void *)k_resident, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      RESIDENT_SMEM));
        c->res_attr = true;
    }
    ResArgs a;
    std::memset(&a, 0, sizeof(a));
    ResInst &I = a.inst;
    a.col = col;
    a.w = w;
    a.adj = (int2 *)c->adj.ptr;
    a.xs = (const uint32_t *)c->kp->xs.ptr;
    a.out = (ResOut *)c->res_out.ptr;
    a.arcs = arcs;
    a.check = check;
    a.smem = RESIDENT_SMEM;
    a.spin_limit = res_spin_limit(n, arcs, p.rows);
    for (int32_t m = 0; m <= kt + 1; m++) a.lvl[m] = (int32_t)c->kp->xs_off[(size_t)m];
    for (int32_t t = 0; t < k; t++) a.terms[t] = terms[t];
    I.row_ptr = row_ptr;
    I.adj = a.adj;
    I.slices = c->res_arcs.ptr;
    I.table = table;
    I.cost = &a.out->cost;
    I.unreached = &a.out->unreached;
    I.rounds = &a.out->rounds;
    I.ns = a.out->ns;
    I.ld = ld;
    I.n = n;
    I.k = k;
    I.kt = kt;
    I.vec = ld % 4 == 0 && ((uintptr_t)table & 15) == 0;
    I.want_rows = p.rows;
    I.mw = p.mw;
    I.max_rounds = max_sweeps(c, n, SWEEP_RATE);
    I.inv_slices = res_inv_slices(n);
    I.hub_min = hub_min;
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
    static_assert(PINNED_RES + sizeof(ResOut) <= PINNED_TB, "result words fit the pinned buffer");
    CUDA_TRY(cudaMemcpyAsync((char *)c->pinned + PINNED_RES, a.out, sizeof(ResOut), cudaMemcpyDeviceToHost, st));
    return EMV_OK;
}

int resident_finish(emv_ctx *c, int32_t n, int32_t k, bool check, bool spanned, int64_t *cost_out, emv_timing *tm)
{
    const ResOut *h = (const ResOut *)((char *)c->pinned + PINNED_RES);
    if (check) {
        const int r = scan_status(h->scan, n);
        if (r) return r;
    }
    if (h->err) return emv_dev_status_to_emv(h->err);
    if (spanned && h->unreached)
        return emv_fail(EMV_ERR_DISCONNECTED, "graph: not connected (a vertex is unreachable from terminal 1)");
    *cost_out = k >= 2 ? h->cost : INT64_MAX;
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
