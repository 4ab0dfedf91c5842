// emv_device.cu -- solver context and the single-instance GPU DP (C ABI).
//
// Reference counterparts (reader/reader-el.c):
//   emv_kernel              R:1966-2139  -> emv_kernel_dev
//   erickson_monma_veinott  R:2141-2343  -> emv_solve / emv_solve_dev
//   dijkstra (-dijkstra)    R:1762-1880, R:2454-2484 -> emv_sssp
#include "emv_kernels.cuh"
#include "emv_resident.h"
#include "emv_solver.h"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <new>
#include <numeric>
#include <vector>

using namespace emv;

int emv_dev_status_to_emv(uint32_t s)
{
    if (s == 0) return EMV_OK;
    if (s & (EMV_DEV_BARRIER_TIMEOUT | EMV_DEV_SWEEP_LIMIT | EMV_DEV_TB_STEPS | EMV_DEV_QUEUE_TIMEOUT))
        return emv_fail(EMV_ERR_TIMEOUT, "device loop bound reached (status 0x%x)", s);
    if (s & EMV_DEV_BAD_VALUE) return emv_fail(EMV_ERR_BAD_INPUT, "an input value is above 2^30 (status 0x%x)", s);
    if (s & EMV_DEV_OVERFLOW)
        return emv_fail(EMV_ERR_OVERFLOW, "a finite value plus an arc weight reached 2^30 (status 0x%x)", s);
    return emv_fail(EMV_ERR_INTERNAL, "device status 0x%x", s);
}

extern "C" const char *emv_version(void) { return "emv-gb300 1.0 sm_103a"; }

// ------------------------------------------------------------ buffers

int dev_reserve(DevBuf &b, size_t bytes)
{
    if (b.bytes >= bytes) return EMV_OK;
    if (b.ptr) cudaFree(b.ptr);
    b.ptr = nullptr;
    b.bytes = 0;
    size_t want = std::max<size_t>(bytes, 256);
    cudaError_t e = cudaMalloc(&b.ptr, want);
    if (e != cudaSuccess) {
        cudaGetLastError();
        b.ptr = nullptr;
        return emv_fail(e == cudaErrorMemoryAllocation ? EMV_ERR_OOM : EMV_ERR_CUDA,
                        "cudaMalloc(%zu): %s", want, cudaGetErrorString(e));
    }
    b.bytes = want;
    return EMV_OK;
}

void dev_release(DevBuf &b)
{
    if (b.ptr) cudaFree(b.ptr);
    b.ptr = nullptr;
    b.bytes = 0;
}

// ------------------------------------------------------------ context

// Relaxation kernels by record width: k_relax<1, 2, 4, 5, 8> with 32-bit,
// then with 16-bit records (32 * VEC words a vertex).
static const void *const relax_fns[RELAX_VARIANTS] = {
    (const void *)k_relax<1>,       (const void *)k_relax<2>,       (const void *)k_relax<4>,
    (const void *)k_relax<5>,       (const void *)k_relax<8>,       (const void *)k_relax<1, true>,
    (const void *)k_relax<2, true>, (const void *)k_relax<4, true>, (const void *)k_relax<5, true>,
    (const void *)k_relax<8, true>,
    // for graphs with hubs
    (const void *)k_relax<1, false, true>, (const void *)k_relax<2, false, true>, (const void *)k_relax<4, false, true>,
    (const void *)k_relax<5, false, true>, (const void *)k_relax<8, false, true>, (const void *)k_relax<1, true, true>,
    (const void *)k_relax<2, true, true>,  (const void *)k_relax<4, true, true>,  (const void *)k_relax<5, true, true>,
    (const void *)k_relax<8, true, true>};

// Narrow-record kernels by width (4, 8, 16 or 32 rows).
static const void *const narrow_fns[NARROW_VARIANTS] = {(const void *)k_narrow<1>, (const void *)k_narrow<2>,
                                                        (const void *)k_narrow<4>, (const void *)k_narrow<8>};

extern "C" int emv_create(emv_ctx **out, int32_t device)
{
    if (!out) return emv_fail(EMV_ERR_BAD_INPUT, "null ctx pointer");
    *out = nullptr;
    int ndev = 0;
    CUDA_TRY(cudaGetDeviceCount(&ndev));
    if (device < 0 || device >= ndev) return emv_fail(EMV_ERR_BAD_INPUT, "device %d of %d", device, ndev);
    CUDA_TRY(cudaSetDevice(device));
    cudaDeviceProp prop;
    CUDA_TRY(cudaGetDeviceProperties(&prop, device));
    if (!prop.cooperativeLaunch) return emv_fail(EMV_ERR_CUDA, "device lacks cooperative launch");
    emv_ctx *c = new (std::nothrow) emv_ctx();
    if (!c) return emv_fail(EMV_ERR_OOM, "ctx");
    c->device = device;
    c->sms = prop.multiProcessorCount;
    c->l2_bytes = prop.l2CacheSize;
    for (int i = 0; i < RELAX_VARIANTS; i++) {
        int per_sm = 0;
        CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, relax_fns[i], RELAX_THREADS, 0));
        c->relax_blocks_max[i] = std::max(1, per_sm) * c->sms;
    }
    for (int i = 0; i < NARROW_VARIANTS; i++) {
        int per_sm = 0;
        CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, narrow_fns[i], NARROW_THREADS, 0));
        c->narrow_blocks_max[i] = std::max(1, per_sm) * c->sms;
    }
    int st = dev_reserve(c->ctrl, sizeof(uint32_t) * C_WORDS);
    if (!st) st = dev_reserve(c->stat, sizeof(DevStat));
    if (!st) st = dev_reserve(c->lvlmax, sizeof(uint32_t) * (EMV_MAX_K + 1));
    if (!st) st = dev_reserve(c->gscan, sizeof(GraphScan));
    if (!st) {
        if (cudaMallocHost(&c->pinned, PINNED_BYTES) != cudaSuccess) { cudaGetLastError(); st = emv_fail(EMV_ERR_OOM, "pinned"); }
    }
    for (int i = 0; !st && i < MAX_EVENTS; i++)
        if (cudaEventCreate(&c->ev[i]) != cudaSuccess) st = emv_fail(EMV_ERR_CUDA, "event create");
    for (int i = 0; !st && i <= EMV_MAX_K; i++)
        if (cudaEventCreateWithFlags(&c->evmax[i], cudaEventDisableTiming) != cudaSuccess)
            st = emv_fail(EMV_ERR_CUDA, "event create");
    if (st) {
        emv_destroy(c);
        return st;
    }
    *out = c;
    return EMV_OK;
}

extern "C" int emv_set_sweep_limit(emv_ctx *c, int64_t limit)
{
    if (!c || limit < 0) return emv_fail(EMV_ERR_BAD_INPUT, "emv_set_sweep_limit: bad arguments");
    c->sweep_limit = limit;
    return EMV_OK;
}

extern "C" int emv_set_value_bits(emv_ctx *c, int32_t bits)
{
    if (!c || (bits != 0 && bits != 32)) return emv_fail(EMV_ERR_BAD_INPUT, "emv_set_value_bits: bits 0 or 32");
    c->value_bits = bits;
    return EMV_OK;
}

extern "C" int emv_destroy(emv_ctx *c)
{
    if (!c) return EMV_OK;
    cudaSetDevice(c->device);
    cudaDeviceSynchronize();
    for (DevBuf *b : {&c->ctrl, &c->stat, &c->lvlmax, &c->gscan, &c->shadow, &c->scratch, &c->act, &c->adj, &c->mark, &c->hubs, &c->terms, &c->g_all,
                      &c->table, &c->tb_edges, &c->tb_out, &c->tb_work, &c->res_arcs, &c->res_out,
                      &c->bxs, &c->bxs_off, &c->b_costs})
        dev_release(*b);
    for (KPlan *p : c->kplans) {
        if (!p) continue;
        for (DevBuf *b : {&p->xs, &p->mpairs, &p->movr, &p->mstream_data, &p->mstream_phases, &p->mblock_data,
                          &p->mblock_phases})
            dev_release(*b);
        delete p;
    }
    for (int i = 0; i < MAX_EVENTS; i++)
        if (c->ev[i]) cudaEventDestroy(c->ev[i]);
    for (int i = 0; i <= EMV_MAX_K; i++)
        if (c->evmax[i]) cudaEventDestroy(c->evmax[i]);
    for (BatchLane &L : c->blane) {
        for (DevBuf *b : {&L.row, &L.adj, &L.term, &L.desc, &L.table, &L.ctrl, &L.arcs}) dev_release(*b);
        for (BatchGraphExec &G : L.graph) batch_graph_release(G);
        if (L.stage) cudaFreeHost(L.stage);
    }
    for (cudaEvent_t e : c->bev)
        if (e) cudaEventDestroy(e);
    if (c->bstream) cudaStreamDestroy(c->bstream);
    if (c->g_stage) cudaFreeHost(c->g_stage);
    if (c->h_dist) cudaFreeHost(c->h_dist);
    if (c->pinned) cudaFreeHost(c->pinned);
    delete c;
    return EMV_OK;
}

// ------------------------------------------------------------ the DP

static int grid_for(int64_t work, int threads, int cap)
{
    int64_t g = (work + threads - 1) / threads;
    return (int)std::max<int64_t>(1, std::min<int64_t>(g, cap));
}

// Vertices of more arcs than this are relaxed by a whole block: two windows of
// a warp, and well above the mean degree (with near-equal degrees every warp
// has its share of long vertices anyway).  n = 30 000, k = 10, power-law degrees:
// 3.56 ms of relaxation from 128 arcs on, 3.16 from 64, 3.15 from 32 (but 2.82
// against 2.50 at n = 10^5).
static int32_t relax_hub_min(int32_t n, int64_t arcs) { return (int32_t)std::max<int64_t>(64, 4 * arcs / n); }

// Chunks of at most this many rows are closed on narrow records, several
// vertices a warp, instead of 128-byte records, a vertex a warp: n = 2^17,
// degree 8, k = 7 (chunks of 21, 7 and 1 rows) 1.99 -> 1.57 ms of relaxation,
// n = 10^5, degree 20, k = 12 (12 and 1) 9.93 -> 9.80.  With hubs only a single
// row, whose sweeps are nearly all barrier: narrow records leave a hub to one
// warp (n = 30 000, power-law degrees, k = 10, a chunk of 10 rows: 2.36 -> 2.52).
constexpr int32_t RELAX_NARROW = 32;

// Bound on the sweeps of a closure: n + 1, or the caller's limit, which counts
// sweeps of k_relax.  There a change travels two arcs a sweep in the frontier's
// tail; narrow records and the one-launch solver move it by one and need up to
// 2.1 times as many (grids of n = 10^4: 196 rounds for 93 sweeps, of n = 10^5: 660
// for 314; random graphs 1.5 times), each of a third of the time or less.  They
// are allowed SWEEP_RATE for one.
int32_t max_sweeps(const emv_ctx *c, int32_t n, int32_t rate)
{
    const int64_t bound = (int64_t)n + 1;
    return (int32_t)(c->sweep_limit > 0 && c->sweep_limit < bound ? std::min(bound, c->sweep_limit * rate) : bound);
}

// Launches the relaxation of one chunk of at most CHUNK_ROWS rows (2 *
// CHUNK_ROWS with 16-bit records, which the caller takes only for rows whose
// values are all at most 32767) as one cooperative, persistent kernel; the
// record width follows the row count.
int launch_relax(emv_ctx *c, const int32_t *row_ptr, const int2 *adj, int32_t n, int64_t ld, int32_t *table,
                 const uint32_t *rows, int32_t nrows, cudaStream_t st, bool u16 = false, uint16_t *shadow = nullptr,
                 int64_t shadow_ld = 0)
{
    RelaxArgs a;
    a.mark = (int2 *)c->mark.ptr;
    a.high = (int32_t *)(a.mark + n);
    a.row_ptr = row_ptr;
    a.adj = adj;
    a.n = n;
    a.ld = ld;
    a.table = table;
    a.rows = rows;
    a.nrows = nrows;
    a.scratch = (int32_t *)c->scratch.ptr;
    a.act0 = (uint8_t *)c->act.ptr;
    a.act1 = (uint8_t *)c->act.ptr + ((size_t)n + 255) / 256 * 256;
    a.ctrl = (uint32_t *)c->ctrl.ptr;
    a.stat = (DevStat *)c->stat.ptr;
    a.max_sweeps = max_sweeps(c, n, 1);
    // Dense sweeps pay off while almost every vertex has a changed neighbour:
    // with mean degree d and a fraction f of vertices changed, a vertex has none
    // with probability (1 - f)^d; take every vertex while that is below 10 %.
    const double deg = (double)c->relax_arcs / (double)n;
    a.dense_min = deg > 0 ? (int32_t)std::min<double>((double)n, (double)n * (1.0 - std::pow(0.1, 1.0 / deg))) : n;
    a.shadow = shadow;
    a.shadow_ld = shadow_ld;
    const int32_t words = u16 ? (nrows + 1) / 2 : nrows;  // int32 words a vertex record needs
    const int wi = words <= 32 ? 0 : words <= 64 ? 1 : words <= 128 ? 2 : words <= 160 ? 3 : 4;
    const int vi = wi + (u16 ? 5 : 0) + (c->relax_nhubs > 0 ? 10 : 0);
    a.hubs = (const int32_t *)c->hubs.ptr;
    a.nhubs = c->relax_nhubs;
    a.hub_min = relax_hub_min(n, c->relax_arcs);
    const void *fn = relax_fns[vi];
    // A warp per 8 vertices is enough; small graphs use fewer blocks (cheaper barriers).
    const int vpb = 8 * (RELAX_THREADS / 32);
    int bmax = c->relax_blocks_max[vi];
    if (c->relax_sm_cap > 0 && c->relax_sm_cap < c->sms) bmax = std::max(1, bmax / c->sms * c->relax_sm_cap);
    const int blocks = std::min(bmax, std::max(1, (n + vpb - 1) / vpb));
    CUDA_TRY(cudaMemsetAsync(a.ctrl, 0, sizeof(uint32_t) * C_WORDS, st));
    void *args[] = {&a};
    CUDA_TRY(cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(RELAX_THREADS), args, 0, st));
    c->launches += 1;  // the kernel (the control-word memset is not a kernel)
    return EMV_OK;
}

// Launches the closures of at most 32 rows as one cooperative kernel: the
// single-source distances of terms[r] in rows[r] (device arrays), or, with
// terms null, the closures of the rows as they are; vmax (or null) receives the
// largest value written.
int launch_narrow(emv_ctx *c, const int32_t *row_ptr, const int2 *adj, int32_t n, int64_t ld, int32_t *table,
                  const uint32_t *rows, int32_t nrows, const int32_t *terms, cudaStream_t st, uint32_t *vmax = nullptr,
                  uint16_t *shadow = nullptr, int64_t shadow_ld = 0, const GraphScan *scan = nullptr)
{
    const int vi = nrows <= 4 ? 0 : nrows <= 8 ? 1 : nrows <= 16 ? 2 : 3;
    NarrowLaunch a;
    a.na.row_ptr = row_ptr;
    a.na.n = n;
    a.na.rec = (int4 *)c->scratch.ptr;
    a.na.act0 = (uint8_t *)c->act.ptr;
    a.na.act1 = (uint8_t *)c->act.ptr + ((size_t)n + 255) / 256 * 256;
    a.na.ctrl = (uint32_t *)c->ctrl.ptr;
    a.na.max_sweeps = max_sweeps(c, n, SWEEP_RATE);
    a.na.dense_min = narrow_dense_min(n, c->relax_arcs);
    a.adj = adj;
    a.terms = terms;
    a.rows = rows;
    a.nrows = nrows;
    a.table = table;
    a.ld = ld;
    a.vmax = vmax;
    a.shadow = shadow;
    a.shadow_ld = shadow_ld;
    a.stat = (DevStat *)c->stat.ptr;
    a.scan = scan;
    const int vpb = narrow_vertices(1 << vi) * (NARROW_THREADS / 32);  // one group of vertices a warp
    int bmax = c->narrow_blocks_max[vi];
    if (c->relax_sm_cap > 0 && c->relax_sm_cap < c->sms) bmax = std::max(1, bmax / c->sms * c->relax_sm_cap);
    const int blocks = std::min(bmax, std::max(1, (n + vpb - 1) / vpb));
    CUDA_TRY(cudaMemsetAsync(a.na.ctrl, 0, sizeof(uint32_t) * C_WORDS, st));
    void *args[] = {&a};
    CUDA_TRY(cudaLaunchCooperativeKernel(narrow_fns[vi], dim3(blocks), dim3(NARROW_THREADS), args, 0, st));
    c->launches += 1;
    return EMV_OK;
}

int32_t relax_chunk_rows_level(const emv_ctx *c, int32_t n, bool u16, int64_t cnt)
{
    return relax_rows_per_level_chunk(n, c->l2_bytes, u16, cnt);
}

int reserve_relax(emv_ctx *c, int32_t n)
{
    const size_t npad = ((size_t)n + 31) / 32 * 32;
    int st = dev_reserve(c->scratch, npad * CHUNK_ROWS * sizeof(int32_t));
    if (!st) st = dev_reserve(c->act, 2 * (((size_t)n + 255) / 256 * 256));
    if (!st) st = dev_reserve(c->mark, (sizeof(int2) + sizeof(int32_t)) * (size_t)n);
    return st;
}

constexpr int32_t MERGE_SMEM_BYTES = 220 * 1024;
constexpr int32_t MERGE_SMEM_KMAX = 15;  // staged slots must fit 16 bits

constexpr int32_t STREAM_SMEM_BYTES = 224 * 1024;

// Plans the streamed merge of the levels of k that have no block merge, on the
// host (emv_plan.cpp), and uploads the plan data and the per-launch phase
// descriptors.  (Of all levels: 24 of the 30 ms of a context's first solve, n =
// 2000, k = 12.)
int plan_stream_merge(emv_ctx *c, int32_t k, cudaStream_t st)
{
    const std::vector<uint32_t> &xs = c->kp->xs_host;
    const std::vector<int64_t> &off = c->kp->xs_off;
    c->kp->mstream_groups.assign((size_t)k + 2, {});
    if (k > MERGE_SMEM_KMAX) return EMV_OK;
    std::vector<uint32_t> data;
    std::vector<std::vector<HostGroup>> plan;
    std::vector<bool> block;
    for (const BlockLevel &L : c->kp->mblock_levels) block.push_back(L.nphase > 0);
    plan_stream_levels(k, xs, off, STREAM_SMEM_BYTES, data, plan, block);
    if (data.empty()) return EMV_OK;
    int r = dev_reserve(c->kp->mstream_data, sizeof(uint32_t) * data.size());
    if (r) return r;
    std::vector<MergePhase> phases;
    const uint32_t *base = (const uint32_t *)c->kp->mstream_data.ptr;
    for (int32_t m = 2; m <= k; m++)
        for (const HostGroup &G : plan[(size_t)m]) {
            StreamGroup sg;
            sg.x0 = G.x0;
            sg.cnt = G.cnt;
            sg.smem = G.smem;
            sg.phase_off = (int64_t)phases.size();
            sg.nphase = (int64_t)G.phases.size();
            if (sg.smem > STREAM_SMEM_BYTES) return emv_fail(EMV_ERR_INTERNAL, "merge plan: %lld bytes of shared memory",
                                                             (long long)sg.smem);
            for (const HostPhase &hp : G.phases) {
                if (hp.pairs_at % 4 != 0) return emv_fail(EMV_ERR_INTERNAL, "merge plan: pair block not 16-byte aligned");
                MergePhase mp;
                mp.rows = base + hp.rows_at;
                mp.qoff = base + hp.qoff_at;
                mp.pairs = base + hp.pairs_at;
                mp.nrows = hp.nrows;
                mp.pad_ = 0;
                phases.push_back(mp);
            }
            c->kp->mstream_groups[(size_t)m].push_back(sg);
        }
    r = dev_reserve(c->kp->mstream_phases, sizeof(MergePhase) * std::max<size_t>(1, phases.size()));
    if (r) return r;
    CUDA_TRY(cudaMemcpyAsync(c->kp->mstream_data.ptr, data.data(), sizeof(uint32_t) * data.size(), cudaMemcpyHostToDevice,
                             st));
    if (!phases.empty())
        CUDA_TRY(cudaMemcpyAsync(c->kp->mstream_phases.ptr, phases.data(), sizeof(MergePhase) * phases.size(),
                                 cudaMemcpyHostToDevice, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    return EMV_OK;
}

// Plans the block merge of every level of k and uploads it.
// From BLOCK_KMIN on, where a level has pairs enough (n = 4 * 10^5, k = 6: 1.34 ->
// 0.68 ms of merges); every level up to BLOCK_KMAX fits.
constexpr int32_t BLOCK_KMIN = 6, BLOCK_KMAX = 12;
static int plan_block_merge(emv_ctx *c, int32_t k, cudaStream_t st)
{
    c->kp->mblock_levels.assign((size_t)k + 2, {});
    if (k < BLOCK_KMIN || k > BLOCK_KMAX) return EMV_OK;
    std::vector<uint32_t> data;
    std::vector<HostBlockLevel> plan;
    plan_block_levels(k, BLOCK_LOW, c->kp->xs_host, c->kp->xs_off, STREAM_SMEM_BYTES, data, plan);
    int r = dev_reserve(c->kp->mblock_data, sizeof(uint32_t) * std::max<size_t>(1, data.size()));
    if (r) return r;
    const uint32_t *base = (const uint32_t *)c->kp->mblock_data.ptr;
    std::vector<BlockPhase> phases;
    for (int32_t m = 3; m <= k; m++) {
        const HostBlockLevel &L = plan[(size_t)m];
        BlockLevel &to = c->kp->mblock_levels[(size_t)m];
        to.phase_off = (int64_t)phases.size();
        to.nphase = (int64_t)L.phases.size();
        to.rows = L.rows;
        to.split = L.split;
        for (const HostBlockPhase &P : L.phases)
            phases.push_back({base + P.warps_at, base + P.units_at, base + P.words_at, (int32_t)P.y0, (int32_t)P.ny,
                              (int32_t)P.z0, (int32_t)P.nz});
    }
    r = dev_reserve(c->kp->mblock_phases, sizeof(BlockPhase) * std::max<size_t>(1, phases.size()));
    if (r) return r;
    CUDA_TRY(cudaMemcpyAsync(c->kp->mblock_data.ptr, data.data(), sizeof(uint32_t) * data.size(), cudaMemcpyHostToDevice,
                             st));
    CUDA_TRY(cudaMemcpyAsync(c->kp->mblock_phases.ptr, phases.data(), sizeof(BlockPhase) * phases.size(),
                             cudaMemcpyHostToDevice, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    return EMV_OK;
}

static int build_plan(emv_ctx *c, int32_t k, cudaStream_t st);

int prepare_subsets(emv_ctx *c, int32_t k, cudaStream_t st)
{
    if (c->xs_k == k) return EMV_OK;
    if (k < 1 || k > EMV_MAX_K) return emv_fail(EMV_ERR_BAD_INPUT, "k = %d", k);
    if (c->kplans[k]) {  // built before on this context
        c->kp = c->kplans[k];
        c->xs_k = k;
        return EMV_OK;
    }
    KPlan *plan = new (std::nothrow) KPlan();
    if (!plan) return emv_fail(EMV_ERR_OOM, "plan");
    c->kp = plan;
    c->xs_k = -1;
    const int r0 = build_plan(c, k, st);
    if (r0) {
        for (DevBuf *b : {&plan->xs, &plan->mpairs, &plan->movr, &plan->mstream_data, &plan->mstream_phases,
                          &plan->mblock_data, &plan->mblock_phases})
            dev_release(*b);
        delete plan;
        c->kp = nullptr;
        return r0;
    }
    c->kplans[k] = plan;
    c->xs_k = k;
    return EMV_OK;
}

// Builds c->kp for k: subsets, slot lists and the streamed merge plan.
static int build_plan(emv_ctx *c, int32_t k, cudaStream_t st)
{
    subset_levels(k, c->kp->xs_host, c->kp->xs_off);
    int r = dev_reserve(c->kp->xs, sizeof(uint32_t) * std::max<size_t>(1, c->kp->xs_host.size()));
    if (r) return r;
    CUDA_TRY(cudaMemcpyAsync(c->kp->xs.ptr, c->kp->xs_host.data(), sizeof(uint32_t) * c->kp->xs_host.size(),
                             cudaMemcpyHostToDevice, st));
    r = plan_block_merge(c, k, st);
    if (!r) r = plan_stream_merge(c, k, st);
    if (r) return r;
    // Pair and override slot lists of the staged-all-rows merge, for the levels
    // the others have no plan for (level order).
    c->kp->mpair_base.assign((size_t)k + 2, 0);
    c->kp->movr_base.assign((size_t)k + 2, 0);
    std::vector<uint32_t> pairs, ovr;
    if (k <= MERGE_SMEM_KMAX) {
        std::vector<uint32_t> lidx((size_t)1 << k, 0);
        for (size_t i = 0; i < c->kp->xs_host.size(); i++) lidx[c->kp->xs_host[i]] = (uint32_t)i;
        for (int32_t m = 2; m <= k; m++) {
            c->kp->mpair_base[(size_t)m] = (int64_t)pairs.size();
            c->kp->movr_base[(size_t)m] = (int64_t)ovr.size();
            if (c->kp->mblock_levels[(size_t)m].nphase > 0 || !c->kp->mstream_groups[(size_t)m].empty()) continue;
            for (int64_t i = c->kp->xs_off[(size_t)m]; i < c->kp->xs_off[(size_t)m + 1]; i++) {
                const uint32_t X = c->kp->xs_host[(size_t)i];
                const uint32_t low = X & (0u - X), rest = X ^ low;
                uint32_t sm = 0;
                do {
                    const uint32_t Y = low | sm;
                    pairs.push_back(lidx[Y] | (lidx[X ^ Y] << 16));
                    sm = (sm - rest) & rest;
                } while (sm != rest);
                for (int32_t t = 0; t < k; t++)
                    if (X >> t & 1u) ovr.push_back(((uint32_t)t << 16) | lidx[X ^ (1u << t)]);
            }
        }
    }
    if (!pairs.empty()) {
        r = dev_reserve(c->kp->mpairs, sizeof(uint32_t) * pairs.size());
        if (!r) r = dev_reserve(c->kp->movr, sizeof(uint32_t) * ovr.size());
        if (r) return r;
        CUDA_TRY(cudaMemcpyAsync(c->kp->mpairs.ptr, pairs.data(), sizeof(uint32_t) * pairs.size(), cudaMemcpyHostToDevice,
                                 st));
        CUDA_TRY(cudaMemcpyAsync(c->kp->movr.ptr, ovr.data(), sizeof(uint32_t) * ovr.size(), cudaMemcpyHostToDevice, st));
    }
    CUDA_TRY(cudaStreamSynchronize(st));
    return EMV_OK;
}

template <int VB>
static cudaError_t merge_smem_launch(emv_ctx *c, int32_t *table, int64_t ld, int32_t n, int32_t k, int32_t m,
                                     const int32_t *d_terms, cudaStream_t st)
{
    const int64_t b = c->kp->xs_off[(size_t)m], cnt = c->kp->xs_off[(size_t)m + 1] - b;
    const int32_t nstage = (int32_t)c->kp->xs_off[(size_t)m];
    const uint32_t *xs = (const uint32_t *)c->kp->xs.ptr;
    const size_t smem = sizeof(int32_t) * (size_t)nstage * VB;
    const int32_t npairs = (1 << (m - 1)) - 1;
    k_merge_smem<VB><<<(unsigned)((n + VB - 1) / VB), 1024, smem, st>>>(
        table, ld, n, xs + b, (int32_t)cnt, xs, nstage, (const uint32_t *)c->kp->mpairs.ptr + c->kp->mpair_base[(size_t)m],
        npairs, (const uint32_t *)c->kp->movr.ptr + c->kp->movr_base[(size_t)m], m, d_terms);
    (void)k;
    return cudaGetLastError();
}

// Merge of level m: the shared-memory kernel with the widest vertex block
// whose staging fits, else the direct kernel (k above MERGE_SMEM_KMAX).
int launch_merge(emv_ctx *c, int32_t *table, int64_t ld, int32_t n, int32_t k, int32_t m, const int32_t *d_terms,
                 cudaStream_t st, bool u16 = false, const uint16_t *shadow = nullptr, int64_t shadow_ld = 0)
{
    if (!c->merge_attr) {
        const void *fns[6] = {(const void *)k_merge_smem<32>, (const void *)k_merge_smem<16>,
                              (const void *)k_merge_smem<8>, (const void *)k_merge_smem<4>,
                              (const void *)k_merge_smem<2>, (const void *)k_merge_smem<1>};
        for (const void *f : fns)
            CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, MERGE_SMEM_BYTES));
        CUDA_TRY(cudaFuncSetAttribute((const void *)k_merge_stream, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      STREAM_SMEM_BYTES));
        CUDA_TRY(cudaFuncSetAttribute((const void *)k_merge_stream16, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      STREAM_SMEM_BYTES));
        for (const void *f : {(const void *)k_merge_block<false>, (const void *)k_merge_block<true>})
            CUDA_TRY(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, STREAM_SMEM_BYTES));
        c->merge_attr = true;
    }
    const int64_t nstage = c->kp->xs_off[(size_t)m];
    cudaError_t e = cudaSuccess;
    c->merge16_last = false;
    c->launches++;
    const BlockLevel &L = c->kp->mblock_levels[(size_t)m];
    if (L.nphase > 0 || !c->kp->mstream_groups[(size_t)m].empty()) {
        // these merges record the level's largest value (other kernels leave it unknown)
        CUDA_TRY(cudaMemsetAsync((uint32_t *)c->lvlmax.ptr + m, 0, sizeof(uint32_t), st));
        const int64_t b = c->kp->xs_off[(size_t)m];
        if (L.nphase == 0) c->launches += (int64_t)c->kp->mstream_groups[(size_t)m].size() - 1;
        // 16-bit staging reads int2 pairs of vertices: even stride and base
        u16 = u16 && ld % 2 == 0 && ((uintptr_t)table & 7) == 0;
        c->merge16_last = u16;
        if (L.nphase > 0) {
            const int32_t cnt = (int32_t)(c->kp->xs_off[(size_t)m + 1] - b);
            const int64_t acc = (u16 && L.split ? 2 : 1) * cnt;
            const int64_t ring = std::max(L.rows, std::min(2 * L.rows, BLOCK_SMEM_ROWS - acc));
            const size_t smem = 128 * (size_t)(acc + ring);
            const BlockPhase *pg = (const BlockPhase *)c->kp->mblock_phases.ptr + L.phase_off;
            // one block an SM, of those this context may take: a block that waits for an SM would double the time
            const int sms = c->relax_sm_cap > 0 && c->relax_sm_cap < c->sms ? c->relax_sm_cap : c->sms;
            const unsigned blocks = (unsigned)std::min(u16 ? (n + 63) / 64 : (n + 31) / 32, sms);
            auto *fn = u16 ? k_merge_block<true> : k_merge_block<false>;
            fn<<<blocks, 32 * BLOCK_WARPS, smem, st>>>(table, ld, n, (const uint32_t *)c->kp->xs.ptr, (int32_t)b, cnt, pg,
                                                       (int32_t)L.nphase, L.split, (int32_t)ring, d_terms, k,
                                                       (uint32_t *)c->lvlmax.ptr + m, shadow, shadow_ld);
            e = cudaGetLastError();
        } else for (const StreamGroup &g : c->kp->mstream_groups[(size_t)m]) {
            const uint32_t *xg = (const uint32_t *)c->kp->xs.ptr + b + g.x0;
            const MergePhase *pg = (const MergePhase *)c->kp->mstream_phases.ptr + g.phase_off;
            if (u16)
                k_merge_stream16<<<(unsigned)((n + 63) / 64), 1024, (size_t)g.smem, st>>>(
                    table, ld, n, xg, (int32_t)g.cnt, pg, (int32_t)g.nphase, d_terms, k, (uint32_t *)c->lvlmax.ptr + m,
                    shadow, shadow_ld);
            else
                k_merge_stream<<<(unsigned)((n + 31) / 32), 1024, (size_t)g.smem, st>>>(
                    table, ld, n, xg, (int32_t)g.cnt, pg, (int32_t)g.nphase, d_terms, k, (uint32_t *)c->lvlmax.ptr + m);
            e = cudaGetLastError();
            if (e != cudaSuccess) break;
        }
    } else if (k <= MERGE_SMEM_KMAX) {
        const int64_t row_bytes = nstage * 4;
        if (row_bytes * 32 <= MERGE_SMEM_BYTES) e = merge_smem_launch<32>(c, table, ld, n, k, m, d_terms, st);
        else if (row_bytes * 16 <= MERGE_SMEM_BYTES) e = merge_smem_launch<16>(c, table, ld, n, k, m, d_terms, st);
        else if (row_bytes * 8 <= MERGE_SMEM_BYTES) e = merge_smem_launch<8>(c, table, ld, n, k, m, d_terms, st);
        else if (row_bytes * 4 <= MERGE_SMEM_BYTES) e = merge_smem_launch<4>(c, table, ld, n, k, m, d_terms, st);
        else if (row_bytes * 2 <= MERGE_SMEM_BYTES) e = merge_smem_launch<2>(c, table, ld, n, k, m, d_terms, st);
        else e = merge_smem_launch<1>(c, table, ld, n, k, m, d_terms, st);
    } else {
        const int64_t b = c->kp->xs_off[(size_t)m], cnt = c->kp->xs_off[(size_t)m + 1] - b;
        const int32_t xper = (int32_t)std::min<int64_t>(cnt, 64);
        dim3 grid((unsigned)((n + 31) / 32), (unsigned)((cnt + xper - 1) / xper));
        k_merge<<<grid, 256, 0, st>>>(table, ld, n, (const uint32_t *)c->kp->xs.ptr + b, (int32_t)cnt, xper, d_terms, k);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) return emv_fail(EMV_ERR_CUDA, "merge launch: %s", cudaGetErrorString(e));
    return EMV_OK;
}

// Status of a device CSR check: the same statuses, bound and messages as the
// host check emv_graph_check, whose connectivity part comes from the level-1
// closures instead (run_dp).
int scan_status(const GraphScan &s, int32_t n)
{
    if (s.bad & SCAN_BAD_ROWS) return emv_fail(EMV_ERR_BAD_INPUT, "graph: row_ptr not from 0 to arcs, non-decreasing");
    if (s.bad & SCAN_BAD_HEAD) return emv_fail(EMV_ERR_BAD_INPUT, "graph: arc head out of range");
    if (s.bad & SCAN_BAD_WEIGHT) return emv_fail(EMV_ERR_BAD_INPUT, "graph: negative weight");
    if (s.bad & SCAN_BIG_WEIGHT) return emv_fail(EMV_ERR_OVERFLOW, "graph: an arc weight reaches 2^30");
    // every finite d[X][v] is a Steiner tree's weight: at most (n-1) * max_w
    // and at most the weight of all edges (two arcs each)
    const int64_t bound = std::min<int64_t>((int64_t)(n - 1) * (int64_t)s.maxw, (int64_t)(s.sumw / 2));
    if (bound >= INF)
        return emv_fail(EMV_ERR_OVERFLOW, "graph: table values may reach 2^30 (bound %lld)", (long long)bound);
    return EMV_OK;
}

// Packs the arcs as int2 (c->adj) and checks the device CSR in the same
// kernel.  With check set, waits for the check and returns its status before
// any kernel of the DP reads the graph; the scan result stays in c->gscan.
static int pack_and_check(emv_ctx *c, int32_t n, int64_t arcs, const int32_t *row_ptr, const int32_t *col,
                          const int32_t *w, bool check, cudaStream_t st)
{
    int r = dev_reserve(c->adj, sizeof(int2) * (size_t)std::max<int64_t>(arcs, 1));
    if (!r) r = dev_reserve(c->hubs, sizeof(int32_t) * (size_t)n);
    if (r) return r;
    c->relax_arcs = arcs;
    GraphScan *d_scan = (GraphScan *)c->gscan.ptr;
    CUDA_TRY(cudaMemsetAsync(d_scan, 0, sizeof(GraphScan), st));
    k_pack_scan<<<grid_for(std::max<int64_t>(arcs, (int64_t)n + 1), 256, 4096), 256, 0, st>>>(
        row_ptr, n, col, w, (int2 *)c->adj.ptr, arcs, d_scan, relax_hub_min(n, arcs), (int32_t *)c->hubs.ptr);
    CUDA_TRY(cudaGetLastError());
    c->launches++;
    GraphScan *h = (GraphScan *)((char *)c->pinned + 1024);
    CUDA_TRY(cudaMemcpyAsync(h, d_scan, sizeof(GraphScan), cudaMemcpyDeviceToHost, st));
    if (!check) return EMV_OK;  // read later, behind an event or a synchronisation
    CUDA_TRY(cudaStreamSynchronize(st));
    return scan_status(*h, n);
}

// The DP proper on device data with packed arcs over the first kt of the k
// terminals (kt = k: the whole table; kt = k - 1: the rows of the subsets of
// C = {t_0..t_{k-2}}, all that the cost d[C][t_{k-1}] and a tree traced back
// from it read); fills those 2^kt rows.
// With check set, a level-1 closure that left a vertex unreached (the graph
// is not connected: the reference's table is undefined there, R:2077) makes
// the solve EMV_ERR_DISCONNECTED; the table is then not meaningful.
int run_dp(emv_ctx *c, int32_t n, const int32_t *row_ptr, const int2 *adj, int32_t k_all, int32_t kt,
           const int32_t *terms_host, int32_t *table, int64_t ld, cudaStream_t st, int64_t *cost_out, emv_timing *tm,
           bool check)
{
    const int32_t k = kt;
    int r = prepare_subsets(c, k, st);
    if (!r) r = reserve_relax(c, n);
    if (!r) r = dev_reserve(c->terms, sizeof(int32_t) * (size_t)k_all);
    if (r) return r;
    int32_t *d_terms = (int32_t *)c->terms.ptr;
    CUDA_TRY(cudaMemcpyAsync(d_terms, terms_host, sizeof(int32_t) * (size_t)k_all, cudaMemcpyHostToDevice, st));
    CUDA_TRY(cudaMemsetAsync(c->stat.ptr, 0, sizeof(DevStat), st));
    const uint32_t *xs = (const uint32_t *)c->kp->xs.ptr;
    int ev = 0;
    cudaEvent_t *E = c->ev;
    CUDA_TRY(cudaEventRecord(E[ev++], st));  // 0: start

    // Row 0 is the only row no level writes (R:2243-2259 fills every row).
    k_fill<<<grid_for(n, 256, 1024), 256, 0, st>>>(table, n, INF);
    c->launches++;
    CUDA_TRY(cudaEventRecord(E[ev++], st));  // 1: after fill

    // Level maxima: lvlmax[m] = largest value the merge of level m wrote
    // (level 1: its relaxation), all ones where the kernel does not record it.
    // They reach the host one level late, so no wait idles the device.
    uint32_t *d_max = (uint32_t *)c->lvlmax.ptr, *h_max = (uint32_t *)c->pinned + 64;
    // 16-bit shadow of the relaxed rows (stride a multiple of 64 vertices):
    // the 16-bit merge stages from it with 16-byte asynchronous copies.  Taken
    // when 16-bit values are allowed and the memory is free (with 1 GiB to
    // spare); without it the merge packs the int32 rows itself.
    uint16_t *shadow = nullptr;
    const int64_t sld = ((int64_t)n + 63) / 64 * 64;
    if (c->value_bits == 0 && k >= 3 && k <= MERGE_SMEM_KMAX) {  // the streamed merge's k
        const size_t need = sizeof(uint16_t) * (size_t)sld << k;
        size_t fr = 0, tot = 0;
        if (c->shadow.bytes >= need ||
            (cudaMemGetInfo(&fr, &tot) == cudaSuccess && need + ((size_t)1 << 30) < fr && dev_reserve(c->shadow, need) == EMV_OK))
            shadow = (uint16_t *)c->shadow.ptr;
        cudaGetLastError();
    }
    int64_t levels16 = 0, merges16 = 0, relax_launches = 1;
    CUDA_TRY(cudaMemsetAsync(d_max, 0xff, sizeof(uint32_t) * (EMV_MAX_K + 1), st));
    CUDA_TRY(cudaMemsetAsync(d_max + 1, 0, sizeof(uint32_t), st));

    // Level 1: k single-source closures (R:1988-2031).
    r = launch_narrow(c, row_ptr, adj, n, ld, table, xs + c->kp->xs_off[1], k, d_terms, st, d_max + 1, shadow, sld);
    if (r) return r;
    CUDA_TRY(cudaEventRecord(E[ev++], st));  // 2: after level 1
    CUDA_TRY(cudaMemcpyAsync(h_max + 1, d_max + 1, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaEventRecord(c->evmax[1], st));

    for (int32_t m = 2; m <= k; m++) {
        const int64_t b = c->kp->xs_off[(size_t)m], cnt = c->kp->xs_off[(size_t)m + 1] - b;
        // 16-bit merge staging when every sum of two lower-level values is
        // at most 65533 (M(j) bounds level j's values); from level 3 on, where
        // waiting for level m-1's maximum leaves its relaxation queued.
        // 16-bit relaxation records when M(m-1) + M(1) <= 32767: the split
        // {X \ t, t} bounds every merged value of level m by it, and relaxed
        // values never exceed merged ones (level 2 decides after its merge is
        // queued, so that no wait idles the device).
        bool m16 = false, u16 = false;
        if (c->value_bits == 0 && m >= 3) {
            CUDA_TRY(cudaEventSynchronize(c->evmax[m - 1]));
            m16 = merge16_allowed(h_max, m);
            u16 = relax16_allowed(h_max, m);
        }
        r = launch_merge(c, table, ld, n, k, m, d_terms, st, m16, shadow, sld);
        if (r) return r;
        merges16 += c->merge16_last;
        CUDA_TRY(cudaEventRecord(E[ev++], st));  // merge end of level m
        CUDA_TRY(cudaMemcpyAsync(h_max + m, d_max + m, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
        CUDA_TRY(cudaEventRecord(c->evmax[m], st));
        if (m == 2) {  // the scan's hub count has arrived too
            CUDA_TRY(cudaEventSynchronize(c->evmax[m - 1]));
            c->relax_nhubs = (int32_t)((const GraphScan *)((char *)c->pinned + 1024))->hubs;
            if (c->value_bits == 0) u16 = relax16_allowed(h_max, m);
        }
        levels16 += u16;
        const int32_t chunk = relax_chunk_rows_level(c, n, u16, cnt);
        for (int64_t off = 0; off < cnt; off += chunk) {
            const int32_t rows = (int32_t)std::min<int64_t>(chunk, cnt - off);
            if (rows <= (c->relax_nhubs > 0 ? 1 : RELAX_NARROW))
                r = launch_narrow(c, row_ptr, adj, n, ld, table, xs + b + off, rows, nullptr, st, nullptr, shadow, sld);
            else r = launch_relax(c, row_ptr, adj, n, ld, table, xs + b + off, rows, st, u16, shadow, sld);
            if (r) return r;
            relax_launches++;
        }
        CUDA_TRY(cudaEventRecord(E[ev++], st));  // relax end of level m
    }

    // Cost d[C][q] (R:2137-2138) and the device status, then one host sync.
    int32_t *hp = (int32_t *)c->pinned;
    if (k_all >= 2) {
        const int64_t C = ((int64_t)1 << (k_all - 1)) - 1;
        CUDA_TRY(cudaMemcpyAsync(hp, table + C * ld + terms_host[k_all - 1], sizeof(int32_t), cudaMemcpyDeviceToHost,
                                 st));
    } else {
        hp[0] = INF;
    }
    CUDA_TRY(cudaMemcpyAsync(hp + 2, c->stat.ptr, sizeof(DevStat), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    CUDA_TRY(cudaGetLastError());
    DevStat ds;
    std::memcpy(&ds, hp + 2, sizeof(ds));
    if (ds.err) return emv_dev_status_to_emv(ds.err);
    if (check && h_max[1] >= (uint32_t)INF)
        return emv_fail(EMV_ERR_DISCONNECTED, "graph: not connected (a vertex is unreachable from terminal 1)");
    *cost_out = (k_all >= 2 && hp[0] < INF) ? (int64_t)hp[0] : INT64_MAX;
    if (tm) {
        float ms = 0;
        cudaEventElapsedTime(&ms, E[0], E[1]);
        tm->zero_ms = ms;
        cudaEventElapsedTime(&ms, E[1], E[2]);
        tm->level1_ms = ms;
        tm->merge_ms = tm->relax_ms = 0;
        for (int32_t m = 2; m <= k; m++) {
            const int b = 2 + 2 * (m - 2);  // E[b] merge start, E[b+1] relax start, E[b+2] level end
            cudaEventElapsedTime(&ms, E[b], E[b + 1]);
            tm->merge_ms += ms;
            cudaEventElapsedTime(&ms, E[b + 1], E[b + 2]);
            tm->relax_ms += ms;
        }
        cudaEventElapsedTime(&ms, E[1], E[ev - 1]);
        tm->kernel_ms = ms;
        tm->relax_sweeps = (int64_t)ds.sweeps;
        tm->relax16_levels = levels16;
        tm->merge16_levels = merges16;
        tm->relax_launches = relax_launches;
    }
    return EMV_OK;
}

static int check_k(int32_t n, int32_t k, const int32_t *terms)
{
    if (k < 1 || k > EMV_MAX_K) return emv_fail(EMV_ERR_BAD_INPUT, "k = %d outside [1, %d]", k, EMV_MAX_K);
    if (!terms) return emv_fail(EMV_ERR_BAD_INPUT, "null terminals");
    for (int32_t i = 0; i < k; i++)
        if (terms[i] < 0 || terms[i] >= n) return emv_fail(EMV_ERR_BAD_INPUT, "terminal %d out of range", i);
    return EMV_OK;
}

// Whether a solve over kt terminals' subsets runs as one launch (then p is its
// shape).  If not, the graph has been packed, and checked with check set; past
// the line of resident_plan that tells whether it has hubs.
static int plan_solve(emv_ctx *c, int32_t n, int64_t arcs, const int32_t *row_ptr, const int32_t *col, const int32_t *w,
                      int32_t kt, bool host_table, bool check, cudaStream_t st, ResidentPlan &p, bool &resident)
{
    resident = resident_plan(c, n, arcs, kt, host_table, false, p);
    if (resident) return EMV_OK;
    const int r = pack_and_check(c, n, arcs, row_ptr, col, w, check, st);
    if (r || !resident_plan(c, n, arcs, kt, host_table, true, p)) return r;
    if (!check) CUDA_TRY(cudaStreamSynchronize(st));
    resident = ((const GraphScan *)((char *)c->pinned + 1024))->hubs > 0;
    return EMV_OK;
}

extern "C" int emv_kernel_dev(emv_ctx *c, int32_t n, int64_t arcs, const int32_t *d_row_ptr, const int32_t *d_col,
                              const int32_t *d_w, int32_t k, const int32_t *terminals, int32_t *d_table, int64_t ld,
                              int64_t *cost_out, void *stream)
{
    if (!c || !d_row_ptr || (arcs > 0 && (!d_col || !d_w)) || !d_table || !cost_out || n <= 0 || arcs < 0 ||
        arcs >= INT32_MAX || ld < n)
        return emv_fail(EMV_ERR_BAD_INPUT, "emv_kernel_dev: bad arguments");
    int r = check_k(n, k, terminals);
    if (r) return r;
    CUDA_TRY(cudaSetDevice(c->device));
    cudaStream_t st = (cudaStream_t)stream;
    c->launches = 0;
    ResidentPlan plan;
    bool resident;
    r = plan_solve(c, n, arcs, d_row_ptr, d_col, d_w, k, false, true, st, plan, resident);
    if (r) return r;
    if (resident) {
        r = resident_launch(c, plan, n, arcs, d_row_ptr, d_col, d_w, terminals, k, k, d_table, ld, true, st);
        if (r) return r;
        CUDA_TRY(cudaStreamSynchronize(st));
        return resident_finish(c, n, k, true, true, cost_out, nullptr);
    }
    return run_dp(c, n, d_row_ptr, (const int2 *)c->adj.ptr, k, k, terminals, d_table, ld, st, cost_out, nullptr, true);
}

// Words of the traceback's result that come back with its first copy.
constexpr size_t TB_FIRST_EDGES = 1024;
constexpr size_t TB_FIRST_WORDS = TB_HEAD + 3 * TB_FIRST_EDGES;
static_assert(PINNED_TB + 4 * TB_FIRST_WORDS <= PINNED_BYTES, "traceback words fit the pinned buffer");

static int32_t traceback_cap(int32_t n) { return std::max(64, 2 * n); }
static int32_t traceback_chunks(int32_t n) { return traceback_cap(n) / TB_CHUNK + TB_TASKS + 1; }

// Buffers of a traceback, to be had before anything of the solve is enqueued
// that would still run when a failed call returns.
static int reserve_traceback(emv_ctx *c, int32_t n)
{
    int r = dev_reserve(c->tb_edges, sizeof(int32_t) * (TB_CHUNK * 3 + 1) * (size_t)traceback_chunks(n));
    if (!r)
        r = dev_reserve(c->tb_out,
                        sizeof(int32_t) * (TB_HEAD + 3 * std::max<size_t>((size_t)traceback_cap(n), TB_FIRST_EDGES)));
    if (!r) r = dev_reserve(c->tb_work, sizeof(int32_t) * 3 * (size_t)n);
    return r;
}

// Enqueues the traceback (its buffers are reserved) and the copy of its head
// and first edges into the pinned buffer.  skip_err, skip_refused (or null):
// device words that say, where not 0, that there is nothing to trace.
static int launch_traceback(emv_ctx *c, int32_t n, const int32_t *row_ptr, const int2 *adj, int32_t k,
                            const int32_t *d_terms, const int32_t *table, int64_t ld, const uint32_t *skip_err,
                            const uint32_t *skip_refused, cudaStream_t st)
{
    const int32_t cap = traceback_cap(n), nchunks = traceback_chunks(n);
    int32_t *work = (int32_t *)c->tb_work.ptr;
    TbArgs a;
    a.table = table;
    a.ld = ld;
    a.n = n;
    a.k = k;
    a.row_ptr = row_ptr;
    a.adj = adj;
    a.terms = d_terms;
    a.skip_err = skip_err;
    a.skip_refused = skip_refused;
    a.chunks = (int32_t *)c->tb_edges.ptr;
    a.next = a.chunks + (size_t)nchunks * TB_CHUNK * 3;
    a.nchunks = nchunks;
    a.out = (int32_t *)c->tb_out.ptr;
    a.cap = cap;
    a.queue = work;
    a.parent = work + n;
    a.stamp = work + 2 * (size_t)n;
    a.max_steps = 4 * n + 64 * k + 1024;
    k_traceback<<<1, 32 * TB_WARPS, 0, st>>>(a);
    CUDA_TRY(cudaGetLastError());
    c->launches++;
    CUDA_TRY(cudaMemcpyAsync((char *)c->pinned + PINNED_TB, a.out, sizeof(int32_t) * TB_FIRST_WORDS, cudaMemcpyDeviceToHost,
                             st));
    return EMV_OK;
}

// Reduces the edges of a finished traceback (the stream has been waited for)
// to a tree.
static int finish_traceback(emv_ctx *c, int32_t n, emv_result *out)
{
    const int32_t *head = (const int32_t *)((char *)c->pinned + PINNED_TB), *e = head + TB_HEAD;
    const size_t edges = (size_t)head[0];
    uint64_t ns;
    std::memcpy(&ns, head + 2, sizeof(ns));
    out->timing.traceback_ms = (float)(ns * 1e-6);
    if (head[1]) return emv_dev_status_to_emv((uint32_t)head[1]);
    std::vector<int32_t> all;
    if (edges > TB_FIRST_EDGES) {
        all.resize(3 * edges);
        CUDA_TRY(cudaMemcpy(all.data(), (const int32_t *)c->tb_out.ptr + TB_HEAD, sizeof(int32_t) * all.size(),
                            cudaMemcpyDeviceToHost));
        e = all.data();
    }
    // Keep a spanning forest of the emitted edges: duplicates and zero-weight
    // cycles (possible only through zero-weight arcs) are dropped.  Vertices
    // are their own parent (-1) until an edge touches them, and again after.
    if (c->forest.size() < (size_t)n) c->forest.assign((size_t)n, -1);
    std::vector<int32_t> &parent = c->forest;
    auto find = [&](int32_t x) {
        while (parent[(size_t)x] >= 0) {
            const int32_t p = parent[(size_t)x];
            if (parent[(size_t)p] >= 0) parent[(size_t)x] = parent[(size_t)p];
            x = p;
        }
        return x;
    };
    int64_t count = 0, weight = 0;
    for (size_t i = 0; i < edges; i++) {
        const int32_t u = e[3 * i], v = e[3 * i + 1], wt = e[3 * i + 2];
        const int32_t ru = find(u), rv = find(v);
        if (ru == rv) continue;
        parent[(size_t)ru] = rv;
        if (out->tree && count < out->tree_cap) {
            out->tree[3 * count] = u;
            out->tree[3 * count + 1] = v;
            out->tree[3 * count + 2] = wt;
        }
        count++;
        weight += wt;
    }
    for (size_t i = 0; i < edges; i++) parent[(size_t)e[3 * i]] = parent[(size_t)e[3 * i + 1]] = -1;
    out->tree_count = count;
    out->tree_weight = weight;
    if (out->tree && count > out->tree_cap)
        return emv_fail(EMV_ERR_BAD_INPUT, "tree buffer holds %lld edges, need %lld", (long long)out->tree_cap,
                        (long long)count);
    return EMV_OK;
}

int solve_on_device(emv_ctx *c, int32_t n, int64_t arcs, const int32_t *row_ptr, const int32_t *col,
                    const int32_t *w, const int32_t *terms, int32_t k, int32_t flags, emv_result *out,
                    cudaStream_t st)
{
    const bool check = !(flags & EMV_SOLVE_NOCHECK);
    const int64_t ld = ((int64_t)n + 31) / 32 * 32;
    // Without a table to return, the rows of subsets that hold the last
    // terminal are read by nothing: neither by the cost d[C][t_{k-1}] nor by
    // the rows and the traceback below it.
    const bool whole = ((flags & EMV_SOLVE_TABLE) && out->table) || (flags & EMV_SOLVE_ALL_ROWS);
    const int32_t kt = whole ? k : table_terminals(k);
    const size_t tbytes = sizeof(int32_t) * (size_t)ld << kt;
    ResidentPlan plan;
    bool resident;
    int r = plan_solve(c, n, arcs, row_ptr, col, w, kt, (flags & EMV_SOLVE_TABLE) && out->table, check, st, plan, resident);
    if (!r) r = dev_reserve(c->table, tbytes);
    if (r) return r;
    int32_t *table = (int32_t *)c->table.ptr;
    std::memset(&out->timing, 0, sizeof(out->timing));
    out->tree_count = 0;
    out->tree_weight = 0;
    const bool tree = (flags & EMV_SOLVE_TREE) && k >= 2;
    if (tree) r = reserve_traceback(c, n);
    if (r) return r;
    if (resident) {  // one wait for the solve and its tree
        r = resident_launch(c, plan, n, arcs, row_ptr, col, w, terms, k, kt, table, ld, check, st);
        if (!r && tree) {
            const ResidentWords d = resident_words(c);
            r = launch_traceback(c, n, row_ptr, (const int2 *)c->adj.ptr, k, d.terms, table, ld, d.err, d.refused, st);
        }
        if (r) return r;
        CUDA_TRY(cudaStreamSynchronize(st));
        r = resident_finish(c, n, k, check, check, &out->cost, &out->timing);
    } else {
        const int2 *adj = (const int2 *)c->adj.ptr;
        r = run_dp(c, n, row_ptr, adj, k, kt, terms, table, ld, st, &out->cost, &out->timing, check);
        if (!r && tree) {
            r = launch_traceback(c, n, row_ptr, adj, k, (const int32_t *)c->terms.ptr, table, ld, nullptr, nullptr, st);
            if (r) return r;
            CUDA_TRY(cudaStreamSynchronize(st));
        }
    }
    if (!r && tree) r = finish_traceback(c, n, out);
    if (r) return r;
    if ((flags & EMV_SOLVE_TABLE) && out->table) {
        CUDA_TRY(cudaMemcpy2DAsync(out->table, sizeof(int32_t) * (size_t)n, table, sizeof(int32_t) * (size_t)ld,
                                   sizeof(int32_t) * (size_t)n, (size_t)1 << k, cudaMemcpyDeviceToHost, st));
        CUDA_TRY(cudaStreamSynchronize(st));
    }
    out->timing.launches = c->launches;
    return EMV_OK;
}

// Copies a host CSR to the device.  Graphs of up to GRAPH_STAGE_BYTES go through
// one pinned buffer in one copy (three copies from pageable memory cost a
// small solve 15 us); larger ones straight from the caller's arrays, which the
// driver reads at 160-180 GB/s, close to the 200 GB/s from pinned memory.
constexpr size_t GRAPH_STAGE_BYTES = 1 << 20;

static int graph_to_device(emv_ctx *c, const emv_graph *g, cudaStream_t st, const int32_t **row, const int32_t **col,
                           const int32_t **w)
{
    const size_t rows = (size_t)g->n + 1, arcs = (size_t)g->arcs;
    const size_t col_at = (rows + 3) / 4 * 4, w_at = col_at + (arcs + 3) / 4 * 4, words = w_at + arcs;
    int r = dev_reserve(c->g_all, sizeof(int32_t) * words);
    if (r) return r;
    int32_t *d = (int32_t *)c->g_all.ptr;
    *row = d;
    *col = d + col_at;
    *w = d + w_at;
    if (sizeof(int32_t) * words <= GRAPH_STAGE_BYTES && !c->g_stage &&
        cudaMallocHost(&c->g_stage, GRAPH_STAGE_BYTES) != cudaSuccess) {
        cudaGetLastError();
        c->g_stage = nullptr;
    }
    if (sizeof(int32_t) * words <= GRAPH_STAGE_BYTES && c->g_stage) {
        // every call waits for its stream before it returns, so the buffer is free
        int32_t *h = (int32_t *)c->g_stage;
        std::memcpy(h, g->row_ptr, sizeof(int32_t) * rows);
        if (arcs > 0) {
            std::memcpy(h + col_at, g->col, sizeof(int32_t) * arcs);
            std::memcpy(h + w_at, g->w, sizeof(int32_t) * arcs);
        }
        CUDA_TRY(cudaMemcpyAsync(d, h, sizeof(int32_t) * words, cudaMemcpyHostToDevice, st));
        return EMV_OK;
    }
    CUDA_TRY(cudaMemcpyAsync(d, g->row_ptr, sizeof(int32_t) * rows, cudaMemcpyHostToDevice, st));
    if (arcs > 0) {
        CUDA_TRY(cudaMemcpyAsync(d + col_at, g->col, sizeof(int32_t) * arcs, cudaMemcpyHostToDevice, st));
        CUDA_TRY(cudaMemcpyAsync(d + w_at, g->w, sizeof(int32_t) * arcs, cudaMemcpyHostToDevice, st));
    }
    return EMV_OK;
}

extern "C" int emv_solve(emv_ctx *c, const emv_graph *g, const int32_t *terminals, int32_t k, int32_t flags,
                         emv_result *out, void *stream)
{
    if (!c || !out) return emv_fail(EMV_ERR_BAD_INPUT, "null argument");
    int r = emv_graph_validate(g);
    if (r) return r;
    r = check_k(g->n, k, terminals);
    if (r) return r;
    CUDA_TRY(cudaSetDevice(c->device));
    cudaStream_t st = (cudaStream_t)stream;
    c->launches = 0;
    const int32_t *row, *col, *w;
    r = graph_to_device(c, g, st, &row, &col, &w);
    if (r) return r;
    return solve_on_device(c, g->n, g->arcs, row, col, w, terminals, k, flags, out, st);
}

extern "C" int emv_solve_dev(emv_ctx *c, const emv_graph *d_g, const int32_t *terminals, int32_t k, int32_t flags,
                             emv_result *out, void *stream)
{
    if (!c || !out) return emv_fail(EMV_ERR_BAD_INPUT, "null argument");
    int r = emv_graph_validate(d_g);
    if (r) return r;
    r = check_k(d_g->n, k, terminals);
    if (r) return r;
    CUDA_TRY(cudaSetDevice(c->device));
    c->launches = 0;
    return solve_on_device(c, d_g->n, d_g->arcs, d_g->row_ptr, d_g->col, d_g->w, terminals, k, flags, out,
                           (cudaStream_t)stream);
}

// Up to here one CTA's shared memory beats the whole GPU's sweeps: one CTA
// reads all arcs in every dense round.  Calls by one launch and by narrow
// records, random graphs of n vertices and arcs: 300, 88 000 0.16 and 0.20 ms;
// 1000, 120 000 0.28 and 0.21; 4000, 100 000 0.239 and 0.239; 8192, 80 000 0.23 and
// 0.22; 8192, 500 000 0.92 and 0.32; grid of 90 x 90 0.38 and 0.95.  Beyond, graphs
// whose arcs crowd in a few vertices stay: narrow records leave 8 neighbouring
// vertices of such a graph to a warp (5368, 192 000 arcs, half of them at 10 or at
// 100 vertices 0.32 and 1.53, 0.27 and 0.65 ms; at random 0.28 and 0.25).
constexpr int32_t SSSP_RESIDENT_N = 8192;
constexpr int64_t SSSP_RESIDENT_ARCS = 100000;
static bool sssp_resident(const emv_graph *g)
{
    if (g->n > SSSP_RESIDENT_N) return false;
    if (g->arcs <= SSSP_RESIDENT_ARCS) return true;
    int64_t most = 0;  // arcs of 8 neighbours
    for (int32_t v = 0; v < g->n; v += 8)
        most = std::max(most, (int64_t)g->row_ptr[std::min(v + 8, g->n)] - g->row_ptr[v]);
    return 64 * most > g->arcs;
}

extern "C" int emv_sssp(emv_ctx *c, const emv_graph *g, int32_t source, int64_t *dist_out, float *ms_out, void *stream)
{
    if (!c || !dist_out) return emv_fail(EMV_ERR_BAD_INPUT, "null argument");
    int r = emv_graph_validate(g);
    if (r) return r;
    if (source < 0 || source >= g->n) return emv_fail(EMV_ERR_BAD_INPUT, "source out of range");
    CUDA_TRY(cudaSetDevice(c->device));
    cudaStream_t st = (cudaStream_t)stream;
    const int32_t n = g->n;
    const int64_t arcs = g->arcs;
    // row 1 = {source}; rows of whole quads
    const int64_t ld = ((int64_t)n + 3) / 4 * 4;
    ResidentPlan plan;
    // the line of resident_plan on arcs is that of solves
    const bool resident = sssp_resident(g) && resident_plan(c, n, 0, 1, false, false, plan);
    r = dev_reserve(c->table, sizeof(int32_t) * 2 * (size_t)ld);
    if (!r) r = prepare_subsets(c, 1, st);
    if (!r && !resident) r = reserve_relax(c, n);
    if (!r && !resident) r = dev_reserve(c->terms, sizeof(int32_t));
    if (!r && c->h_dist_n < n) {
        if (c->h_dist) cudaFreeHost(c->h_dist);
        c->h_dist = nullptr;
        c->h_dist_n = 0;
        if (cudaMallocHost((void **)&c->h_dist, sizeof(int32_t) * (size_t)n) != cudaSuccess) {
            cudaGetLastError();
            r = emv_fail(EMV_ERR_OOM, "pinned distances of %d vertices", n);
        } else {
            c->h_dist_n = n;
        }
    }
    if (r) return r;
    const int32_t *row, *col, *w;
    r = graph_to_device(c, g, st, &row, &col, &w);
    if (r) return r;
    int32_t *table = (int32_t *)c->table.ptr;
    if (resident) {
        int64_t cost;
        r = resident_launch(c, plan, n, arcs, row, col, w, &source, 1, 1, table, ld, true, st);
        if (r) return r;
        CUDA_TRY(cudaMemcpyAsync(c->h_dist, table + ld, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToHost, st));
        CUDA_TRY(cudaStreamSynchronize(st));
        r = resident_finish(c, n, 1, true, false, &cost, nullptr);
        if (r) return r;
    } else {
        CUDA_TRY(cudaMemcpyAsync(c->terms.ptr, &source, sizeof(int32_t), cudaMemcpyHostToDevice, st));
        CUDA_TRY(cudaMemsetAsync(c->stat.ptr, 0, sizeof(DevStat), st));
        r = pack_and_check(c, n, arcs, row, col, w, false, st);
        if (r) return r;
        CUDA_TRY(cudaEventRecord(c->ev[0], st));
        r = launch_narrow(c, row, (const int2 *)c->adj.ptr, n, ld, table, (const uint32_t *)c->kp->xs.ptr, 1,
                          (const int32_t *)c->terms.ptr, st, nullptr, nullptr, 0, (const GraphScan *)c->gscan.ptr);
        if (r) return r;
        CUDA_TRY(cudaEventRecord(c->ev[1], st));
        GraphScan *hs = (GraphScan *)((char *)c->pinned + 1024);
        DevStat *ds = (DevStat *)((char *)c->pinned + 1536);
        CUDA_TRY(cudaMemcpyAsync(ds, c->stat.ptr, sizeof(DevStat), cudaMemcpyDeviceToHost, st));
        CUDA_TRY(cudaMemcpyAsync(c->h_dist, table + ld, sizeof(int32_t) * (size_t)n, cudaMemcpyDeviceToHost, st));
        CUDA_TRY(cudaStreamSynchronize(st));
        r = scan_status(*hs, n);
        if (r) return r;
        if (ds->err) return emv_dev_status_to_emv(ds->err);
    }
    if (ms_out) cudaEventElapsedTime(ms_out, c->ev[0], c->ev[1]);
    for (int32_t v = 0; v < n; v++) dist_out[v] = c->h_dist[v] >= INF ? INT64_MAX : (int64_t)c->h_dist[v];
    return EMV_OK;
}
