// emv_batch.cu -- many independent instances in one persistent launch (C ABI),
// and the autotuner that picks the per-class tile shapes.
//
// No counterpart in the reference, which solves one instance per process
// (reader/reader-el.c:2355-2536); each instance's values are those of its
// emv_kernel (R:1966-2139).
#include "emv_batch.cuh"
#include "emv_solver.h"
#include "emv_batch_host.h"
#include "emv_resident.h"

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

constexpr int32_t BATCH_CUT_MIN = 768;
constexpr int32_t BATCH_FEW_BLOCKS = 16;

namespace {

// f(i) for i in [0, count) on up to 16 host threads (chunks of 16 indices).
template <class F> void host_parallel_for(int64_t count, F f)
{
    const unsigned hw = std::thread::hardware_concurrency();
    const int64_t T = std::min<int64_t>({16, (int64_t)(hw ? hw : 1), (count + 63) / 64});
    if (T <= 1) {
        for (int64_t i = 0; i < count; i++) f(i);
        return;
    }
    std::atomic<int64_t> next{0};
    auto work = [&]() {
        for (;;) {
            const int64_t i0 = next.fetch_add(16);
            if (i0 >= count) return;
            for (int64_t i = i0; i < std::min(count, i0 + 16); i++) f(i);
        }
    };
    std::vector<std::thread> th;
    for (int64_t t = 1; t < T; t++) th.emplace_back(work);
    work();
    for (std::thread &t : th) t.join();
}

}  // namespace

using namespace emv;

namespace {

int32_t pow2_floor(int32_t x)
{
    int32_t p = 1;
    while (p * 2 <= x) p *= 2;
    return p;
}

}  // namespace

int32_t batch_class_of(int32_t n, int32_t k)
{
    const int32_t nb = n <= 256 ? 0 : n <= 1024 ? 1 : n <= 4096 ? 2 : 3;
    const int32_t kb = k <= 6 ? 0 : k <= 8 ? 1 : 2;
    return nb * 3 + kb;
}

bool batch_fits(int32_t n, int32_t k)
{
    return k >= 1 && k <= BATCH_KMAX && (int64_t)n * 2 * 4 <= BATCH_SMEM_BYTES &&
           ((int64_t)32 << k) * 4 <= BATCH_SMEM_BYTES && resident_fits(n, k);
}

uint32_t pack_arcs(const emv_graph &g, int2 *adj)
{
    uint32_t most = 0;
    for (int64_t e = 0; e < g.arcs; e++) {
        adj[e] = make_int2(g.col[e], g.w[e]);
        most = std::max(most, (uint32_t)g.w[e]);
    }
    return most;
}

BatchGraph batch_graph(const int32_t *row_ptr, int32_t n, uint32_t most, int32_t hub_min)
{
    int64_t pairs = 0;
    for (int32_t v0 = 0; v0 < n; v0 += 32) {
        int32_t width = 0;
        for (int32_t v = v0; v < std::min(n, v0 + 32); v++) {
            const int32_t deg = row_ptr[v + 1] - row_ptr[v];
            if (deg <= hub_min) width = std::max(width, (deg + 1) / 2);
        }
        pairs += width;
    }
    const bool narrow = most < RES_MAX_W;
    return {narrow, pairs * 32 * (int64_t)(narrow ? sizeof(uint2) : sizeof(int4))};
}

// Fitted to one-CTA solves (n = 128 .. 4096, kt = 7 .. 9): closures 0.68 ns an
// arc and row, merges 0.016 ns a (subset pair, vertex), 15 us a level.
double batch_work(int32_t n, int32_t kt, int64_t arcs, int32_t lo, int32_t hi)
{
    const double all = 0.68e-3 * std::pow(2.0, kt) * (double)arcs + 0.016e-3 * std::pow(3.0, kt) * n;
    return all * (hi - lo + 1) / kt + 15.0 * (hi - lo + 1);
}

void batch_plan(const std::vector<double> &work, const std::vector<int64_t> &states, int32_t blocks, int32_t max_size,
                std::vector<int32_t> &order, std::vector<int32_t> &size)
{
    const int64_t count = (int64_t)work.size();
    double total = 0;
    for (double w : work) total += w;
    // A team large enough that the instance takes at most a third of the
    // batch's fair time (and not below 100 us, where barriers take over), as
    // far as a CTA has more than a state of the widest level a thread before its
    // team is doubled; two where the teams may have to take turns on the CTAs,
    // eight where there are more than a quarter as many instances as CTAs: a team
    // of CTAs with little to do takes longer in all than one CTA.  107 instances
    // on 152 CTAs, with one state throughout, four and eight: n = 64, 1088 edges,
    // k = 8 0.50, 0.22 and 0.22 ms, n = 33, 560 edges, k = 10 1.08, 0.45 and 0.34, n =
    // 130, 650 edges, k = 10 1.10, 0.72 and 0.64; 20 of n = 33, 560 edges with one and
    // two 0.35 and 0.22; one of n = 500, 40 000 edges, k = 6 0.43 and 0.49.
    const double most = std::max(100.0, total / blocks * 0.35);
    size.assign((size_t)count, 1);
    for (int64_t i = 0; i < count; i++) {
        int32_t g = 1;
        while (2 * g <= max_size && 2 * g <= blocks && work[(size_t)i] / g > most &&
               states[(size_t)i] > (int64_t)RES_THREADS * g * (count * 2 * g <= blocks ? 1 : count * 4 <= blocks ? 2 : 8))
            g *= 2;
        size[(size_t)i] = g;
    }
    order.resize((size_t)count);
    for (int64_t i = 0; i < count; i++) order[(size_t)i] = (int32_t)i;
    std::stable_sort(order.begin(), order.end(), [&](int32_t x, int32_t y) {
        if (size[(size_t)x] != size[(size_t)y]) return size[(size_t)x] > size[(size_t)y];
        return work[(size_t)x] > work[(size_t)y];
    });
}

void batch_shape(const emv_ctx *c, int64_t arcs, BatchInst &d)
{
    const int32_t cls = batch_class_of(d.n, d.k);
    const int32_t rcap = c->tune_rcap[cls] > 0 ? pow2_floor(c->tune_rcap[cls]) : 0;
    const int32_t most = (int32_t)((resident_max_rows(d.kt) + d.size - 1) / d.size);
    d.rows = rcap > 0 ? std::min(most, rcap) : most;
    d.mw = resident_merge_width(d.n, d.kt, d.size, c->tune_mw[cls] > 0 ? 32 * pow2_floor(c->tune_mw[cls]) : 0);
    d.inv_slices = res_inv_slices(d.n);
    d.spin_limit = res_spin_limit(d.n, arcs, most);
    d.hub_min = res_hub_min(d.n, arcs, d.kt);
}

int32_t batch_blocks(const emv_ctx *c, int64_t ctas, int32_t cap)
{
    const int32_t most = cap > 0 ? std::min(cap, c->batch_blocks) : c->batch_blocks;
    return (int32_t)std::min<int64_t>(most, std::max<int64_t>(1, ctas));
}

int prepare_batch_subsets(emv_ctx *c, cudaStream_t st)
{
    if (c->bxs_ready) return EMV_OK;
    std::vector<uint32_t> all;
    std::vector<int32_t> off((size_t)(BATCH_KMAX + 1) * (BATCH_KMAX + 2), 0);
    for (int32_t k = 1; k <= BATCH_KMAX; k++) {
        std::vector<uint32_t> xs;
        std::vector<int64_t> lo;
        subset_levels(k, xs, lo);
        const int32_t base = (int32_t)all.size();
        for (int32_t m = 0; m <= k + 1; m++) off[(size_t)k * (BATCH_KMAX + 2) + m] = base + (int32_t)lo[(size_t)m];
        all.insert(all.end(), xs.begin(), xs.end());
    }
    int r = dev_reserve(c->bxs, sizeof(uint32_t) * all.size());
    if (!r) r = dev_reserve(c->bxs_off, sizeof(int32_t) * off.size());
    if (r) return r;
    CUDA_TRY(cudaMemcpyAsync(c->bxs.ptr, all.data(), sizeof(uint32_t) * all.size(), cudaMemcpyHostToDevice, st));
    CUDA_TRY(cudaMemcpyAsync(c->bxs_off.ptr, off.data(), sizeof(int32_t) * off.size(), cudaMemcpyHostToDevice, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    c->bxs_ready = true;
    return EMV_OK;
}

int batch_kernel_setup(emv_ctx *c)
{
    if (c->batch_blocks > 0) return EMV_OK;
    CUDA_TRY(cudaFuncSetAttribute(k_batch, cudaFuncAttributeMaxDynamicSharedMemorySize, RESIDENT_SMEM));
    int per_sm = 0;
    CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch, RES_THREADS, RESIDENT_SMEM));
    c->batch_blocks = std::max(1, per_sm) * c->sms;
    return EMV_OK;
}

// Whether some team has more than one CTA.
static bool batch_teams(const BatchArgs &a) { return a.end[BATCH_SIZES - 2] > 0; }

// Launches k_batch on `blocks` CTAs over prepared descriptors.  Teams wait for
// their CTAs, so the launch is cooperative unless every team is a single CTA.
int launch_batch(emv_ctx *c, const BatchArgs &args, int32_t blocks, int32_t lines, cudaStream_t st)
{
    int r = batch_kernel_setup(c);
    if (r) return r;
    CUDA_TRY(cudaMemsetAsync(args.ctl, 0, sizeof(uint32_t) * 32 * (size_t)lines, st));
    BatchArgs a = args;
    void *p[] = {&a};
    if (batch_teams(a))
        CUDA_TRY(cudaLaunchCooperativeKernel((const void *)k_batch, dim3((unsigned)blocks), dim3(RES_THREADS), p,
                                             (size_t)RESIDENT_SMEM, st));
    else
        CUDA_TRY(cudaLaunchKernel((const void *)k_batch, dim3((unsigned)blocks), dim3(RES_THREADS), p,
                                  (size_t)RESIDENT_SMEM, st));
    return EMV_OK;
}

// Where a batch is cut into two launches: behind the instances of teams and at
// least half of the work, so that the host checks and packs the other (smaller)
// instances while these run.  Packing takes about a fifth of the time that
// the packed instances run, so a batch of a few hundred gains nothing.
static int32_t batch_cut(const BatchOrder &ord)
{
    const int32_t count = (int32_t)ord.ids.size();
    if (count < BATCH_CUT_MIN) return count;
    double total = 0, part = 0;
    for (double w : ord.work) total += w;
    int32_t cut = 0;
    while (cut < count && (ord.size[(size_t)cut] > 1 || part < 0.5 * total)) part += ord.work[(size_t)cut++];
    return count - cut < BATCH_CUT_MIN / 2 ? count : cut;
}

// emv_batch_solve and emv_batch_solve_tables: tables_out (or null) receives
// the finished table of every instance whose entry is not null.
static int batch_solve(emv_ctx *c, const emv_instance *inst, int32_t count, int64_t *costs_out,
                       int32_t *const *tables_out, emv_batch_stats *stats, void *stream)
{
    if (!c || (count > 0 && (!inst || !costs_out)) || count < 0)
        return emv_fail(EMV_ERR_BAD_INPUT, "emv_batch_solve: bad arguments");
    if (count == 0) return EMV_OK;
    CUDA_TRY(cudaSetDevice(c->device));
    cudaStream_t st = (cudaStream_t)stream;
    const auto t0 = std::chrono::steady_clock::now();
    // Admission checks: sizes first (the layout follows from them), the arrays
    // when an instance is packed; the failing instance of the lowest index is
    // reported.
    std::vector<int> bad((size_t)count, 0);
    std::vector<std::string> why((size_t)count);
    auto noted = [&](int64_t i, int r) {
        if (r) {
            bad[(size_t)i] = r;
            why[(size_t)i] = emv_last_error();
        }
        return r == 0;
    };
    auto check_sizes = [&](int64_t i) {
        const emv_instance &I = inst[i];
        int r = emv_graph_validate(&I.g);
        if (!r && !batch_fits(I.g.n, I.k))
            r = emv_fail(EMV_ERR_BAD_INPUT, "n = %d, k = %d outside the batched range (k <= %d)", I.g.n, I.k, BATCH_KMAX);
        if (!r && !I.terminals) r = emv_fail(EMV_ERR_BAD_INPUT, "null terminals");
        return noted(i, r);
    };
    auto check_arrays = [&](int64_t i) {
        const emv_instance &I = inst[i];
        int r = EMV_OK;
        for (int32_t t = 0; !r && t < I.k; t++)
            if (I.terminals[t] < 0 || I.terminals[t] >= I.g.n) r = emv_fail(EMV_ERR_BAD_INPUT, "terminal out of range");
        if (!r) r = emv_graph_check(&I.g, nullptr);
        return noted(i, r);
    };
    auto first_bad = [&]() {
        for (int32_t i = 0; i < count; i++)
            if (bad[(size_t)i]) return emv_fail(bad[(size_t)i], "instance %d: %s", i, why[(size_t)i].c_str());
        return (int)EMV_OK;
    };
    bool sizes_ok = true;
    for (int32_t i = 0; i < count; i++) sizes_ok &= check_sizes(i);
    if (!sizes_ok) {  // an instance before it may fail the other checks
        host_parallel_for(count, [&](int64_t i) {
            if (!bad[(size_t)i]) check_arrays(i);
        });
        return first_bad();
    }
    int r = batch_kernel_setup(c);
    if (!r) r = dev_reserve(c->b_costs, sizeof(int64_t) * (size_t)count);
    if (!r && !c->bstream) {
        CUDA_TRY(cudaStreamCreateWithFlags(&c->bstream, cudaStreamNonBlocking));
        for (cudaEvent_t &e : c->bev) CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    if (r) return r;
    const bool whole = tables_out != nullptr;
    std::vector<int32_t> ids((size_t)count);
    for (int32_t i = 0; i < count; i++) ids[(size_t)i] = i;
    BatchOrder ord = batch_order(c, inst, ids, whole, 0);
    int32_t cut = batch_cut(ord);
    BatchPack pk[BATCH_LANES];
    BatchArgs a[BATCH_LANES];
    int lanes = 1;
    auto check = [&](int32_t i) { return check_arrays(i); };
    // A batch whose memory cannot be had in two parts with room to spare is solved
    // as one, in buffers of its size, at last with the arc slices of a few CTAs or one.
    bool spare = true;
    for (int32_t blocks = 0;;) {
        lanes = cut < count ? 2 : 1;
        CUDA_TRY(cudaEventRecord(c->bev[0], st));  // the second lane starts behind the caller's work too
        int status = EMV_OK;
        bool failed = false;
        for (int l = 0; l < lanes && !status && !failed; l++) {
            cudaStream_t ls = l ? c->bstream : st;
            pk[l].lane = l;
            status = batch_layout(c, inst, ord, l ? cut : 0, l ? count : cut, whole, blocks, pk[l]);
            if (!status) status = batch_fill(c, inst, pk[l], check);
            for (const BatchInst &d : pk[l].desc) failed |= bad[(size_t)d.orig] != 0;
            if (status || failed) break;
            if (l) CUDA_TRY(cudaStreamWaitEvent(ls, c->bev[0], 0));
            status = batch_upload(c, pk[l], spare, ls);
            if (status) break;
            a[l] = batch_args(c, pk[l]);
            if (l == 0) CUDA_TRY(cudaEventRecord(c->ev[0], st));
            // The control reset and the persistent launch are replayed as one CUDA graph.
            status = batch_graph_launch(c, l, a[l], pk[l].blocks, ls);
            if (!status && l) {
                CUDA_TRY(cudaEventRecord(c->bev[1], ls));
                CUDA_TRY(cudaStreamWaitEvent(st, c->bev[1], 0));
            }
        }
        if (!status && !failed) break;
        if (failed && lanes == 2 && pk[1].desc.empty())  // the second part was not looked at yet
            host_parallel_for(count - cut, [&](int64_t j) { check_arrays(ord.ids[(size_t)(cut + j)]); });
        CUDA_TRY(cudaStreamSynchronize(c->bstream));
        CUDA_TRY(cudaStreamSynchronize(st));
        if (failed) return first_bad();
        if (status != EMV_ERR_OOM || blocks == 1) return status;
        for (int l = 0; l < BATCH_LANES; l++) {
            BatchLane &L = c->blane[l];
            for (DevBuf *b : {&L.row, &L.adj, &L.term, &L.desc, &L.table, &L.arcs}) dev_release(*b);
            pk[l] = BatchPack();
        }
        if (!spare) {
            blocks = blocks == 0 ? BATCH_FEW_BLOCKS : 1;
            ord = batch_order(c, inst, ids, whole, blocks);
        }
        spare = false;
        cut = count;
    }
    CUDA_TRY(cudaEventRecord(c->ev[1], st));
    CUDA_TRY(cudaMemcpyAsync(costs_out, c->b_costs.ptr, sizeof(int64_t) * (size_t)count, cudaMemcpyDeviceToHost, st));
    uint32_t err[BATCH_LANES] = {};
    for (int l = 0; l < lanes; l++)
        CUDA_TRY(cudaMemcpyAsync(&err[l], a[l].ctl, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    if (err[0] | err[1]) return emv_dev_status_to_emv(err[0] | err[1]);
    if (tables_out) {
        for (int l = 0; l < lanes; l++) {
            k_close_rows<<<(unsigned)pk[l].count, RES_THREADS, 0, st>>>(a[l].inst);
            CUDA_TRY(cudaGetLastError());
            for (const BatchInst &d : pk[l].desc)
                if (tables_out[d.orig])
                    CUDA_TRY(cudaMemcpyAsync(tables_out[d.orig], d.table, sizeof(int32_t) * ((size_t)d.n << d.kt),
                                             cudaMemcpyDeviceToHost, st));
        }
        CUDA_TRY(cudaStreamSynchronize(st));
    }
    if (stats) {
        float ms = 0;
        cudaEventElapsedTime(&ms, c->ev[0], c->ev[1]);
        stats->total_ms = ms;
        stats->upload_ms = (float)std::chrono::duration<double, std::milli>(pk[lanes - 1].t_upload_end - t0).count();
        stats->work_items = count;
        stats->table_bytes = (pk[0].table_words + pk[1].table_words) * 4;
        stats->merge_tile = 32;
        stats->relax_rows = std::max(pk[0].rcap_used, pk[1].rcap_used);
    }
    return EMV_OK;
}

extern "C" int emv_batch_solve(emv_ctx *c, const emv_instance *inst, int32_t count, int64_t *costs_out,
                               emv_batch_stats *stats, void *stream)
{
    return batch_solve(c, inst, count, costs_out, nullptr, stats, stream);
}

extern "C" int emv_batch_solve_tables(emv_ctx *c, const emv_instance *inst, int32_t count, int64_t *costs_out,
                                      int32_t *const *tables_out, emv_batch_stats *stats, void *stream)
{
    if (!tables_out) return emv_fail(EMV_ERR_BAD_INPUT, "emv_batch_solve_tables: null table list");
    return batch_solve(c, inst, count, costs_out, tables_out, stats, stream);
}

// ---------------------------------------------------------------- packing

BatchOrder batch_order(const emv_ctx *c, const emv_instance *inst, const std::vector<int32_t> &ids, bool whole,
                       int32_t blocks)
{
    const int32_t count = (int32_t)ids.size();
    std::vector<double> work((size_t)count);
    std::vector<int64_t> states((size_t)count);
    for (int32_t j = 0; j < count; j++) {
        const emv_instance &I = inst[ids[(size_t)j]];
        const int32_t kt = whole ? I.k : table_terminals(I.k);
        work[(size_t)j] = batch_work(I.g.n, kt, I.g.arcs, 1, kt);
        states[(size_t)j] = resident_max_rows(kt) * I.g.n;
    }
    std::vector<int32_t> order, size((size_t)count, 1);
    if (blocks > 0) {
        order.resize((size_t)count);
        for (int32_t j = 0; j < count; j++) order[(size_t)j] = j;
    } else {
        batch_plan(work, states, c->batch_blocks, 1 << (BATCH_SIZES - 1), order, size);
    }
    BatchOrder o;
    for (int32_t j : order) {
        o.ids.push_back(ids[(size_t)j]);
        o.size.push_back(size[(size_t)j]);
        o.work.push_back(work[(size_t)j]);
    }
    return o;
}

int batch_layout(emv_ctx *c, const emv_instance *inst, const BatchOrder &ord, int32_t from, int32_t to, bool whole,
                 int32_t blocks, BatchPack &pk)
{
    const int32_t count = to - from;
    BatchLane &L = c->blane[pk.lane];
    pk.desc.resize((size_t)count);
    pk.row_off.resize((size_t)count);
    pk.arc_off.resize((size_t)count);
    pk.term_off.resize((size_t)count);
    pk.table_off.resize((size_t)count);
    int64_t rows = 0, arcs = 0, terms = 0, words = 0, ctas = 0;
    for (int32_t j = 0; j < count; j++) {
        const int32_t id = ord.ids[(size_t)(from + j)];
        const emv_instance &I = inst[id];
        BatchInst &d = pk.desc[(size_t)j];
        std::memset(&d, 0, sizeof(d));
        d.n = I.g.n;
        d.k = I.k;
        d.kt = whole ? I.k : table_terminals(I.k);
        d.size = ord.size[(size_t)(from + j)];
        batch_shape(c, I.g.arcs, d);
        d.orig = id;
        d.lo = 1;
        d.hi = d.kt;
        for (int32_t cl = 0; cl < BATCH_SIZES; cl++)
            if (d.size >= 1 << (BATCH_SIZES - 1 - cl)) pk.end[cl] = j + 1;
        pk.row_off[(size_t)j] = rows;
        pk.arc_off[(size_t)j] = arcs;
        pk.term_off[(size_t)j] = terms;
        pk.table_off[(size_t)j] = words;
        rows += I.g.n + 1;
        arcs += I.g.arcs;
        terms += I.k;
        words += (int64_t)batch_ld(I.g.n) << d.kt;
        ctas += d.size;
        pk.rcap_used = std::max(pk.rcap_used, d.rows);
        pk.cost_slots = std::max<int64_t>(pk.cost_slots, (int64_t)d.orig + 1);
    }
    pk.blocks = batch_blocks(c, ctas, blocks);
    pk.rows = rows;
    pk.arcs = arcs;
    pk.terms = terms;
    pk.table_words = words;
    pk.count = count;
    // Host staging (pinned, reused): adj | row_ptr | terms | desc
    const size_t bytes = sizeof(int32_t) * (size_t)rows + sizeof(int2) * (size_t)arcs + sizeof(int32_t) * (size_t)terms +
                         sizeof(BatchInst) * (size_t)count + 64;
    if (L.stage_bytes < bytes) {
        if (L.stage) cudaFreeHost(L.stage);
        L.stage = nullptr;
        L.stage_bytes = 0;
        const size_t want = bytes + bytes / 4;  // the next batch of this kind is a little larger or smaller
        if (cudaMallocHost(&L.stage, want) != cudaSuccess) {
            cudaGetLastError();
            return emv_fail(EMV_ERR_OOM, "pinned staging of %zu bytes", want);
        }
        L.stage_bytes = want;
    }
    pk.h_adj = (int2 *)L.stage;
    pk.h_row = (int32_t *)(pk.h_adj + arcs);
    pk.h_term = pk.h_row + rows;
    pk.h_desc = (BatchInst *)(((uintptr_t)(pk.h_term + terms) + 15) & ~(uintptr_t)15);
    return EMV_OK;
}

int batch_fill(emv_ctx *c, const emv_instance *inst, BatchPack &pk, const std::function<bool(int32_t)> &check)
{
    (void)c;
    std::vector<int64_t> arc_bytes((size_t)pk.count);
    host_parallel_for(pk.count, [&](int64_t j) {  // disjoint ranges of the staging buffer
        const int32_t id = pk.desc[(size_t)j].orig;
        if (check && !check(id)) return;
        const emv_instance &I = inst[id];
        const uint32_t most = pack_arcs(I.g, pk.h_adj + pk.arc_off[(size_t)j]);
        const BatchGraph bg = batch_graph(I.g.row_ptr, I.g.n, most, pk.desc[(size_t)j].hub_min);
        pk.desc[(size_t)j].narrow = bg.narrow;
        arc_bytes[(size_t)j] = bg.arc_bytes;
        std::memcpy(pk.h_row + pk.row_off[(size_t)j], I.g.row_ptr, sizeof(int32_t) * ((size_t)I.g.n + 1));
        std::memcpy(pk.h_term + pk.term_off[(size_t)j], I.terminals, sizeof(int32_t) * (size_t)I.k);
    });
    for (int64_t b : arc_bytes) pk.arc_bytes = std::max(pk.arc_bytes, b);
    return EMV_OK;
}

// dev_reserve with a quarter to spare when a buffer grows (exactly what is
// needed where that does not fit): batches of one kind differ a little in
// size, and a larger one would free and allocate gigabytes again.
static int reserve_more(DevBuf &b, size_t bytes)
{
    if (b.bytes >= bytes) return EMV_OK;
    return dev_reserve(b, bytes + bytes / 4) == EMV_OK ? (int)EMV_OK : dev_reserve(b, bytes);
}

int batch_upload(emv_ctx *c, BatchPack &pk, bool spare, cudaStream_t st)
{
    BatchLane &L = c->blane[pk.lane];
    auto reserve = spare ? reserve_more : dev_reserve;
    int r = reserve(L.row, sizeof(int32_t) * (size_t)pk.rows);
    if (!r) r = reserve(L.adj, sizeof(int2) * (size_t)std::max<int64_t>(pk.arcs, 1));
    if (!r) r = reserve(L.term, sizeof(int32_t) * (size_t)std::max<int64_t>(pk.terms, 1));
    if (!r) r = reserve(L.desc, sizeof(BatchInst) * (size_t)pk.count);
    if (!r) r = reserve(L.table, sizeof(int32_t) * (size_t)pk.table_words);
    // costs are written at index orig (the caller's instance index), which can
    // exceed the number of instances in this launch when it is a part or a sample
    if (!r) r = dev_reserve(c->b_costs, sizeof(int64_t) * (size_t)std::max<int64_t>(pk.cost_slots, 1));
    if (!r) r = dev_reserve(L.ctrl, sizeof(uint32_t) * 32 * (size_t)batch_ctl_lines(c->batch_blocks));
    if (!r) r = reserve(L.arcs, (size_t)batch_arc_stride(pk.arc_bytes) * (size_t)pk.blocks);
    if (!r) r = prepare_batch_subsets(c, st);
    if (r) return r;
    for (int32_t j = 0; j < pk.count; j++) {
        BatchInst &d = pk.desc[(size_t)j];
        if (d.orig < 0 || d.orig >= pk.cost_slots) return emv_fail(EMV_ERR_INTERNAL, "batch: cost slot out of range");
        d.row_ptr = (const int32_t *)L.row.ptr + pk.row_off[(size_t)j];
        d.adj = (const int2 *)L.adj.ptr + pk.arc_off[(size_t)j];
        d.terms = (const int32_t *)L.term.ptr + pk.term_off[(size_t)j];
        d.table = (int32_t *)L.table.ptr + pk.table_off[(size_t)j];
        pk.h_desc[j] = d;
    }
    CUDA_TRY(cudaMemcpyAsync(L.row.ptr, pk.h_row, sizeof(int32_t) * (size_t)pk.rows, cudaMemcpyHostToDevice, st));
    if (pk.arcs > 0)
        CUDA_TRY(cudaMemcpyAsync(L.adj.ptr, pk.h_adj, sizeof(int2) * (size_t)pk.arcs, cudaMemcpyHostToDevice, st));
    CUDA_TRY(cudaMemcpyAsync(L.term.ptr, pk.h_term, sizeof(int32_t) * (size_t)pk.terms, cudaMemcpyHostToDevice, st));
    CUDA_TRY(cudaMemcpyAsync(L.desc.ptr, pk.h_desc, sizeof(BatchInst) * (size_t)pk.count, cudaMemcpyHostToDevice, st));
    pk.t_upload_end = std::chrono::steady_clock::now();
    return EMV_OK;
}

// With one element a lane to spare: a closure that keeps arcs in registers loads
// the first element of its slice also where the slice has none (its vertices have
// no arcs), and a last slice's would lie behind the others.
int64_t batch_arc_stride(int64_t arc_bytes)
{
    return (arc_bytes + 32 * (int64_t)sizeof(int4) + 255) / 256 * 256;
}

BatchArgs batch_args(emv_ctx *c, const BatchPack &pk)
{
    BatchArgs a;
    std::memset(&a, 0, sizeof(a));
    const BatchLane &L = c->blane[pk.lane];
    a.inst = (const BatchInst *)L.desc.ptr;
    a.xs = (const uint32_t *)c->bxs.ptr;
    a.xs_off = (const int32_t *)c->bxs_off.ptr;
    a.costs = (int64_t *)c->b_costs.ptr;
    a.ctl = (uint32_t *)L.ctrl.ptr;
    a.scratch = (char *)L.arcs.ptr;
    a.scratch_stride = batch_arc_stride(pk.arc_bytes);
    a.smem = RESIDENT_SMEM;
    std::copy(pk.end, pk.end + BATCH_SIZES, a.end);
    return a;
}

// Launches {control reset, persistent kernel} as one graph, captured once per
// lane and kind of launch.  The arguments of another batch (its classes, its
// CTAs) go into the kernel's node: a capture and its instantiation for each took
// as long as the solve of a few small instances.
int batch_graph_launch(emv_ctx *c, int32_t lane, const BatchArgs &a, int32_t blocks, cudaStream_t st)
{
    int r = batch_kernel_setup(c);
    if (r) return r;
    BatchGraphExec &G = c->blane[lane].graph[batch_teams(a)];
    if (!G.exec || G.ctl != a.ctl) {
        batch_graph_release(G);
        cudaStream_t cap;
        CUDA_TRY(cudaStreamCreateWithFlags(&cap, cudaStreamNonBlocking));
        cudaError_t e = cudaStreamBeginCapture(cap, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            r = launch_batch(c, a, blocks, batch_ctl_lines(c->batch_blocks), cap);  // lines of any batch
            e = cudaStreamEndCapture(cap, &G.graph);
        }
        cudaStreamDestroy(cap);
        size_t count = 8;
        cudaGraphNode_t nodes[8];
        if (!r && e == cudaSuccess) e = cudaGraphGetNodes(G.graph, nodes, &count);
        for (size_t i = 0; !r && e == cudaSuccess && i < count; i++) {
            cudaGraphNodeType type;
            e = cudaGraphNodeGetType(nodes[i], &type);
            if (e == cudaSuccess && type == cudaGraphNodeTypeKernel) G.node = nodes[i];
        }
        if (!r && e == cudaSuccess) e = cudaGraphInstantiate(&G.exec, G.graph, 0);
        if (r || e != cudaSuccess || !G.node) {
            cudaGetLastError();
            batch_graph_release(G);
            return r ? r : emv_fail(EMV_ERR_CUDA, "batch graph: %s", cudaGetErrorString(e));
        }
        G.ctl = a.ctl;
    } else {
        BatchArgs args = a;
        void *p[] = {&args};
        cudaKernelNodeParams kp = {};
        kp.func = (void *)k_batch;
        kp.gridDim = dim3((unsigned)blocks);
        kp.blockDim = dim3(RES_THREADS);
        kp.sharedMemBytes = RESIDENT_SMEM;
        kp.kernelParams = p;
        CUDA_TRY(cudaGraphExecKernelNodeSetParams(G.exec, G.node, &kp));
    }
    CUDA_TRY(cudaGraphLaunch(G.exec, st));
    return EMV_OK;
}

void batch_graph_release(BatchGraphExec &G)
{
    if (G.exec) cudaGraphExecDestroy(G.exec);
    if (G.graph) cudaGraphDestroy(G.graph);
    G = BatchGraphExec();
}

// --------------------------------------------------------------- autotuner

namespace {

// Device time of one batched launch over the sample `ids` with the current
// tuning, at about four sample instances per block, as in a full batch where
// every block solves many: the time then follows a block's throughput, not
// the single slowest instance.  Best of three.
int time_sample(emv_ctx *c, const emv_instance *inst, const std::vector<int32_t> &ids, cudaStream_t st, float &ms)
{
    BatchPack pk;
    const int32_t blocks = std::max<int32_t>(1, ((int32_t)ids.size() + 3) / 4);
    int r = batch_kernel_setup(c);
    if (!r) {
        const BatchOrder ord = batch_order(c, inst, ids, false, blocks);
        r = batch_layout(c, inst, ord, 0, (int32_t)ids.size(), false, blocks, pk);
    }
    if (!r) r = batch_fill(c, inst, pk, nullptr);
    if (!r) r = batch_upload(c, pk, true, st);
    if (r) return r;
    BatchArgs a = batch_args(c, pk);
    ms = 1e30f;
    for (int rep = 0; rep < 3; rep++) {
        CUDA_TRY(cudaEventRecord(c->ev[0], st));
        r = launch_batch(c, a, pk.blocks, batch_ctl_lines(pk.blocks), st);
        if (r) return r;
        CUDA_TRY(cudaEventRecord(c->ev[1], st));
        CUDA_TRY(cudaStreamSynchronize(st));
        float t = 0;
        cudaEventElapsedTime(&t, c->ev[0], c->ev[1]);
        ms = std::min(ms, t);
    }
    return EMV_OK;
}

}  // namespace

// For every instance class present in `inst`, times the relaxation's
// rows-per-chunk candidates on a sample of that class and keeps the fastest,
// then, with it, the merge's vertex-block widths (32, 64, 128 or 256
// vertices; candidates whose staged rows do not fit are skipped) and keeps
// the fastest (in the context, and in out_rcap / out_mw[class] when given).
static int batch_autotune(emv_ctx *c, const emv_instance *inst, int32_t count, int32_t *out_rcap, int32_t *out_mw,
                   cudaStream_t st)
{
    std::vector<std::vector<int32_t>> by_class(BATCH_CLASSES);
    for (int32_t i = 0; i < count; i++) {
        if (!batch_fits(inst[i].g.n, inst[i].k)) continue;
        const int32_t cls = batch_class_of(inst[i].g.n, inst[i].k);
        if (by_class[(size_t)cls].size() < 64) by_class[(size_t)cls].push_back(i);
    }
    for (int32_t cls = 0; cls < BATCH_CLASSES; cls++) {
        auto &ids = by_class[(size_t)cls];
        if (ids.empty()) continue;
        int32_t nmax = 0, kmin = BATCH_KMAX;
        for (int32_t i : ids) {
            nmax = std::max(nmax, inst[i].g.n);
            kmin = std::min(kmin, inst[i].k);
        }
        c->tune_mw[cls] = 1;
        float best_ms = 1e30f;
        int32_t best = 0;
        for (int32_t cand : {4, 8, 16, 32, 64, 128}) {
            c->tune_rcap[cls] = cand;
            float ms = 0;
            const int r = time_sample(c, inst, ids, st, ms);
            if (r) return r;
            if (ms < best_ms) {
                best_ms = ms;
                best = cand;
            }
        }
        c->tune_rcap[cls] = best;
        int32_t best_mw = 1;
        for (int32_t mw = 2; mw <= BATCH_MW_MAX && 16 * mw < nmax && resident_merge_width(nmax, table_terminals(kmin), 1, 32 * mw) > 16 * mw; mw *= 2) {
            c->tune_mw[cls] = mw;
            float ms = 0;
            const int r = time_sample(c, inst, ids, st, ms);
            if (r) return r;
            if (ms < best_ms) {
                best_ms = ms;
                best_mw = mw;
            }
        }
        c->tune_mw[cls] = best_mw;
    }
    if (out_rcap)
        for (int32_t cls = 0; cls < BATCH_CLASSES; cls++) out_rcap[cls] = c->tune_rcap[cls];
    if (out_mw)
        for (int32_t cls = 0; cls < BATCH_CLASSES; cls++) out_mw[cls] = c->tune_mw[cls];
    return EMV_OK;
}

extern "C" int emv_batch_autotune(emv_ctx *c, const emv_instance *inst, int32_t count, int32_t *out_rcap,
                                  void *stream)
{
    if (!c || (count > 0 && !inst)) return emv_fail(EMV_ERR_BAD_INPUT, "emv_batch_autotune: bad arguments");
    CUDA_TRY(cudaSetDevice(c->device));
    return batch_autotune(c, inst, count, out_rcap, nullptr, (cudaStream_t)stream);
}

extern "C" int emv_batch_autotune2(emv_ctx *c, const emv_instance *inst, int32_t count, int32_t *out_rcap,
                                   int32_t *out_mw, void *stream)
{
    if (!c || (count > 0 && !inst)) return emv_fail(EMV_ERR_BAD_INPUT, "emv_batch_autotune2: bad arguments");
    CUDA_TRY(cudaSetDevice(c->device));
    return batch_autotune(c, inst, count, out_rcap, out_mw, (cudaStream_t)stream);
}

extern "C" int emv_batch_set_tuning2(emv_ctx *c, const int32_t *rcap, const int32_t *mw, int32_t classes)
{
    if (!c || !rcap || !mw || classes != BATCH_CLASSES)
        return emv_fail(EMV_ERR_BAD_INPUT, "emv_batch_set_tuning2: bad arguments");
    for (int32_t i = 0; i < classes; i++)
        if (rcap[i] < 0 || mw[i] < 0) return emv_fail(EMV_ERR_BAD_INPUT, "emv_batch_set_tuning2: negative entry");
    for (int32_t i = 0; i < classes; i++) {
        c->tune_rcap[i] = rcap[i];
        c->tune_mw[i] = mw[i];
    }
    return EMV_OK;
}

extern "C" int emv_batch_set_tuning(emv_ctx *c, const int32_t *rcap, int32_t classes)
{
    if (!c || !rcap || classes != BATCH_CLASSES) return emv_fail(EMV_ERR_BAD_INPUT, "emv_batch_set_tuning: bad arguments");
    for (int32_t i = 0; i < classes; i++) c->tune_rcap[i] = rcap[i];
    return EMV_OK;
}
