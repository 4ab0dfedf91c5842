// emv_noalloc.cu -- a shortest-path closure entry point that allocates no
// device memory (C ABI, include/emv.h: emv_closure_noalloc).
//
// Some callers of this library cannot allocate device memory at the time they
// call it: code that runs while another framework owns every byte of the
// device through its own pool, code that must not trigger the device-wide
// synchronisation of cudaMalloc/cudaFree in a latency-critical loop, and
// plug-ins whose host application forbids allocation after start-up.  For
// them this file keeps the closure's working memory in one file-scope device
// array of fixed size, reserved when the library is loaded on a device and
// held until the process exits, and reuses it on every call.
//
// The computation is the same multi-source closure as the relaxation kernel
// of emv_kernels.cuh (the reference's dijkstra run from a virtual source,
// reader/reader-el.c:1762-1880 and 2109-2130), in a variant that reads the
// CSR's col and w arrays as given instead of a packed copy:
//   out[r][v] = min over u of init[r][u] + dist(u, v),  r < rows <= 32.
// The kernel first checks the CSR and returns before the closure reads a
// faulty one (EMV_ERR_BAD_INPUT / EMV_ERR_OVERFLOW).  Where the largest input
// value plus the longest possible path stays below EMV_INF32 no sum can reach
// it, and the closure runs on narrow records (emv_narrow.cuh); otherwise on
// 128-byte ones, where a value plus a weight saturates at EMV_INF32 instead of
// wrapping, and a finite candidate that saturates where no smaller one exists
// is reported as EMV_ERR_OVERFLOW.
#include <algorithm>
#include <cstring>
#include <mutex>

#include "emv_device_util.cuh"
#include "emv_narrow.cuh"
#include "emv_solver.h"

using namespace emv;

namespace {

constexpr int32_t NOALLOC_MAX_N = 131072;      // vertices
constexpr int32_t NOALLOC_MAX_ROWS = 32;       // rows per call (one per lane)
constexpr size_t REC_BYTES = (size_t)NOALLOC_MAX_N * NOALLOC_MAX_ROWS * sizeof(int32_t);  // 16 MiB
constexpr size_t FLAG_BYTES = (size_t)NOALLOC_MAX_N;                                     // per flag array
constexpr size_t CTRL_OFF = REC_BYTES + 2 * FLAG_BYTES;
constexpr size_t STAT_OFF = CTRL_OFF + (sizeof(uint32_t) * C_WORDS + 255) / 256 * 256;
static_assert(CTRL_OFF % 128 == 0, "control words on their own lines");
constexpr size_t SCAN_OFF = STAT_OFF + 64;
constexpr size_t MAXV_OFF = STAT_OFF + 128;
constexpr size_t NOALLOC_BYTES = STAT_OFF + 256;
static_assert(SCAN_OFF + sizeof(GraphScan) <= MAXV_OFF, "scan words inside the status area");
constexpr int NOALLOC_THREADS = NARROW_THREADS;
constexpr int NOALLOC_VARIANTS = 4;                // kernels by record width (4, 8, 16 or 32 rows)
constexpr int MAX_DEVICES = 64;

// The scratch of every call on this device: vertex-major records, two
// active-flag arrays, the barrier words and the status words.
static __device__ __align__(256) unsigned char g_noalloc_scratch[NOALLOC_BYTES];

std::mutex g_setup_mu;
unsigned char *g_scratch_ptr[MAX_DEVICES] = {};
int g_blocks[MAX_DEVICES][NOALLOC_VARIANTS] = {};

struct NoallocArgs {
    const int32_t *row_ptr;
    const int32_t *col;
    const int32_t *w;
    const int32_t *init;
    int32_t *out;
    int64_t ld;
    int32_t n;
    int32_t rows;
    int64_t arcs;
    int32_t dense_min;
    int32_t *rec;
    uint8_t *act0;
    uint8_t *act1;
    uint32_t *ctrl;
    DevStat *stat;
    GraphScan *scan;
    uint32_t *maxv;  // largest finite input value
};

// val + wt saturated at INF (wt is in [0, INF) after the scan, val <= INF);
// *sat is set when a finite val saturated.
__device__ __forceinline__ int32_t sat_add(int32_t val, int32_t wt, bool *sat)
{
    const int32_t room = INF - wt;
    *sat |= (val < INF) & (val >= room);
    return min(val, room) + wt;
}

// Closure on 128-byte records with saturating sums: rows -> records, frontier
// sweeps, records -> rows.
__device__ void noalloc_saturating(const NoallocArgs &a, int *ok_word)
{
    __shared__ int32_t tile[32][33];
    int &s_ok = *ok_word;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwb = blockDim.x >> 5;
    const int32_t n = a.n, ntiles = (n + 31) >> 5;
    for (int32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        const int32_t v = t * 32 + lane;
        for (int r = warp; r < 32; r += nwb)
            tile[r][lane] = (r < a.rows && v < n) ? min(a.init[(int64_t)r * a.ld + v], INF) : INF;
        __syncthreads();
        for (int vv = warp; vv < 32; vv += nwb) {
            const int32_t v2 = t * 32 + vv;
            if (v2 < n) __stcg(a.rec + (int64_t)v2 * 32 + lane, tile[lane][vv]);
        }
        __syncthreads();
    }
    for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        a.act0[v] = 1;
        a.act1[v] = 0;
    }
    bool overflow = false;
    if (!grid_barrier(a.ctrl, &s_ok)) {
        if (threadIdx.x == 0) atomicOr(&a.stat->err, a.ctrl[C_ERR]);
        return;
    }
    const int32_t gw = (int32_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int32_t nwg = (int32_t)((gridDim.x * blockDim.x) >> 5);
    volatile uint32_t *vctrl = a.ctrl;
    int32_t s = 0;
    bool converged = false;
    for (; s <= n; s++) {
        uint8_t *cur = (s & 1) ? a.act1 : a.act0;
        uint8_t *nxt = (s & 1) ? a.act0 : a.act1;
        if (blockIdx.x == 0 && threadIdx.x == 0) vctrl[C_SLOT0 + (s + 1) % 3] = 0;
        bool any = false;
        for (int32_t blk = gw; blk < ntiles; blk += nwg) {
            const int32_t v = blk * 32 + lane;
            const bool f = v < n && __ldcg(cur + v) != 0;
            unsigned act = __ballot_sync(FULL, f);
            if (!act) continue;
            if (f) cur[v] = 0;
            const int32_t rp0 = v < n ? __ldg(a.row_ptr + v) : 0;
            const int32_t rp1 = v < n ? __ldg(a.row_ptr + v + 1) : 0;
            while (act) {
                const int j = __ffs(act) - 1;
                act &= act - 1;
                const int32_t vv = blk * 32 + j;
                const int32_t beg = __shfl_sync(FULL, rp0, j), end = __shfl_sync(FULL, rp1, j);
                int32_t *mine = a.rec + (int64_t)vv * 32 + lane;
                const int32_t old = __ldcg(mine);
                int32_t acc = old;
                bool sat = false;
                for (int32_t e0 = beg; e0 < end; e0 += 32) {
                    int32_t cu = 0, cw = 0;
                    if (e0 + lane < end) {
                        cu = __ldg(a.col + e0 + lane);
                        cw = __ldg(a.w + e0 + lane);
                    }
                    const int cnt = min(32, end - e0);
                    for (int g = 0; g < cnt; g += 8) {
                        int32_t val[8], wt[8];
#pragma unroll
                        for (int i = 0; i < 8; i++) {
                            const int32_t u = __shfl_sync(FULL, cu, (g + i) & 31);
                            wt[i] = __shfl_sync(FULL, cw, (g + i) & 31);
                            val[i] = (g + i < cnt) ? __ldcg(a.rec + (int64_t)u * 32 + lane) : INF;
                        }
#pragma unroll
                        for (int i = 0; i < 8; i++) acc = min(acc, sat_add(val[i], wt[i], &sat));
                    }
                }
                overflow |= sat & (acc >= INF);
                const bool dec = acc < old;
                if (dec) __stcg(mine, acc);
                if (__ballot_sync(FULL, dec)) {
                    any = true;
                    for (int32_t e = beg + lane; e < end; e += 32) nxt[__ldg(a.col + e)] = 1;
                }
            }
        }
        any = __syncthreads_or(any);
        if (any && threadIdx.x == 0) vctrl[C_SLOT0 + s % 3] = 1;
        if (!grid_barrier(a.ctrl, &s_ok)) {
            if (threadIdx.x == 0) atomicOr(&a.stat->err, a.ctrl[C_ERR]);
            return;
        }
        if (vctrl[C_SLOT0 + s % 3] == 0) {
            converged = true;
            break;
        }
    }
    if (__any_sync(FULL, overflow) && lane == 0) atomicOr(&a.stat->err, (uint32_t)EMV_DEV_OVERFLOW);
    if (!converged) {
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&a.stat->err, (uint32_t)EMV_DEV_SWEEP_LIMIT);
        return;
    }
    for (int32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
        for (int vv = warp; vv < 32; vv += nwb) {
            const int32_t v2 = t * 32 + vv;
            tile[vv][lane] = (v2 < n) ? __ldcg(a.rec + (int64_t)v2 * 32 + lane) : INF;
        }
        __syncthreads();
        const int32_t v = t * 32 + lane;
        if (v < n)
            for (int r = warp; r < a.rows; r += nwb) a.out[(int64_t)r * a.ld + v] = tile[lane][r];
        __syncthreads();
    }
}

// The whole call: CSR check and largest input value, then the closure of rows
// kept in records of 4 * LPV rows.
template <int LPV> __global__ void __launch_bounds__(NOALLOC_THREADS, 2) k_closure_noalloc(NoallocArgs a)
{
    __shared__ int s_ok;
    const int32_t n = a.n;
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    scan_csr(a.row_ptr, n, a.col, a.w, nullptr, a.arcs, a.scan);
    bool bad_value = false;
    uint32_t top = 0;
    int4 *rec = reinterpret_cast<int4 *>(a.rec);
    for (int g = 0; g < LPV; g++)  // four rows of a vertex a thread
        for (int64_t v = first; v < n; v += stride) {
            int32_t y[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                y[q] = 4 * g + q < a.rows ? a.init[(int64_t)(4 * g + q) * a.ld + v] : INF;  // d_out may be d_init
                bad_value |= y[q] > INF;
                if (y[q] < INF) top = max(top, (uint32_t)max(y[q], 0));
            }
            __stcg(rec + v * LPV + g, make_int4(y[0], y[1], y[2], y[3]));
        }
    top = __reduce_max_sync(FULL, top);
    if ((threadIdx.x & 31) == 0 && top) atomicMax(a.maxv, top);
    if (__any_sync(FULL, bad_value) && (threadIdx.x & 31) == 0) atomicOr(&a.stat->err, (uint32_t)EMV_DEV_BAD_VALUE);
    for (int64_t v = first; v < n; v += stride) a.act0[v] = a.act1[v] = 0;
    if (!grid_barrier(a.ctrl, &s_ok)) {
        if (threadIdx.x == 0) atomicOr(&a.stat->err, a.ctrl[C_ERR]);
        return;
    }
    if (__ldcg(&a.scan->bad) || __ldcg(&a.stat->err)) return;  // the host names the fault
    // a path visits a vertex, and so an arc, once
    const long long longest = min((long long)(n - 1) * (long long)__ldcg(&a.scan->maxw), (long long)__ldcg(&a.scan->sumw));
    if ((long long)__ldcg(a.maxv) + longest >= INF) {
        noalloc_saturating(a, &s_ok);
        return;
    }
    const NarrowArgs na{a.row_ptr, n, rec, a.act0, a.act1, a.ctrl, n + 1, a.dense_min};
    if (narrow_sweeps<LPV>(na, NarrowSplit{a.col, a.w}, false, &a.stat->err, &s_ok) < 0) return;
    for (int g = 0; g < LPV; g++)
        for (int64_t v = first; v < n; v += stride) {
            const int4 x = __ldcg(rec + v * LPV + g);
            const int32_t y[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (4 * g + q < a.rows) a.out[(int64_t)(4 * g + q) * a.ld + v] = y[q];
        }
}

const void *const noalloc_fns[NOALLOC_VARIANTS] = {
    (const void *)k_closure_noalloc<1>, (const void *)k_closure_noalloc<2>, (const void *)k_closure_noalloc<4>,
    (const void *)k_closure_noalloc<8>};

// Per-device set-up, done once with that device current: the device address
// of the scratch array (its host-side name is only a stand-in) and the
// cooperative grid size.  No allocation happens here either.
int setup_device(int dev)
{
    std::lock_guard<std::mutex> lk(g_setup_mu);
    if (g_scratch_ptr[dev]) return EMV_OK;
    int coop = 0;
    cudaError_t ec = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
    if (ec != cudaSuccess || !coop) {
        cudaGetLastError();
        return emv_fail(EMV_ERR_CUDA, "emv_closure_noalloc: device %d does not support cooperative launches", dev);
    }
    void *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess || !p) {
        cudaGetLastError();
        return emv_fail(EMV_ERR_CUDA, "scratch symbol address: %s", cudaGetErrorString(e));
    }
    int sms = 0;
    e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    for (int i = 0; e == cudaSuccess && i < NOALLOC_VARIANTS; i++) {
        int per_sm = 0;
        e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, noalloc_fns[i], NOALLOC_THREADS, 0);
        g_blocks[dev][i] = std::max(1, per_sm) * std::max(1, sms);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return emv_fail(EMV_ERR_CUDA, "occupancy query: %s", cudaGetErrorString(e));
    }
    g_scratch_ptr[dev] = (unsigned char *)p;
    return EMV_OK;
}

}  // namespace

extern "C" int emv_closure_noalloc(int32_t n, int64_t arcs, const int32_t *d_row_ptr, const int32_t *d_col,
                                   const int32_t *d_w, const int32_t *d_init, int32_t rows, int64_t ld,
                                   int32_t *d_out, void *stream)
{
    if (n <= 0 || arcs < 0 || arcs >= INT32_MAX || !d_row_ptr || (arcs > 0 && (!d_col || !d_w)) || !d_init ||
        !d_out || rows < 1 || ld < n)
        return emv_fail(EMV_ERR_BAD_INPUT, "emv_closure_noalloc: bad arguments");
    if (n > NOALLOC_MAX_N || rows > NOALLOC_MAX_ROWS)
        return emv_fail(EMV_ERR_BAD_INPUT,
                        "emv_closure_noalloc: n = %d, rows = %d exceed the fixed scratch (n <= %d, rows <= %d)", n,
                        rows, NOALLOC_MAX_N, NOALLOC_MAX_ROWS);
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= MAX_DEVICES) return emv_fail(EMV_ERR_BAD_INPUT, "device %d", dev);
    int r = setup_device(dev);
    if (r) return r;
    unsigned char *base = g_scratch_ptr[dev];
    cudaStream_t st = (cudaStream_t)stream;
    // The call waits on the stream (the check and the status reads), which a
    // capturing stream does not allow: refuse before touching the stream.
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    CUDA_TRY(cudaStreamIsCapturing(st, &cap));
    if (cap != cudaStreamCaptureStatusNone)
        return emv_fail(EMV_ERR_BAD_INPUT, "emv_closure_noalloc: the stream is capturing; this call cannot be captured");
    NoallocArgs a;
    a.row_ptr = d_row_ptr;
    a.col = d_col;
    a.w = d_w;
    a.init = d_init;
    a.out = d_out;
    a.ld = ld;
    a.n = n;
    a.rows = rows;
    a.arcs = arcs;
    a.dense_min = narrow_dense_min(n, arcs);
    a.scan = (GraphScan *)(base + SCAN_OFF);
    a.maxv = (uint32_t *)(base + MAXV_OFF);
    a.rec = (int32_t *)base;
    a.act0 = base + REC_BYTES;
    a.act1 = base + REC_BYTES + FLAG_BYTES;
    a.ctrl = (uint32_t *)(base + CTRL_OFF);
    a.stat = (DevStat *)(base + STAT_OFF);
    // The array keeps the last call's contents: the barrier, status and check
    // words must start at zero (records and flags are rewritten by the kernel).
    CUDA_TRY(cudaMemsetAsync(base + CTRL_OFF, 0, NOALLOC_BYTES - CTRL_OFF, st));
    const int vi = rows <= 4 ? 0 : rows <= 8 ? 1 : rows <= 16 ? 2 : 3;
    const int vpb = narrow_vertices(1 << vi) * (NOALLOC_THREADS / 32);  // one group of vertices a warp
    const int blocks = std::min(g_blocks[dev][vi], std::max(1, (n + vpb - 1) / vpb));
    void *args[] = {&a};
    CUDA_TRY(cudaLaunchCooperativeKernel(noalloc_fns[vi], dim3(blocks), dim3(NOALLOC_THREADS), args, 0, st));
    unsigned char words[MAXV_OFF - STAT_OFF];
    CUDA_TRY(cudaMemcpyAsync(words, base + STAT_OFF, sizeof(words), cudaMemcpyDeviceToHost, st));
    CUDA_TRY(cudaStreamSynchronize(st));
    DevStat ds;
    GraphScan hs;
    std::memcpy(&ds, words, sizeof(ds));
    std::memcpy(&hs, words + (SCAN_OFF - STAT_OFF), sizeof(hs));
    if (hs.bad & SCAN_BAD_ROWS) return emv_fail(EMV_ERR_BAD_INPUT, "emv_closure_noalloc: row_ptr not from 0 to arcs, non-decreasing");
    if (hs.bad & SCAN_BAD_HEAD) return emv_fail(EMV_ERR_BAD_INPUT, "emv_closure_noalloc: arc head out of range");
    if (hs.bad & SCAN_BAD_WEIGHT) return emv_fail(EMV_ERR_BAD_INPUT, "emv_closure_noalloc: negative weight");
    if (hs.bad & SCAN_BIG_WEIGHT) return emv_fail(EMV_ERR_OVERFLOW, "emv_closure_noalloc: an arc weight reaches 2^30");
    if (ds.err) return emv_dev_status_to_emv(ds.err);
    return EMV_OK;
}
