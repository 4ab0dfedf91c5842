// emv_kernels.cuh -- sm_103a kernels of the EMV dynamic program.
//
// Table: int32 d[X * ld + v], subset-major like the reference's FV_INDEX
// (reader/reader-el.c:691), EMV_INF32 = 2^30 for "no value".  All finite
// values are below 2^30 (checked before the DP runs), so a + b of two table values
// fits in uint32 and a value + an arc weight fits in int32.
//
// Kernels (reference step each one replaces):
//   k_fill        f_v = INF                          R:2243-2259
//   k_pack_scan   (col, w) arcs packed as int2        R:794-826 (adjacency fill)
//                 and the device CSR checked
//   k_merge, k_merge_smem, k_merge_stream, k_merge_stream16, k_merge_block
//                 subset merge of one level           R:2068-2107
//   k_relax<VEC, U16>  multi-source closure of <= 32*VEC rows (64*VEC with
//                 16-bit records; VEC = 1, 2, 4, 5, 8) R:2109-2130, R:1762-1880
//   k_narrow<LPV>  closures of at most 32 rows: the    R:1988-2031, R:2109-2130,
//                  k level-1 SSSPs, -dijkstra, ...     R:2454-2484
//   k_traceback   tree recovery by recomputation      R:1907-1944
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <type_traits>

#include "emv_common.cuh"
#include "emv_device_util.cuh"
#include "emv_narrow.cuh"
#include "emv_plan.h"

namespace emv {

struct RelaxArgs {
    const int32_t *row_ptr;
    const int2 *adj;
    int32_t n;
    int64_t ld;
    int32_t *table;
    const uint32_t *rows;   // subsets of this chunk
    int32_t nrows;          // <= 32 * VEC of the launch
    int32_t *scratch;       // vertex-major records, n * 32 * VEC int32
    uint8_t *act0;          // active flags, n bytes each
    uint8_t *act1;
    uint32_t *ctrl;         // C_WORDS words
    DevStat *stat;
    int32_t max_sweeps;
    int2 *mark;             // n: last sweep in which the vertex changed (-1 none), lowest excess of its record
    int32_t *high;          // n: highest excess of its record
    int32_t dense_min;      // a sweep after one with more changed vertices takes every vertex
    const int32_t *hubs;    // HUBS: the nhubs vertices of more than hub_min arcs
    int32_t nhubs;
    int32_t hub_min;
    uint16_t *shadow;       // if set: phase C also writes min(value, 0xffff) to shadow[X * shadow_ld + v]
    int64_t shadow_ld;
};

__global__ void k_fill(int32_t *__restrict__ p, int64_t count, int32_t value)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (; i < count; i += stride) p[i] = value;
}

// Packs the (col, w) arcs as int2 and checks the device CSR on the way (the
// admission check of the device entry points; the reference reads only
// well-formed STP, R:473-618): heads in [0, n), weights in [0, 2^30), row_ptr
// from 0 to arcs and non-decreasing.  Reduces the largest weight and the
// weight sum for the value bound, and lists the vertices of more than hub_min
// arcs (in no particular order).  *scan must be zero before the launch.
__global__ void k_pack_scan(const int32_t *__restrict__ row_ptr, int32_t n, const int32_t *__restrict__ col,
                            const int32_t *__restrict__ w, int2 *__restrict__ adj, int64_t arcs,
                            GraphScan *__restrict__ scan, int32_t hub_min, int32_t *__restrict__ hubs)
{
    scan_csr(row_ptr, n, col, w, adj, arcs, scan);
    for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x)
        if ((int64_t)row_ptr[v + 1] - row_ptr[v] > hub_min) hubs[atomicAdd(&scan->hubs, 1u)] = v;
}

// Subset merge of one level m (R:2068-2088) plus the terminal override of
// the virtual-source arcs (R:2099-2107).  Block (vertex block of 32, group
// of subsets); a warp takes one subset X at a time and its lanes 32 vertices.
// The unordered pairs {Y, X\Y} are enumerated once each (Y holds the lowest
// terminal of X); min is order-independent, so the values equal the
// reference's ordered-pair loop.  Lower-level rows are read-only here.
__global__ void __launch_bounds__(256) k_merge(int32_t *__restrict__ table, int64_t ld, int32_t n,
                                               const uint32_t *__restrict__ xs, int32_t cnt, int32_t xper,
                                               const int32_t *__restrict__ terms, int32_t k)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int32_t v = blockIdx.x * 32 + lane;
    const int32_t xb = blockIdx.y * xper, xe = min(cnt, xb + xper);
    if (v >= n) return;
    for (int32_t xi = xb + warp; xi < xe; xi += nw) {
        const uint32_t X = __ldg(xs + xi);
        const uint32_t low = X & (0u - X), rest = X ^ low;
        uint32_t acc = (uint32_t)INF;
        uint32_t s = 0;
        do {
            const uint32_t Y = low | s, Z = X ^ Y;
            const uint32_t a = (uint32_t)__ldg(table + (int64_t)Y * ld + v);
            const uint32_t b = (uint32_t)__ldg(table + (int64_t)Z * ld + v);
            acc = min(acc, a + b);
            s = (s - rest) & rest;
        } while (s != rest);
        for (uint32_t bits = X; bits; bits &= bits - 1) {
            const int t = __ffs(bits) - 1;
            if (__ldg(terms + t) == v) acc = (uint32_t)__ldg(table + (int64_t)(X ^ (1u << t)) * ld + v);
        }
        table[(int64_t)X * ld + v] = (int32_t)acc;
    }
}

// Shared-memory subset merge of one level m (R:2068-2107).  Block = VB
// consecutive vertices; it stages every row of size 1..m-1 for them once
// (S[slot][VB], slot = position in level order), then computes all C(k,m)
// rows of the level: a warp takes one subset X at a time, lane = (slice,
// vertex) with 32/VB slices splitting X's pair list, combined by shuffles.
// pairs[x * npairs + p] packs the staged slots of Y and X\Y of the p-th
// unordered pair {Y, X\Y} of the x-th subset (Y holds the lowest terminal of
// X); ovr[x * m + i] packs (terminal index << 16 | slot of X\{t}) for the
// override of the virtual-source arcs (R:2099-2107).
template <int VB>
__global__ void __launch_bounds__(1024) k_merge_smem(int32_t *__restrict__ table, int64_t ld, int32_t n,
                                                     const uint32_t *__restrict__ xs_level, int32_t cnt,
                                                     const uint32_t *__restrict__ stage_rows, int32_t nstage,
                                                     const uint32_t *__restrict__ pairs, int32_t npairs,
                                                     const uint32_t *__restrict__ ovr, int32_t m,
                                                     const int32_t *__restrict__ terms)
{
    extern __shared__ int32_t S[];
    __shared__ uint32_t red[32 * 32];  // per-subset partial minima when warps share a subset
    constexpr int G = 32 / VB;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int32_t v0 = blockIdx.x * VB;
    for (int32_t idx = threadIdx.x; idx < nstage * VB; idx += blockDim.x) {
        const int32_t i = idx / VB, j = idx - i * VB;
        const int32_t v = v0 + j;
        S[idx] = (v < n) ? __ldg(table + (int64_t)__ldg(stage_rows + i) * ld + v) : INF;
    }
    // Few subsets (the top levels): split each subset's pairs over `parts` warps.
    const int parts = cnt >= nw ? 1 : nw / cnt;
    if (parts > 1)
        for (int i = threadIdx.x; i < cnt * VB; i += blockDim.x) red[i] = (uint32_t)INF;
    __syncthreads();
    const int slice = lane / VB, j = lane % VB;
    const int32_t v = v0 + j;
    const int32_t tasks = cnt * parts;
    for (int32_t t = warp; t < tasks; t += nw) {
        const int32_t xi = t / parts, part = t - xi * parts;
        const uint32_t *P = pairs + (int64_t)xi * npairs;
        const int32_t step = G * parts;
        uint32_t acc = (uint32_t)INF, acc2 = (uint32_t)INF;
        int32_t p = part * G + slice;
        for (; p + step < npairs; p += 2 * step) {
            const uint32_t q0 = __ldg(P + p), q1 = __ldg(P + p + step);
            acc = min(acc, (uint32_t)S[(q0 & 0xffffu) * VB + j] + (uint32_t)S[(q0 >> 16) * VB + j]);
            acc2 = min(acc2, (uint32_t)S[(q1 & 0xffffu) * VB + j] + (uint32_t)S[(q1 >> 16) * VB + j]);
        }
        if (p < npairs) {
            const uint32_t q0 = __ldg(P + p);
            acc = min(acc, (uint32_t)S[(q0 & 0xffffu) * VB + j] + (uint32_t)S[(q0 >> 16) * VB + j]);
        }
        acc = min(acc, acc2);
#pragma unroll
        for (int off = 16; off >= VB; off >>= 1) acc = min(acc, __shfl_xor_sync(FULL, acc, off));
        if (parts > 1) {
            if (slice == 0) atomicMin(&red[xi * VB + j], acc);
            continue;
        }
        if (slice == 0 && v < n) {
            const uint32_t *O = ovr + (int64_t)xi * m;
            for (int i = 0; i < m; i++) {
                const uint32_t o = __ldg(O + i);
                if (__ldg(terms + (o >> 16)) == v) acc = (uint32_t)S[(o & 0xffffu) * VB + j];
            }
            table[(int64_t)__ldg(xs_level + xi) * ld + v] = (int32_t)acc;
        }
    }
    if (parts > 1) {
        __syncthreads();
        for (int32_t xi = warp; xi < cnt; xi += nw) {
            if (slice != 0 || v >= n) continue;
            uint32_t acc = red[xi * VB + j];
            const uint32_t *O = ovr + (int64_t)xi * m;
            for (int i = 0; i < m; i++) {
                const uint32_t o = __ldg(O + i);
                if (__ldg(terms + (o >> 16)) == v) acc = (uint32_t)S[(o & 0xffffu) * VB + j];
            }
            table[(int64_t)__ldg(xs_level + xi) * ld + v] = (int32_t)acc;
        }
    }
}

// One phase of the streamed merge: a set of staged rows (of sizes j and m-j)
// and, for every subset X of the launch's group, the pairs {Y, X\Y} whose
// halves are both staged, as staged positions (posY | posZ << 16) padded with
// (pad, pad) to whole quads (pad = nrows, a staged row of INF).  X's quads are
// pairs[4 * qoff[x] .. 4 * qoff[x + 1]).
struct MergePhase {
    const uint32_t *rows;   // staged subsets
    const uint32_t *pairs;  // 16-byte aligned
    const uint32_t *qoff;   // cnt + 1 quad offsets
    int32_t nrows;
    int32_t pad_;
};

// Streamed subset merge of level m (R:2068-2107).  Block = 32 consecutive
// vertices; the minima of a group of the level's subsets (all C(k,m) when
// they fit) live in shared memory (acc) while the phases stage only rows of
// sizes j and m-j (all of them, or tiles of them for large k).
// The pair loop runs on quarter-warps: the 8 lanes of a quarter hold 4
// vertices each, so one 16-byte shared load per lane brings a whole staged
// row (128 bytes, one conflict-free wavefront per quarter) and one decoded
// pair serves 32 vertices; the four quarters of a warp take four different
// subsets.  Subsets with few pairs (the top levels) split their list over
// several quarters; partial minima meet in acc through shared-memory
// atomicMin.  The terminal override of the virtual-source arcs
// (R:2099-2107) is applied last, from the finished level m-1 rows.

__device__ __forceinline__ void merge_pair4(uint4 &a, const uint4 *__restrict__ S4, uint32_t pr)
{
    const uint4 y = S4[(pr & 0xffffu) * 8];
    const uint4 z = S4[(pr >> 16) * 8];
    a.x = min(a.x, y.x + z.x);
    a.y = min(a.y, y.y + z.y);
    a.z = min(a.z, y.z + z.z);
    a.w = min(a.w, y.w + z.w);
}

__global__ void __launch_bounds__(1024) k_merge_stream(int32_t *__restrict__ table, int64_t ld, int32_t n,
                                                       const uint32_t *__restrict__ xs_level, int32_t cnt,
                                                       const MergePhase *__restrict__ phases, int32_t nphase,
                                                       const int32_t *__restrict__ terms, int32_t k,
                                                       uint32_t *__restrict__ level_max)
{
    extern __shared__ __align__(16) uint32_t sm[];
    uint32_t *acc = sm;
    uint32_t *S = sm + (size_t)cnt * 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int nq = nw * 4, qid = warp * 4 + (lane >> 3), ql = lane & 7;
    const int32_t v0 = blockIdx.x * 32, v = v0 + lane;
    __shared__ uint32_t s_max;
    if (threadIdx.x == 0) s_max = 0;
    for (int32_t i = threadIdx.x; i < cnt * 32; i += blockDim.x) acc[i] = (uint32_t)INF;
    const int parts = cnt >= nq ? 1 : nq / cnt;
    const uint4 *S4 = reinterpret_cast<const uint4 *>(S) + ql;  // staged row r, this lane's 4 vertices: S4[r * 8]
    const uint4 inf4 = make_uint4((uint32_t)INF, (uint32_t)INF, (uint32_t)INF, (uint32_t)INF);
    for (int32_t ph = 0; ph < nphase; ph++) {
        const MergePhase P = phases[ph];
        __syncthreads();
        if (v0 + 32 <= n) {
            // staging of a full vertex block: 4-byte asynchronous copies, so a
            // warp has all its rows in flight at once (row ids 32 at a time)
            for (int32_t c0 = warp * 32; c0 < P.nrows; c0 += nw * 32) {
                const uint32_t myr = c0 + lane < P.nrows ? __ldg(P.rows + c0 + lane) : 0u;
                const int32_t nr = min(32, P.nrows - c0);
                for (int32_t j = 0; j < nr; j++) {
                    const uint32_t r = __shfl_sync(FULL, myr, j);
                    cp_async4(S + (c0 + j) * 32 + lane, table + (int64_t)r * ld + v);
                }
            }
            if (warp == nw - 1) S[P.nrows * 32 + lane] = (uint32_t)INF;
            cp_async_wait_all();
        } else {
            for (int32_t i = warp; i <= P.nrows; i += nw)
                S[i * 32 + lane] = (i < P.nrows && v < n)
                                       ? (uint32_t)__ldg(table + (int64_t)__ldg(P.rows + i) * ld + v)
                                       : (uint32_t)INF;
        }
        __syncthreads();
        for (int32_t t = qid; t < cnt * parts; t += nq) {
            const int32_t xi = t / parts, part = t - xi * parts;
            const uint32_t qb = __ldg(P.qoff + xi);
            const int32_t quads = (int32_t)(__ldg(P.qoff + xi + 1) - qb);
            const uint4 *Q = reinterpret_cast<const uint4 *>(P.pairs) + qb;
            uint4 a0 = inf4, a1 = inf4;
            int32_t qi = part;
            // two quads of pairs in flight ahead of the one being reduced
            const uint4 zq = make_uint4(0, 0, 0, 0);
            uint4 q = qi < quads ? __ldg(Q + qi) : zq;
            uint4 q1 = qi + parts < quads ? __ldg(Q + qi + parts) : zq;
            while (qi < quads) {
                const int32_t q2i = qi + 2 * parts;
                const uint4 q2 = q2i < quads ? __ldg(Q + q2i) : zq;
                merge_pair4(a0, S4, q.x);
                merge_pair4(a1, S4, q.y);
                merge_pair4(a0, S4, q.z);
                merge_pair4(a1, S4, q.w);
                q = q1;
                q1 = q2;
                qi += parts;
            }
            uint32_t *A = acc + xi * 32 + ql * 4;
            const uint4 r = make_uint4(min(a0.x, a1.x), min(a0.y, a1.y), min(a0.z, a1.z), min(a0.w, a1.w));
            if (parts == 1) {
                uint4 *A4 = reinterpret_cast<uint4 *>(A);
                const uint4 o = *A4;
                *A4 = make_uint4(min(o.x, r.x), min(o.y, r.y), min(o.z, r.z), min(o.w, r.w));
            } else {
                atomicMin(A + 0, r.x);
                atomicMin(A + 1, r.y);
                atomicMin(A + 2, r.z);
                atomicMin(A + 3, r.w);
            }
        }
    }
    __syncthreads();
    bool has_term = false;
    for (int t = 0; t < k; t++) {
        const int32_t tv = __ldg(terms + t);
        has_term |= (tv >= v0 && tv < v0 + 32);
    }
    uint32_t vmax = 0;  // largest value written: the relaxation's record width follows it
    if (v < n)
        for (int32_t xi = warp; xi < cnt; xi += nw) {
            const uint32_t X = __ldg(xs_level + xi);
            uint32_t a = acc[xi * 32 + lane];
            if (has_term)
                for (uint32_t bits = X; bits; bits &= bits - 1) {
                    const int t = __ffs(bits) - 1;
                    if (__ldg(terms + t) == v) a = (uint32_t)table[(int64_t)(X ^ (1u << t)) * ld + v];
                }
            table[(int64_t)X * ld + v] = (int32_t)a;
            vmax = max(vmax, a);
        }
    vmax = __reduce_max_sync(FULL, vmax);
    if (lane == 0) atomicMax(&s_max, vmax);
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(level_max, s_max);
}

// 16-bit streamed merge: the same plan and phases as k_merge_stream, for a
// level whose sums of two staged values are all at most 65533 (the host
// checks the level maxima).  A block takes 64 vertices; a staged row holds
// them as 32 words of two 16-bit values (the same 128 bytes per row), so one
// 16-byte shared load brings 8 vertices and one min(y + z, a) per halfword
// (__viaddmin_u16x2) serves two.  The pad row is all ones: a pad pair sums to
// at least 0xfffe, above every real candidate.  Rows are staged through
// registers (int2 loads, packed to 16 bits), so the table stride and base
// must be even.  Minima live in acc as 16-bit pairs, or as one uint32 per
// vertex where quarters split a subset's pairs (shared-memory atomicMin).
__device__ __forceinline__ void merge_pair8(uint4 &a, const uint4 *__restrict__ S4, uint32_t pr)
{
    const uint4 y = S4[(pr & 0xffffu) * 8];
    const uint4 z = S4[(pr >> 16) * 8];
    a.x = addmin16(y.x, z.x, a.x);
    a.y = addmin16(y.y, z.y, a.y);
    a.z = addmin16(y.z, z.z, a.z);
    a.w = addmin16(y.w, z.w, a.w);
}

__device__ __forceinline__ uint32_t pack16(int2 x)
{
    return min((uint32_t)x.x, 0xffffu) | min((uint32_t)x.y, 0xffffu) << 16;
}

__global__ void __launch_bounds__(1024) k_merge_stream16(int32_t *__restrict__ table, int64_t ld, int32_t n,
                                                         const uint32_t *__restrict__ xs_level, int32_t cnt,
                                                         const MergePhase *__restrict__ phases, int32_t nphase,
                                                         const int32_t *__restrict__ terms, int32_t k,
                                                         uint32_t *__restrict__ level_max,
                                                         const uint16_t *__restrict__ shadow, int64_t sld)
{
    extern __shared__ __align__(16) uint32_t sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int nq = nw * 4, qid = warp * 4 + (lane >> 3), ql = lane & 7;
    const int parts = cnt >= nq ? 1 : nq / cnt;
    const int acc_words = parts > 1 ? 64 : 32;  // per subset
    uint32_t *acc = sm;
    uint32_t *S = sm + (size_t)cnt * acc_words;
    const int32_t v0 = blockIdx.x * 64, va = v0 + 2 * lane;  // this lane's vertices in staging and epilogue
    const bool full = v0 + 64 <= n;
    __shared__ uint32_t s_max;
    if (threadIdx.x == 0) s_max = 0;
    for (int32_t i = threadIdx.x; i < cnt * acc_words; i += blockDim.x) acc[i] = 0xffffffffu;
    const uint4 *S4 = reinterpret_cast<const uint4 *>(S) + ql;  // staged row r, this lane's 8 vertices: S4[r * 8]
    const uint4 ones4 = make_uint4(0xffffffffu, 0xffffffffu, 0xffffffffu, 0xffffffffu);
    for (int32_t ph = 0; ph < nphase; ph++) {
        const MergePhase P = phases[ph];
        __syncthreads();
        if (shadow) {
            // 16-bit shadow rows (stride sld, a multiple of 64 vertices): eight
            // lanes copy a staged row with 16-byte cp.async, all of a warp's
            // rows in flight; vertices past n are read but never stored
            const int sub = lane >> 3, sl = lane & 7;
            for (int32_t c0 = warp * 32; c0 < P.nrows; c0 += nw * 32) {
                const uint32_t myr = c0 + lane < P.nrows ? __ldg(P.rows + c0 + lane) : 0u;
                const int32_t nr = min(32, P.nrows - c0);
                for (int32_t j0 = 0; j0 < nr; j0 += 4) {
                    const int32_t j = j0 + sub;
                    const uint32_t r = __shfl_sync(FULL, myr, j & 31);
                    if (j < nr) cp_async16(S + (c0 + j) * 32 + sl * 4, shadow + (int64_t)r * sld + v0 + sl * 8);
                }
            }
            cp_async_wait_all();
        } else
        // staging through registers: a warp takes 32 rows at a time, 16 row
        // loads in flight per lane (8: 1.4 % slower merge; 32 spills)
        for (int32_t c0 = warp * 32; c0 < P.nrows; c0 += nw * 32) {
            const uint32_t myr = c0 + lane < P.nrows ? __ldg(P.rows + c0 + lane) : 0u;
            const int32_t nr = min(32, P.nrows - c0);
            for (int32_t j0 = 0; j0 < nr; j0 += 16) {
                int2 x[16];
#pragma unroll
                for (int u = 0; u < 16; u++) {
                    const uint32_t r = __shfl_sync(FULL, myr, j0 + u);
                    const int32_t *row = table + (int64_t)r * ld;
                    x[u] = make_int2(-1, -1);
                    if (j0 + u < nr) {
                        if (full) x[u] = __ldg(reinterpret_cast<const int2 *>(row + v0) + lane);
                        else if (va < n) x[u] = make_int2(__ldg(row + va), va + 1 < n ? __ldg(row + va + 1) : -1);
                    }
                }
#pragma unroll
                for (int u = 0; u < 16; u++)
                    if (j0 + u < nr) S[(c0 + j0 + u) * 32 + lane] = pack16(x[u]);
            }
        }
        if (warp == nw - 1) S[P.nrows * 32 + lane] = 0xffffffffu;
        __syncthreads();
        for (int32_t t = qid; t < cnt * parts; t += nq) {
            const int32_t xi = t / parts, part = t - xi * parts;
            const uint32_t qb = __ldg(P.qoff + xi);
            const int32_t quads = (int32_t)(__ldg(P.qoff + xi + 1) - qb);
            const uint4 *Q = reinterpret_cast<const uint4 *>(P.pairs) + qb;
            uint4 a0 = ones4, a1 = ones4;
            int32_t qi = part;
            const uint4 zq = make_uint4(0, 0, 0, 0);
            uint4 q = qi < quads ? __ldg(Q + qi) : zq;
            uint4 q1 = qi + parts < quads ? __ldg(Q + qi + parts) : zq;
            while (qi < quads) {
                const int32_t q2i = qi + 2 * parts;
                const uint4 q2 = q2i < quads ? __ldg(Q + q2i) : zq;
                merge_pair8(a0, S4, q.x);
                merge_pair8(a1, S4, q.y);
                merge_pair8(a0, S4, q.z);
                merge_pair8(a1, S4, q.w);
                q = q1;
                q1 = q2;
                qi += parts;
            }
            const uint4 r = make_uint4(__vminu2(a0.x, a1.x), __vminu2(a0.y, a1.y), __vminu2(a0.z, a1.z),
                                       __vminu2(a0.w, a1.w));
            if (parts == 1) {
                uint4 *A4 = reinterpret_cast<uint4 *>(acc + xi * 32 + ql * 4);
                const uint4 o = *A4;
                *A4 = make_uint4(__vminu2(o.x, r.x), __vminu2(o.y, r.y), __vminu2(o.z, r.z), __vminu2(o.w, r.w));
            } else {
                uint32_t *A = acc + xi * 64 + ql * 8;
                const uint32_t w[4] = {r.x, r.y, r.z, r.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    atomicMin(A + 2 * i, w[i] & 0xffffu);
                    atomicMin(A + 2 * i + 1, w[i] >> 16);
                }
            }
        }
    }
    __syncthreads();
    bool has_term = false;
    for (int t = 0; t < k; t++) {
        const int32_t tv = __ldg(terms + t);
        has_term |= (tv >= v0 && tv < v0 + 64);
    }
    uint32_t vmax = 0;  // largest value written: the relaxation's record width follows it
    if (va < n)
        for (int32_t xi = warp; xi < cnt; xi += nw) {
            const uint32_t X = __ldg(xs_level + xi);
            uint32_t a0, a1;
            if (parts > 1) {
                a0 = acc[xi * 64 + 2 * lane];
                a1 = acc[xi * 64 + 2 * lane + 1];
            } else {
                const uint32_t wd = acc[xi * 32 + lane];
                a0 = wd & 0xffffu;
                a1 = wd >> 16;
            }
            if (has_term)
                for (uint32_t bits = X; bits; bits &= bits - 1) {
                    const int t = __ffs(bits) - 1;
                    const int32_t tv = __ldg(terms + t);
                    if (tv == va) a0 = (uint32_t)table[(int64_t)(X ^ (1u << t)) * ld + va];
                    if (tv == va + 1) a1 = (uint32_t)table[(int64_t)(X ^ (1u << t)) * ld + va + 1];
                }
            int32_t *dst = table + (int64_t)X * ld + va;
            if (va + 1 < n) {
                *reinterpret_cast<int2 *>(dst) = make_int2((int32_t)a0, (int32_t)a1);
                vmax = max(vmax, max(a0, a1));
            } else {
                *dst = (int32_t)a0;
                vmax = max(vmax, a0);
            }
        }
    vmax = __reduce_max_sync(FULL, vmax);
    if (lane == 0) atomicMax(&s_max, vmax);
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(level_max, s_max);
}

// ---------------------------------------------------------- block merge
//
// Merge of a level whose phases' rows and minima fit shared memory (k <= 12).
// The streamed merge reads two staged rows for every pair: it is bound by
// shared-memory wavefronts, 2 a pair and 64 vertices.  Here the terminals are
// split, X = (Xh, Xl) with B low bits, and a warp reduces all subsets of one Xh
// together: for a split Yh, Xh \ Yh of the high bits it loads the rows of every
// Yl of a bits and every Zl of c bits once (C(B, a) + C(B, c) rows) and forms
// the C(B, a) * C(B - a, c) pairs of disjoint ones in registers, 0.84 loads a
// pair at k = 12, B = 5 (1.1 with B = 4: 4.75 against 4.11 ms at n = 10^5, k =
// 12; 3 % less at k = 8).  A row is a word a lane: 64 vertices of 16-bit values, or 32
// vertices.  Merge of k_merge_stream16 -> here: n = 10^5, k = 12 6.0 -> 3.9 ms,
// n = 2^17, k = 11 3.4 -> 2.1, n = 2^20, k = 10 13.1 -> 6.7 (and 32-bit values, n
// = 30 000, k = 10: 0.85 -> 0.52).  Bound: instruction issue (55 to 60 % of the
// peak) and, in the levels of few subsets, the latency of the staged rows.
// Units are dealt out to the warps by cost on the host; where the
// memory allows a minimum per vertex and subset, a unit's words lie with
// several warps (shared-memory atomicMin), else a unit belongs to one.
struct BlockPhase {
    const uint32_t *warps, *units, *words;  // HostBlockPhase
    int32_t y0, ny, z0, nz;
};

// The i-th number of a bits, and the number of smaller ones with as many bits.
__host__ __device__ constexpr int bits_nth(int a, int i)
{
    for (int s = 0;; s++) {
        int c = 0;
        for (int b = s; b; b &= b - 1) c++;
        if (c == a && i-- == 0) return s;
    }
}
__host__ __device__ constexpr int bits_rank(int x)
{
    int a = 0, r = 0;
    for (int b = x; b; b &= b - 1) a++;
    for (int s = 0; s < x; s++) {
        int c = 0;
        for (int b = s; b; b &= b - 1) c++;
        r += c == a;
    }
    return r;
}
__host__ __device__ constexpr int choose(int n, int r)
{
    int x = 1;
    for (int i = 0; i < r; i++) x = x * (n - i) / (i + 1);
    return x;
}
template <int N, int I = 0, typename F> __device__ __forceinline__ void static_for(F f)
{
    if constexpr (I < N) {
        f(std::integral_constant<int, I>{});
        static_for<N, I + 1>(f);
    }
}

template <bool U16> __device__ __forceinline__ uint32_t block_addmin(uint32_t y, uint32_t z, uint32_t acc)
{
    return U16 ? addmin16(y, z, acc) : __viaddmin_u32(y, z, acc);
}

// The pairs of all Yl of A bits with all Zl of C bits; Y, Z: this lane's word of the first rows.
template <int B, int A, int C, bool U16>
__device__ __forceinline__ void block_pairs(uint32_t (&acc)[choose(B, A + C)], const uint32_t *Y, const uint32_t *Z)
{
    uint32_t y[choose(B, A)], z[choose(B, C)];
#pragma unroll
    for (int i = 0; i < choose(B, A); i++) y[i] = Y[32 * i];
#pragma unroll
    for (int i = 0; i < choose(B, C); i++) z[i] = Z[32 * i];
    static_for<choose(B, A)>([&](auto i) {
        static_for<choose(B, C)>([&](auto j) {
            constexpr int a = bits_nth(A, i.value), c = bits_nth(C, j.value);
            if constexpr ((a & c) == 0) {
                constexpr int o = bits_rank(a | c);
                acc[o] = block_addmin<U16>(y[i.value], z[j.value], acc[o]);
            }
        });
    });
}

// One unit of subsets with Q low bits: S, M: this lane's word of the first
// staged row and of the unit's first minimum.
template <int B, int Q, bool U16>
__device__ __forceinline__ void block_unit(const uint32_t *S, uint32_t *M, bool split, const uint4 &h, uint32_t n45,
                                           const uint32_t *__restrict__ words)
{
    const int lane = threadIdx.x & 31;
    uint32_t acc[choose(B, Q)];
#pragma unroll
    for (int o = 0; o < choose(B, Q); o++) acc[o] = U16 ? 0xffffffffu : (uint32_t)INF;
    // a lane holds every 32nd word (the plan's are followed by 32 that are not used)
    const uint32_t *w = words + h.y + lane;
    uint32_t mine = __ldg(w);
    int32_t d = 0;
    static_for<Q + 1>([&](auto a) {
        constexpr int A = a.value;
        const uint32_t n2 = A < 2 ? h.z : A < 4 ? h.w : n45;
        for (int32_t left = (int32_t)(A % 2 ? n2 >> 16 : n2 & 0xffffu); left > 0; left--) {
            const uint32_t x = __shfl_sync(FULL, mine, d & 31);
            block_pairs<B, A, Q - A, U16>(acc, S + (x & 0xffffu) * 32, S + (x >> 16) * 32);
            if ((++d & 31) == 0) mine = __ldg(w += 32);
        }
    });
#pragma unroll
    for (int o = 0; o < choose(B, Q); o++) {
        if (!U16) atomicMin(M + 32 * o, acc[o]);
        else if (split) {  // vertices 2 * lane and 2 * lane + 1: words lane and 32 + lane
            atomicMin(M + 64 * o, acc[o] & 0xffffu);
            atomicMin(M + 64 * o + 32, acc[o] >> 16);
        } else M[32 * o] = __vminu2(M[32 * o], acc[o]);
    }
}

// Merge of a level of cnt subsets xs[x0..] (R:2068-2107); U16: see
// k_merge_stream16 for the values' bounds and the shadow.  A persistent block
// goes through vertex blocks and phases; the rest of the shared memory is a
// ring of `ring` staged rows, and the rows of the next steps are copied, as far
// as they fit, while this one is reduced.  (A block per vertex block, whose
// phases, a size each, wait for their copies: n = 2^20, k = 10 11.3 ms, 9.1 so.)
template <bool U16>
__global__ void __launch_bounds__(32 * BLOCK_WARPS, 1)
    k_merge_block(int32_t *__restrict__ table, int64_t ld, int32_t n, const uint32_t *__restrict__ xs, int32_t x0,
                  int32_t cnt, const BlockPhase *__restrict__ phases, int32_t nphase, bool split, int32_t ring,
                  const int32_t *__restrict__ terms, int32_t k, uint32_t *__restrict__ level_max,
                  const uint16_t *__restrict__ shadow, int64_t sld)
{
    extern __shared__ __align__(16) uint32_t sm[];
    constexpr int NV = U16 ? 64 : 32, NW = BLOCK_WARPS, B = BLOCK_LOW;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int acc_words = U16 && split ? 64 : 32;  // per subset
    const uint32_t none = U16 ? 0xffffffffu : (uint32_t)INF;
    uint32_t *S0 = sm + (size_t)cnt * acc_words;
    const int32_t nblocks = (n + NV - 1) / NV;
    __shared__ uint32_t s_max;
    if (threadIdx.x == 0) s_max = 0;
    for (int32_t i = threadIdx.x; i < cnt * acc_words; i += 32 * NW) sm[i] = none;
    // copies the rows of a phase and vertex block to S (asynchronously, but for 16-bit values without a shadow)
    auto stage = [&](int32_t vb, const BlockPhase &P, uint32_t *S) {
        const int32_t v0 = vb * NV, va = v0 + (U16 ? 2 * lane : lane), nrows = P.ny + P.nz;
        for (int32_t c0 = warp * 32; c0 < nrows; c0 += NW * 32) {
            const int32_t i = c0 + lane, nr = min(32, nrows - c0);
            const uint32_t myr = i < nrows ? __ldg(xs + (i < P.ny ? P.y0 + i : P.z0 + i - P.ny)) : 0u;
            if (U16 && shadow) {
                // eight lanes copy a row, all of a warp's rows in flight;
                // vertices past n are read but never stored
                const int sub = lane >> 3, sl = lane & 7;
                for (int32_t j0 = 0; j0 < nr; j0 += 4) {
                    const int32_t j = j0 + sub;
                    const uint32_t r = __shfl_sync(FULL, myr, j & 31);
                    if (j < nr) cp_async16(S + (c0 + j) * 32 + sl * 4, shadow + (int64_t)r * sld + v0 + sl * 8);
                }
            } else if (U16) {
                for (int32_t j0 = 0; j0 < nr; j0 += 16) {
                    int2 x[16];
#pragma unroll
                    for (int u = 0; u < 16; u++) {
                        const uint32_t r = __shfl_sync(FULL, myr, (j0 + u) & 31);
                        const int32_t *row = table + (int64_t)r * ld;
                        x[u] = make_int2(-1, -1);
                        if (j0 + u < nr) {
                            if (v0 + NV <= n) x[u] = __ldg(reinterpret_cast<const int2 *>(row + v0) + lane);
                            else if (va < n) x[u] = make_int2(__ldg(row + va), va + 1 < n ? __ldg(row + va + 1) : -1);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 16; u++)
                        if (j0 + u < nr) S[(c0 + j0 + u) * 32 + lane] = pack16(x[u]);
                }
            } else {
                for (int32_t j = 0; j < nr; j++) {
                    const uint32_t r = __shfl_sync(FULL, myr, j);
                    if (va < n) cp_async4(S + (c0 + j) * 32 + lane, table + (int64_t)r * ld + va);
                    else S[(c0 + j) * 32 + lane] = (uint32_t)INF;
                }
            }
        }
        cp_async_commit();
    };
    uint32_t vmax = 0;  // largest value written: the relaxation's record width follows it
    // steps staged but not reduced yet; next step to stage; the ring's end and
    // the rows it holds (with those left out before its end)
    int32_t ahead = 0, nvb = blockIdx.x, nph = 0, end = 0, held = 0, from = 0;
    for (int32_t vb = blockIdx.x; vb < nblocks; vb += gridDim.x) {
        for (int32_t ph = 0; ph < nphase; ph++) {
            if (ahead == 0) end = held = from = 0;
            while (ahead < 4 && nvb < nblocks) {
                const int32_t need = phases[nph].ny + phases[nph].nz;
                const bool wrap = end + need > ring;
                const int32_t take = need + (wrap ? ring - end : 0);
                if (held + take > ring) break;
                if (wrap) end = 0;
                stage(nvb, phases[nph], S0 + (size_t)end * 32);
                end += need;
                held += take;
                ahead++;
                if (++nph == nphase) {
                    nph = 0;
                    nvb += gridDim.x;
                }
            }
            const int32_t here = phases[ph].ny + phases[ph].nz;
            if (from + here > ring) {
                held -= ring - from;
                from = 0;
            }
            uint32_t *S = S0 + (size_t)from * 32;
            from += here;
            held -= here;  // free after this step
            cp_async_wait_but(--ahead);
            __syncthreads();
            const uint32_t *warps = phases[ph].warps, *units = phases[ph].units, *words = phases[ph].words;
            const uint32_t u1 = __ldg(warps + warp + 1);
            for (uint32_t u = __ldg(warps + warp); u < u1; u++) {
                const uint4 h = __ldg(reinterpret_cast<const uint4 *>(units) + 2 * u);
                const uint32_t n45 = __ldg(units + 8 * u + 4);
                uint32_t *M = sm + (h.x & 0xffffu) * acc_words + lane;
                const uint32_t q = h.x >> 16;
                static_for<B + 1>([&](auto Q) {
                    if (q == Q.value) block_unit<B, Q.value, U16>(S + lane, M, split, h, n45, words);
                });
            }
            __syncthreads();
        }
        const int32_t v0 = vb * NV, va = v0 + (U16 ? 2 * lane : lane);
        bool has_term = false;
        for (int t = 0; t < k; t++) {
            const int32_t tv = __ldg(terms + t);
            has_term |= tv >= v0 && tv < v0 + NV;
        }
        for (int32_t xi = warp; xi < cnt; xi += NW) {
            const uint32_t X = __ldg(xs + x0 + xi);
            uint32_t *M = sm + xi * acc_words + lane;
            uint32_t a0 = M[0], a1 = 0;
            M[0] = none;  // for the next vertex block
            if (U16) {
                a1 = split ? M[32] : a0 >> 16;
                if (split) M[32] = none;
                a0 &= 0xffffu;
            }
            if (va >= n) continue;
            if (has_term)
                for (uint32_t bits = X; bits; bits &= bits - 1) {
                    const int t = __ffs(bits) - 1;
                    const int32_t tv = __ldg(terms + t);
                    if (tv == va) a0 = (uint32_t)table[(int64_t)(X ^ (1u << t)) * ld + va];
                    if (U16 && tv == va + 1) a1 = (uint32_t)table[(int64_t)(X ^ (1u << t)) * ld + va + 1];
                }
            int32_t *dst = table + (int64_t)X * ld + va;
            if (U16 && va + 1 < n) {
                *reinterpret_cast<int2 *>(dst) = make_int2((int32_t)a0, (int32_t)a1);
                vmax = max(vmax, max(a0, a1));
            } else {
                *dst = (int32_t)a0;
                vmax = max(vmax, a0);
            }
        }
    }
    vmax = __reduce_max_sync(FULL, vmax);
    if (lane == 0) atomicMax(&s_max, vmax);
    __syncthreads();
    if (threadIdx.x == 0) atomicMax(level_max, s_max);
}

// ------------------------------------------------------------ excesses
//
// Most arcs of a record cannot improve any of its rows: an arc (u, w) of v is
// of use only where d_X[u] + w < d_X[v] for some row X, and random weights are
// often as long as the distances' differences.  The excess of row X at a
// vertex is d_X - c_X with any constant c_X; with the lowest excess low[u] and
// the highest high[v] over the record's rows, low[u] + w >= high[v] rules the
// arc out for all of them, without its 512-byte gather.  c_X is the row's mean
// over 32 vertices spread over the graph, which brings the rows of a record
// close together.  An arc is ruled out until u changes again: high[v] only
// falls, and a change of u stamps it anew.
// Visited arcs of a closure's 13 sweeps, per arc: 13.0 -> 4.6 at n = 10^5,
// degree 20, weights to 100 (2.0 would be enough); 14.6 -> 11.9 at n = 2^17,
// degree 8, weights to 1000 (5.6).  More bounds a vertex, one for each part of
// the rows, rule out little more: 4.4 and 11.5 with 4, 4.1 and 11.0 with 16.

// Minus c_X of every row in the record's layout, as it enters the highest
// (neg) and the lowest (neg + 32 * VEC) excess.  Rows past the chunk's get
// what leaves the one as low and the other as high as can be.
template <int VEC, bool U16> __device__ __forceinline__ void relax_offsets(const RelaxArgs &a, int32_t *neg)
{
    constexpr int R = 32 * VEC, NW = RELAX_THREADS / 32;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t v = (int64_t)a.n * lane / 32;
#pragma unroll 4
    for (int r = warp; r < (U16 ? 2 * R : R); r += NW) {
        const bool real = r < a.nrows;
        const int32_t x = real ? __ldcg(a.table + (int64_t)__ldg(a.rows + r) * a.ld + v) : 0;
        const int32_t c = __reduce_add_sync(FULL, x >> 5) + (__reduce_add_sync(FULL, x & 31) >> 5);
        if (lane) continue;
        if (U16) {
            reinterpret_cast<int16_t *>(neg)[2 * (r % R) + r / R] = (int16_t)(real ? -c : -32768);
            reinterpret_cast<int16_t *>(neg + R)[2 * (r % R) + r / R] = (int16_t)(real ? -c : 32767);
        } else {
            neg[r] = real ? -c : (int32_t)0x80000000;
            neg[R + r] = real ? -c : INF - 1;
        }
    }
}

// x: highest, y: lowest excess of some words of a record.  16-bit values are
// at most 32767 here, so a difference of two fits 16 bits.
template <bool U16> __device__ __forceinline__ int2 excess_none()
{
    return U16 ? make_int2((int32_t)0x80008000, 0x7fff7fff) : make_int2((int32_t)0x80000000, 0x7fffffff);
}
template <bool U16> __device__ __forceinline__ int2 excess_word(int2 b, int32_t d, int32_t nh, int32_t nl)
{
    if (U16)
        return make_int2((int32_t)__viaddmax_s16x2((uint32_t)d, (uint32_t)nh, (uint32_t)b.x),
                         (int32_t)__viaddmin_s16x2((uint32_t)d, (uint32_t)nl, (uint32_t)b.y));
    return make_int2(__viaddmax_s32(d, nh, b.x), __viaddmin_s32(d, nl, b.y));
}
// Over the warp.
template <bool U16> __device__ __forceinline__ int2 excess_reduce(int2 b)
{
    if (U16) b = make_int2(max((int32_t)(int16_t)b.x, b.x >> 16), min((int32_t)(int16_t)b.y, b.y >> 16));
    return make_int2(__reduce_max_sync(FULL, b.x), __reduce_min_sync(FULL, b.y));
}
// Of a record held by a warp (the lanes' shares; rec_ld's layout).
template <int VEC, bool U16>
__device__ __forceinline__ int2 excess_of(typename IVec<VEC>::T x, const int32_t *neg, int lane)
{
    const int32_t *w = reinterpret_cast<const int32_t *>(&x);
    int2 b = excess_none<U16>();
    if constexpr (VEC >= 4) {
#pragma unroll
        for (int q = 0; q + 4 <= VEC; q += 4) {
            const int at = VEC == 8 ? 8 * lane + q : 4 * lane;
            const int4 h = *reinterpret_cast<const int4 *>(neg + at), l = *reinterpret_cast<const int4 *>(neg + 32 * VEC + at);
            b = excess_word<U16>(b, w[q], h.x, l.x);
            b = excess_word<U16>(b, w[q + 1], h.y, l.y);
            b = excess_word<U16>(b, w[q + 2], h.z, l.z);
            b = excess_word<U16>(b, w[q + 3], h.w, l.w);
        }
        if constexpr (VEC == 5) b = excess_word<U16>(b, w[4], neg[128 + lane], neg[160 + 128 + lane]);
    } else {
#pragma unroll
        for (int q = 0; q < VEC; q++)
            b = excess_word<U16>(b, w[q], neg[VEC * lane + q], neg[32 * VEC + VEC * lane + q]);
    }
    return excess_reduce<U16>(b);
}

constexpr int RELAX_LIST = 128;             // at most 64 new entries beside 2 * GROUP - 1 waiting ones
constexpr int32_t RELAX_SELF = -1;          // in place of a weight: the vertex's own record
// A warp's working memory in shared memory.
struct RelaxWarp {
    int4 win[32];             // the window's vertices with arcs: vertex, first arc minus start, start, highest excess
    int4 list[RELAX_LIST / 2];  // ring of records to read, two an element: an arc (head, weight), or (vertex, RELAX_SELF)
};

// A pass over the warp's vertices.  Flags (or, in a dense sweep, every vertex)
// select the vertices, stamps and excesses the arcs.  A vertex is taken when
// its flag in `flags` is set; with clear the flag is cleared first.  Returns
// whether a record changed; counts changed vertices in *s_chg.
//
// The arcs of up to 32 taken vertices are looked at one after another, 32 at a
// time whatever their vertices, two steps ahead: while the arcs of one step are
// selected, the marks of the next and the arcs after those are on their way.
// Selected arcs go to a ring, after an entry for the vertex's own record where
// they are its first, and GROUP records of the ring are always being read: the
// loads of a vertex do not wait for those of the vertex before.  (A vertex at
// a time, with the next one's arcs and marks requested early, a sweep at n =
// 10^5 was bound by its chain of dependent loads: 46 us, 2.2 us a vertex.)
template <int VEC, bool U16, bool HUBS, int GROUP>
__device__ __forceinline__ bool relax_pass(const RelaxArgs &a, int32_t vbeg, int32_t vend, int32_t s, bool dense,
                                           bool dense_next, uint8_t *flags, bool clear, uint8_t *nxt, RelaxWarp &ws,
                                           const int32_t *neg, unsigned *s_chg)
{
    using V = typename IVec<VEC>::T;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1, le = lt << 1 | 1u;
    V val[GROUP], acc = vsplat<V>(0), old = acc;
    int32_t cur = 0, done = 0, made = 0;  // vertex being reduced; entries used, entries listed
    unsigned changed = 0;
#pragma unroll
    for (int g = 0; g < GROUP; g++) val[g] = acc;
    auto finish = [&]() {
        const bool dec = U16 ? vne(acc, old) : vlt(acc, old);
        if (!__ballot_sync(FULL, dec)) return;
        if (dec) rec_st<VEC>(a.scratch, cur, lane, acc);
        const int2 b = excess_of<VEC, U16>(acc, neg, lane);
        if (lane == 0) {
            __stcg(a.mark + cur, make_int2(s, b.y));
            __stcg(a.high + cur, b.x);
        }
        changed++;
        if (!dense_next) {
            const int32_t end = __ldg(a.row_ptr + cur + 1);
            for (int32_t e = __ldg(a.row_ptr + cur) + lane; e < end; e += 32) nxt[__ldg(&a.adj[e].x)] = 1;
        }
    };
    int2 *list = reinterpret_cast<int2 *>(ws.list);
    // the GROUP entries from k (a multiple of GROUP) on
    auto fetch = [&](int32_t k) {
        const int4 *e = ws.list + (k & (RELAX_LIST - 1)) / 2;
#pragma unroll
        for (int g = 0; g < GROUP; g += 2) {
            const int4 x = e[g / 2];
            val[g] = rec_ld<VEC>(a.scratch, x.x, lane);
            val[g + 1] = rec_ld<VEC>(a.scratch, x.z, lane);
        }
    };
    auto use = [&](int32_t vertex, int32_t weight, const V &x) {
        if (weight == RELAX_SELF) {
            finish();
            cur = vertex;
            old = acc = x;
        } else {
            acc = U16 ? vaddmin16(x, weight, acc) : vmin(acc, vadd(x, weight));
        }
    };
    // uses all entries but the last GROUP to 2 * GROUP - 1, the first GROUP of which are being read
    auto drain = [&]() {
        while (made - done >= 2 * GROUP) {
            const int4 *now = ws.list + (done & (RELAX_LIST - 1)) / 2;
            const int4 *then = ws.list + ((done + GROUP) & (RELAX_LIST - 1)) / 2;
#pragma unroll
            for (int g = 0; g < GROUP; g += 2) {
                const int4 e = now[g / 2], next = then[g / 2];
                use(e.x, e.y, val[g]);
                val[g] = rec_ld<VEC>(a.scratch, next.x, lane);
                use(e.z, e.w, val[g + 1]);
                val[g + 1] = rec_ld<VEC>(a.scratch, next.z, lane);
            }
            done += GROUP;
        }
    };
    auto listed = [&](int32_t count) {
        __syncwarp();
        if (made < GROUP && made + count >= GROUP) fetch(0);
        made += count;
        drain();
        __syncwarp();
    };
    for (int32_t base = vbeg; base < vend; base += 32) {
        const int32_t v = base + lane;
        const bool mine = v < vend;
        bool f = mine && (dense || __ldcg(flags + v) != 0);
        if (!__any_sync(FULL, f)) continue;
        const int32_t rp0 = mine ? __ldg(a.row_ptr + v) : 0;
        const int32_t rp1 = mine ? __ldg(a.row_ptr + v + 1) : 0;
        const int32_t hv = mine ? __ldcg(a.high + v) : 0;
        if (HUBS) f = f && rp1 - rp0 <= a.hub_min;  // relax_hubs takes the others
        if (f && clear) flags[v] = 0;
        const int32_t deg = f ? rp1 - rp0 : 0;
        int32_t start = deg;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t t = __shfl_up_sync(FULL, start, o);
            if (lane >= o) start += t;
        }
        const int32_t total = __shfl_sync(FULL, start, 31);
        start -= deg;
        const unsigned some = __ballot_sync(FULL, deg > 0);
        if (deg > 0) ws.win[__popc(some & lt)] = make_int4(v, rp0 - start, start, hv);
        __syncwarp();
        int32_t before = -1;  // the last vertex whose arcs start before the step
        auto request = [&](int32_t p0, int32_t &rank, int2 &arc) {
            const unsigned at = (unsigned)(start - p0);
            const unsigned starts = __reduce_or_sync(FULL, deg > 0 && at < 32 ? 1u << at : 0u);
            rank = before + __popc(starts & le);
            before += __popc(starts);
            arc = p0 + lane < total ? __ldg(a.adj + ws.win[rank].y + p0 + lane) : make_int2(0, 0);
        };
        int32_t rank0 = 0, rank1 = 0, last = -1;  // last: the vertex of the last own entry
        int2 arc0, arc1 = make_int2(0, 0);
        request(0, rank0, arc0);
        int2 mark0 = __ldcg(a.mark + arc0.x);
        if (total > 32) request(32, rank1, arc1);
        for (int32_t p0 = 0; p0 < total; p0 += 32) {
            const int4 w = ws.win[rank0];
            const bool pull = p0 + lane < total && mark0.x >= s - 1 && arc0.y + mark0.y < w.w;
            const unsigned sel = __ballot_sync(FULL, pull);
            // U16: clamped weight in both halves
            const int2 entry = U16 ? make_int2(arc0.x, (int32_t)(min((uint32_t)arc0.y, 32768u) * 0x10001u)) : arc0;
            const int32_t rank = rank0;
            arc0 = arc1;
            rank0 = rank1;
            if (p0 + 32 < total) mark0 = __ldcg(a.mark + arc0.x);
            if (p0 + 64 < total) request(p0 + 64, rank1, arc1);
            if (!sel) continue;
            const unsigned first = __ballot_sync(FULL, pull && rank != last && !(sel & lt & ~0u << max(w.z - p0, 0)));
            const int32_t at = made + __popc(sel & lt) + __popc(first & le);
            if (pull) list[at & (RELAX_LIST - 1)] = entry;
            if (first >> lane & 1u) list[(at - 1) & (RELAX_LIST - 1)] = make_int2(w.x, RELAX_SELF);
            last = __shfl_sync(FULL, rank, 31 - __clz(sel));
            listed(__popc(sel) + __popc(first));
        }
        __syncwarp();
    }
    if (made) {
        // entries that change nothing (a vertex's own record again) until the last one is used
        const int32_t more = (-made & (GROUP - 1)) + 2 * GROUP;
        const int32_t any = list[(made - 1) & (RELAX_LIST - 1)].x;
        __syncwarp();
        if (lane < more) list[(made + lane) & (RELAX_LIST - 1)] = make_int2(any, RELAX_SELF);
        listed(more);
    }
    if (lane == 0 && changed) atomicAdd(s_chg, changed);
    return changed != 0;
}

// Stores a lane's share of a record into shared memory, in the record's layout.
template <int VEC> __device__ __forceinline__ void part_st(int32_t *p, int lane, typename IVec<VEC>::T x)
{
    reinterpret_cast<typename IVec<VEC>::T *>(p)[lane] = x;
}
template <> __device__ __forceinline__ void part_st<5>(int32_t *p, int lane, int5v x)
{
    reinterpret_cast<int4 *>(p)[lane] = x.a;
    p[128 + lane] = x.b;
}

// The sweep's share of the hubs (vertices of more than hub_min arcs): a block
// takes every gridDim.x-th one, its warps 32 arcs each at a time, with the
// selection of relax_pass; the partial minima meet in shared memory
// (part: 32 * VEC words a warp).  One warp walking a hub of 1000 arcs alone
// bounded a sweep (45 us at n = 30 000, power-law degrees, against 18).
template <int VEC, bool U16, int GROUP>
__device__ __noinline__ bool relax_hubs(const RelaxArgs &a, int32_t s, bool dense, bool dense_next, uint8_t *cur,
                                        uint8_t *nxt, int2 *warcs, int32_t *part, const int32_t *neg, unsigned *s_chg)
{
    __shared__ int2 s_excess[VEC];
    using V = typename IVec<VEC>::T;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1;
    bool any = false;
    for (int32_t h = blockIdx.x; h < a.nhubs; h += gridDim.x) {
        const int32_t v = __ldg(a.hubs + h);
        const bool take = dense || __ldcg(cur + v) != 0;
        const int32_t high = __ldcg(a.high + v);
        __syncthreads();  // all have read the flag; the partial minima of the hub before are used
        if (!take) continue;
        if (threadIdx.x == 0) cur[v] = 0;
        const int32_t beg = __ldg(a.row_ptr + v), end = __ldg(a.row_ptr + v + 1);
        V acc = vsplat<V>(U16 ? -1 : INF);
        for (int32_t e0 = beg + warp * 32; e0 < end; e0 += RELAX_THREADS) {
            int2 arc = make_int2(0, 0);
            bool pull = false;
            if (e0 + lane < end) {
                arc = __ldg(a.adj + e0 + lane);
                const int2 m = __ldcg(a.mark + arc.x);
                pull = m.x >= s - 1 && arc.y + m.y < high;
            }
            const unsigned sel = __ballot_sync(FULL, pull);
            const int cnt = __popc(sel);
            if (pull)
                warcs[__popc(sel & lt)] =
                    U16 ? make_int2(arc.x, (int32_t)(min((uint32_t)arc.y, 32768u) * 0x10001u)) : arc;
            __syncwarp();
            for (int i = 0; i < cnt; i += GROUP) {
                V val[GROUP];
                int32_t wt[GROUP];
#pragma unroll
                for (int g = 0; g < GROUP; g++) {
                    const bool ok = i + g < cnt;
                    const int2 aw = warcs[(i + g) & 31];
                    wt[g] = ok ? aw.y : 0;
                    val[g] = ok ? rec_ld<VEC>(a.scratch, aw.x, lane) : vsplat<V>(U16 ? -1 : INF);
                }
#pragma unroll
                for (int g = 0; g < GROUP; g++) acc = U16 ? vaddmin16(val[g], wt[g], acc) : vmin(acc, vadd(val[g], wt[g]));
            }
            __syncwarp();
        }
        part_st<VEC>(part + warp * 32 * VEC, lane, acc);
        __syncthreads();
        bool dec = false;
        if (threadIdx.x < 32 * VEC) {
            int32_t *word = a.scratch + (int64_t)v * 32 * VEC + threadIdx.x;
            const int32_t old = __ldcg(word);
            int32_t x = old;
            for (int w = 0; w < RELAX_THREADS / 32; w++) {
                const int32_t p = part[w * 32 * VEC + threadIdx.x];
                x = U16 ? (int32_t)__vminu2((uint32_t)x, (uint32_t)p) : min(x, p);
            }
            dec = x != old;
            if (dec) __stcg(word, x);
            const int2 b = excess_reduce<U16>(
                excess_word<U16>(excess_none<U16>(), x, neg[threadIdx.x], neg[32 * VEC + threadIdx.x]));
            if (lane == 0) s_excess[warp] = b;
        }
        if (__syncthreads_or(dec)) {
            any = true;
            if (threadIdx.x == 0) {
                int2 b = s_excess[0];
                for (int q = 1; q < VEC; q++) b = make_int2(max(b.x, s_excess[q].x), min(b.y, s_excess[q].y));
                __stcg(a.mark + v, make_int2(s, b.y));
                __stcg(a.high + v, b.x);
                atomicAdd(s_chg, 1u);
            }
            if (!dense_next)
                for (int32_t e = beg + threadIdx.x; e < end; e += RELAX_THREADS) nxt[__ldg(&a.adj[e].x)] = 1;
        }
    }
    return any;
}

// Frontier sweeps over one chunk (phase B of k_relax).  A warp owns a
// contiguous range of n / W vertices (W warps in the grid, so the shares
// differ by one vertex at most; half of them dealt out in windows of 4 or 8 to
// whoever is done: 6 % slower, the windows' first loads cost more than the
// wait for the last warp); for every active vertex it pulls min over its
// arcs (u, w) of rec[u] + w with coalesced 128*VEC-byte gathers -- only from
// heads stamped as changed in the previous sweep (a head that last changed
// earlier was already pulled when that change marked this vertex active), and
// of those only the arcs that the excesses leave.  Only the owner writes a
// record and values only decrease, so no atomics are needed.  Returns the
// number of sweeps, or -1 after an error (recorded).
//
// U16: 16-bit records, two rows per int32 word (64*VEC rows a record).  The
// host takes them only when every value of the chunk's rows is at most
// 32767; the arc weight is then clamped to 32768, so a value plus a weight
// stays below 2^16, and a clamped sum (at least 32768) never beats a value.
template <int VEC, bool U16, bool HUBS>
__device__ int32_t relax_sweeps(const RelaxArgs &a, int *s_ok, RelaxWarp *warps, int32_t *part, const int32_t *neg)
{
    constexpr int GROUP = VEC == 8 ? 2 : 4;  // gathers in flight
    const int32_t n = a.n;
    const int32_t gw = (int32_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int32_t nwg = (int32_t)((gridDim.x * blockDim.x) >> 5);
    const int32_t vbeg = (int32_t)((int64_t)n * gw / nwg), vend = (int32_t)((int64_t)n * (gw + 1) / nwg);
    volatile uint32_t *vctrl = a.ctrl;
    RelaxWarp &ws = warps[threadIdx.x >> 5];
    __shared__ unsigned s_chg;
    // read by thread 0 after each sweep's barrier: [0] the sweep changed a
    // record, [1] its changed count, [2] the count of the sweep before
    __shared__ uint32_t s_ctl[3];
    if (threadIdx.x == 0) {
        s_chg = 0;
        s_ctl[1] = s_ctl[2] = (uint32_t)n;
    }
    __syncthreads();
    // Dense sweeps take every vertex (a vertex with no changed neighbour then
    // selects no arc) and so need no neighbour flags from the sweep before.
    // Sweep s decides whether sweep s + 1 is dense before its own count of
    // changed vertices is known: it predicts that count from the last two
    // (their ratio continued while the counts fall) and makes sweep s + 1
    // dense when the prediction exceeds dense_min.  A wrong guess costs time
    // only: a sparse sweep's flags are written whenever the next one is sparse.
    // Changed counts live in a ring of four words (sweep s: C_CNT0 + s % 4).
    bool dense = true;  // sweep 0: every vertex is active
    int32_t s = 0;
    for (; s < a.max_sweeps; s++) {
        uint8_t *cur = (s & 1) ? a.act1 : a.act0;
        uint8_t *nxt = (s & 1) ? a.act0 : a.act1;
        const uint32_t prev_chg = s_ctl[1];   // n before sweep 0
        const uint32_t prev2_chg = s_ctl[2];  // n before sweeps 0 and 1
        const uint32_t pred_chg = prev_chg < prev2_chg
                                      ? (uint32_t)((uint64_t)prev_chg * prev_chg / prev2_chg)
                                      : prev_chg;
        const bool dense_next = pred_chg > (uint32_t)a.dense_min;
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            vctrl[C_SLOT0 + (s + 1) % 3] = 0;
            vctrl[C_CNT0 + (s + 1) % 4] = 0;
        }
        bool any = relax_pass<VEC, U16, HUBS, GROUP>(a, vbeg, vend, s, dense, dense_next, cur, true, nxt, ws, neg, &s_chg);
        // A sparse sweep whose successor is sparse also takes, once, the vertices
        // already marked for the next sweep (by changes earlier in this sweep; a
        // block's warps wait for each other, so that all of its own are), so a
        // change travels two arcs per sweep in the frontier's tail.  Their marks
        // stay: the next sweep takes them again, after the barrier has made every
        // change of this sweep visible, so a change this early pass missed is
        // still pulled there.  (Relaxation at n = 10^5, degree 20, k = 11, and n =
        // 12 000, degree 3, k = 12: 5.95 and 4.63 ms without the pass, 6.25 and
        // 4.66 without the wait, 6.02 and 4.42 so.)
        if (!dense && !dense_next) {
            __syncthreads();
            any |= relax_pass<VEC, U16, HUBS, GROUP>(a, vbeg, vend, s, false, dense_next, nxt, false, nxt, ws, neg, &s_chg);
        }
        if (HUBS) any |= relax_hubs<VEC, U16, GROUP>(a, s, dense, dense_next, cur, nxt, reinterpret_cast<int2 *>(ws.list),
                                                    part, neg, &s_chg);
        any = __syncthreads_or(any);
        if (threadIdx.x == 0) {
            if (any) vctrl[C_SLOT0 + s % 3] = 1;
            if (s_chg) atomicAdd(a.ctrl + C_CNT0 + s % 4, s_chg);
            s_chg = 0;
        }
        const bool ok = grid_barrier(a.ctrl, s_ok, [&] {
            s_ctl[0] = vctrl[C_SLOT0 + s % 3];
            s_ctl[2] = s_ctl[1];
            s_ctl[1] = vctrl[C_CNT0 + s % 4];
        });
        if (!ok) {
            if (threadIdx.x == 0) atomicOr(&a.stat->err, a.ctrl[C_ERR]);
            return -1;
        }
        if (s_ctl[0] == 0) return s + 1;
        dense = dense_next;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&a.stat->err, (uint32_t)EMV_DEV_SWEEP_LIMIT);
    return -1;
}

// Phase A of a relaxation chunk: rows -> vertex-major records (vertex v owns
// 32*VEC int32 words, word e = row e; U16: word e = rows e | (e + 32*VEC) << 16).
// A tile is 32 vertices by all 32*VEC words, so a warp has all its row loads in
// flight before one barrier.  Rows past the chunk's are INF (U16: 0, which
// no sweep lowers).  Also sets the active flags, stamps and excesses.
template <int VEC, bool U16>
__device__ __forceinline__ int32_t relax_load_value(const RelaxArgs &a, int32_t row, int32_t v)
{
    if (row >= a.nrows || v >= a.n) return U16 ? 0 : INF;
    return __ldcg(a.table + (int64_t)__ldg(a.rows + row) * a.ld + v);
}

template <int VEC, bool U16>
__device__ void relax_load_records(const RelaxArgs &a, int32_t (*tile)[33], int32_t *neg)
{
    constexpr int R = 32 * VEC, NW = RELAX_THREADS / 32, PER = R / NW;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t n = a.n, ntiles = (n + 31) >> 5;
    // software pipeline: the next tile's row loads are in flight while this
    // tile's records are written
    int32_t x[PER], xh[U16 ? PER : 1];
    auto fetch = [&](int32_t t) {
        const int32_t v = t * 32 + lane;
#pragma unroll
        for (int q = 0; q < PER; q++) {
            x[q] = relax_load_value<VEC, U16>(a, warp + q * NW, v);
            if (U16) xh[q] = relax_load_value<VEC, U16>(a, warp + q * NW + R, v);
        }
    };
    if (blockIdx.x < ntiles) fetch(blockIdx.x);
    relax_offsets<VEC, U16>(a, neg);
    for (int32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
#pragma unroll
        for (int q = 0; q < PER; q++)
            tile[warp + q * NW][lane] =
                U16 ? (int32_t)(min((uint32_t)x[q], 0xffffu) | min((uint32_t)xh[U16 ? q : 0], 0xffffu) << 16) : x[q];
        __syncthreads();
        if (t + (int32_t)gridDim.x < ntiles) fetch(t + gridDim.x);
        for (int vv = warp; vv < 32; vv += NW) {
            const int32_t v2 = t * 32 + vv;
            if (v2 >= n) break;
            int2 b = excess_none<U16>();
#pragma unroll
            for (int g = 0; g < VEC; g++) {
                const int32_t x = tile[g * 32 + lane][vv];
                __stcg(a.scratch + (int64_t)v2 * R + g * 32 + lane, x);
                b = excess_word<U16>(b, x, neg[g * 32 + lane], neg[R + g * 32 + lane]);
            }
            b = excess_reduce<U16>(b);
            if (lane == 0) {
                __stcg(a.mark + v2, make_int2(-1, b.y));
                __stcg(a.high + v2, b.x);
            }
        }
        __syncthreads();
    }
    for (int32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
        a.act0[v] = 1;
        a.act1[v] = 0;
    }
}

// Phase C: vertex-major records -> table rows, a whole 32-vertex tile at a
// time.
template <int VEC, bool U16>
__device__ void relax_store_records(const RelaxArgs &a, int32_t (*tile)[33])
{
    constexpr int R = 32 * VEC, NW = RELAX_THREADS / 32, PER = R / NW;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t n = a.n, ntiles = (n + 31) >> 5, nrows = a.nrows;
    // software pipeline: the next tile's record loads are in flight while
    // this tile's rows are written
    constexpr int VPW = 32 / NW;  // vertices of a tile per warp
    int32_t y[VPW][VEC];
    auto fetch = [&](int32_t t) {
#pragma unroll
        for (int i = 0; i < VPW; i++) {
            const int32_t v2 = t * 32 + warp + i * NW;
#pragma unroll
            for (int g = 0; g < VEC; g++) y[i][g] = (v2 < n) ? __ldcg(a.scratch + (int64_t)v2 * R + g * 32 + lane) : INF;
        }
    };
    if (blockIdx.x < ntiles) fetch(blockIdx.x);
    for (int32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
#pragma unroll
        for (int i = 0; i < VPW; i++)
#pragma unroll
            for (int g = 0; g < VEC; g++) tile[g * 32 + lane][warp + i * NW] = y[i][g];
        __syncthreads();
        if (t + (int32_t)gridDim.x < ntiles) fetch(t + gridDim.x);
        const int32_t v = t * 32 + lane;
        if (v < n)
#pragma unroll
            for (int q = 0; q < PER; q++) {
                const int32_t row = warp + q * NW;
                const uint32_t word = (uint32_t)tile[row][lane];
                if (U16) {
                    const uint32_t lo = word & 0xffffu, hi = word >> 16;
                    const int32_t xlo = lo == 0xffffu ? INF : (int32_t)lo, xhi = hi == 0xffffu ? INF : (int32_t)hi;
                    if (row < nrows) {
                        const int64_t X = __ldg(a.rows + row);
                        a.table[X * a.ld + v] = xlo;
                        if (a.shadow) a.shadow[X * a.shadow_ld + v] = (uint16_t)lo;
                    }
                    if (row + R < nrows) {
                        const int64_t X = __ldg(a.rows + row + R);
                        a.table[X * a.ld + v] = xhi;
                        if (a.shadow) a.shadow[X * a.shadow_ld + v] = (uint16_t)hi;
                    }
                } else if (row < nrows) {
                    const int64_t X = __ldg(a.rows + row);
                    a.table[X * a.ld + v] = (int32_t)word;
                    if (a.shadow) a.shadow[X * a.shadow_ld + v] = (uint16_t)min(word, 0xffffu);
                }
            }
        __syncthreads();
    }
}

// Multi-source shortest-path closure of up to 32*VEC rows (R:2109-2130): for
// every row X of the chunk, d[X][v] = min over u of init[u] + dist(u, v).
// One cooperative persistent launch: A. rows -> vertex-major records;
// B. frontier sweeps (relax_sweeps), bounded by n + 1 (the Bellman-Ford
// bound), ending after a sweep that changes nothing; C. records -> rows.
// Records and stamps are read with ld.global.cg (L2), never through a stale
// L1 line.
template <int VEC, bool U16 = false, bool HUBS = false>
__global__ void __launch_bounds__(RELAX_THREADS, 2) k_relax(RelaxArgs a)
{
    // the transposes' tile (32 vertices by all words of the chunk's records);
    // during the sweeps the warps' working memory and the hubs' partial minima
    constexpr int TILE = 32 * VEC * 33, WARPS = RELAX_THREADS / 32 * (int)sizeof(RelaxWarp) / 4;
    constexpr int SWEEP = WARPS + (HUBS ? RELAX_THREADS / 32 * 32 * VEC : 0);
    __shared__ __align__(16) int32_t mem[TILE > SWEEP ? TILE : SWEEP];
    int32_t(*tile)[33] = reinterpret_cast<int32_t(*)[33]>(mem);
    __shared__ __align__(16) int32_t neg[2 * 32 * VEC];  // relax_offsets
    __shared__ int s_ok;
    relax_load_records<VEC, U16>(a, tile, neg);
    if (!grid_barrier(a.ctrl, &s_ok)) {
        if (threadIdx.x == 0) atomicOr(&a.stat->err, a.ctrl[C_ERR]);
        return;
    }
    const int32_t s =
        relax_sweeps<VEC, U16, HUBS>(a, &s_ok, reinterpret_cast<RelaxWarp *>(mem), mem + WARPS, neg);
    if (s < 0) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&a.stat->sweeps, (unsigned long long)s);
    relax_store_records<VEC, U16>(a, tile);
}

// Closures of up to 4 * LPV rows on narrow records: from sources (level 1,
// R:1988-2031, and the -dijkstra command), with sparse sweeps from the sources'
// neighbours on, or of merged rows (R:2109-2130).
struct NarrowLaunch {
    NarrowArgs na;
    const int2 *adj;
    const int32_t *terms;   // source of row r, or null: closures of the rows as they are
    const uint32_t *rows;   // table row of r
    int32_t nrows;          // <= 4 * LPV
    int32_t *table;
    int64_t ld;
    uint32_t *vmax;         // if set: atomicMax of every value written
    uint16_t *shadow;       // if set: min(value, 0xffff) at shadow[row * shadow_ld + v]
    int64_t shadow_ld;
    DevStat *stat;
    const GraphScan *scan;  // if set: the CSR's check; a faulty one is not read
};

template <int LPV>
__global__ void __launch_bounds__(NARROW_THREADS, 2) k_narrow(NarrowLaunch a)
{
    __shared__ int s_ok;
    if (a.scan && a.scan->bad) return;
    const int32_t n = a.na.n;
    const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    if (a.terms) {
        for (int64_t i = first; i < (int64_t)n * LPV; i += stride) __stcg(a.na.rec + i, make_int4(INF, INF, INF, INF));
    } else {
        for (int32_t g = 0; g < LPV; g++)  // four rows of a vertex a thread
            for (int64_t v = first; v < n; v += stride) {
                int32_t y[4];
#pragma unroll
                for (int q = 0; q < 4; q++)
                    y[q] = 4 * g + q < a.nrows ? __ldcg(a.table + (int64_t)__ldg(a.rows + 4 * g + q) * a.ld + v) : INF;
                __stcg(a.na.rec + v * LPV + g, make_int4(y[0], y[1], y[2], y[3]));
            }
    }
    for (int64_t v = first; v < n; v += stride) a.na.act0[v] = a.na.act1[v] = 0;
    if (!grid_barrier(a.na.ctrl, &s_ok)) {
        if (threadIdx.x == 0) atomicOr(&a.stat->err, a.na.ctrl[C_ERR]);
        return;
    }
    if (a.terms && blockIdx.x == 0)  // a warp per source: its distance, and its neighbours take part in sweep 0
        for (int32_t r = threadIdx.x >> 5; r < a.nrows; r += NARROW_THREADS / 32) {
            const int32_t t = __ldg(a.terms + r);
            if ((threadIdx.x & 31) == 0) __stcg(reinterpret_cast<int32_t *>(a.na.rec) + (int64_t)t * 4 * LPV + r, 0);
            for (int32_t e = __ldg(a.na.row_ptr + t) + (threadIdx.x & 31); e < __ldg(a.na.row_ptr + t + 1); e += 32)
                a.na.act0[__ldg(&a.adj[e].x)] = 1;
        }
    if (a.terms && !grid_barrier(a.na.ctrl, &s_ok)) {
        if (threadIdx.x == 0) atomicOr(&a.stat->err, a.na.ctrl[C_ERR]);
        return;
    }
    const int32_t s = narrow_sweeps<LPV>(a.na, NarrowPacked{a.adj}, a.terms != nullptr, &a.stat->err, &s_ok);
    if (s < 0) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(&a.stat->sweeps, (unsigned long long)s);
    uint32_t vmax = 0;
    for (int32_t g = 0; g < LPV && 4 * g < a.nrows; g++)
        for (int64_t v = first; v < n; v += stride) {
            const int4 x = __ldcg(a.na.rec + v * LPV + g);
            const int32_t y[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (4 * g + q < a.nrows) {
                    const int64_t X = __ldg(a.rows + 4 * g + q);
                    a.table[X * a.ld + v] = y[q];
                    if (a.shadow) a.shadow[X * a.shadow_ld + v] = (uint16_t)min((uint32_t)y[q], 0xffffu);
                    vmax = max(vmax, (uint32_t)y[q]);
                }
        }
    if (a.vmax) {
        vmax = __reduce_max_sync(FULL, vmax);
        if ((threadIdx.x & 31) == 0) atomicMax(a.vmax, vmax);
    }
}

// ------------------------------------------------------------- traceback

// The bits of p, lowest first, at the set positions of mask.
__device__ __forceinline__ uint32_t deposit_bits(uint32_t p, uint32_t mask)
{
    uint32_t r = 0;
    for (; p && mask; p >>= 1) {
        const uint32_t lowbit = mask & (0u - mask);
        if (p & 1u) r |= lowbit;
        mask ^= lowbit;
    }
    return r;
}

constexpr int TB_WARPS = 16;
constexpr int TB_TASKS = 64;   // pieces of the tree: at most 2 (k - 1) - 1
constexpr int TB_CHUNK = 64;   // edges of a chunk of a piece's list
constexpr int TB_HEAD = 16;    // words before the edges of the result
constexpr int32_t TB_WAIT = 1 << 22;  // polls for the search arrays while their holder makes no progress (over 0.4 s)

struct TbArgs {
    const int32_t *table;
    int64_t ld;
    int32_t n;
    int32_t k;
    const int32_t *row_ptr;
    const int2 *adj;
    const int32_t *terms;
    const uint32_t *skip_err, *skip_refused;  // if set: words that are 0 where table and arcs may be read
    int32_t *chunks;    // edge lists: chunks of TB_CHUNK edges of 3 words
    int32_t *next;      // the chunk after each chunk
    int32_t nchunks;
    int32_t *out;       // TB_HEAD words ([0] edge count, [1] status, [2, 3] ns), then the edges (3 words each)
    int32_t cap;        // edges that fit
    int32_t *queue;     // n
    int32_t *parent;    // n
    int32_t *stamp;     // n
    int32_t max_steps;
};

// Witness of d[X][v] = D (warp-collective, all lanes return the same):
// 0 leaf (X = {i}, v = t_i); 1 split d[Y][v] + d[X\Y][v] = D (the lowest
// pair index; DY = d[Y][v]); 2 arc (u, v) of positive weight with d[X][u] + w
// = D; 3 none of those (a zero-weight predecessor must exist).  [beg, end):
// v's arcs, on return of 2 (with WALK set) u's.  A step's time is its chain of dependent loads
// (arc, value at its head), so the first 32 arcs are requested before the
// pairs are looked at, and the bounds of a head's own arcs with its value.
// (Without WALK, in searches, the bounds are left out: with them cliques of 600 and
// 700 vertices and weights of 0 to 3 took 35 to 68 ms, 26 to 50 so.)
template <bool WALK>
__device__ int tb_witness(const TbArgs &a, uint32_t X, int32_t v, int32_t D, int32_t &beg, int32_t &end, uint32_t &Y,
                          int32_t &DY, int32_t &u, int32_t &wt)
{
    const int lane = threadIdx.x & 31;
    const int pc = __popc(X);
    if (pc == 1 && v == __ldg(a.terms + (__ffs(X) - 1))) return 0;
    const int32_t *row = a.table + (int64_t)X * a.ld;
    int2 arc;
    int32_t du = INF, ub = 0, ue = 0;
    auto head = [&](int32_t e) {  // arc e, its head's value and arcs
        du = INF;
        if (e < end) {
            arc = a.adj[e];
            du = row[arc.x];
            if (WALK) {
                ub = a.row_ptr[arc.x];
                ue = a.row_ptr[arc.x + 1];
            }
        }
    };
    head(beg + lane);
    if (pc >= 2) {
        const uint32_t low = X & (0u - X), rest = X ^ low;
        const uint32_t npairs = (1u << __popc(rest)) - 1;
        const uint32_t mine = deposit_bits((uint32_t)lane, rest);  // the pair index's low five bits
        uint32_t high = rest;                                      // positions of its other bits
        for (int i = 0; i < 5; i++) high &= high - 1;
        for (uint32_t base = 0; base < npairs; base += 128) {
            uint32_t y[4];
            int32_t x1[4], x2[4];
#pragma unroll
            for (int q = 0; q < 4; q++) {
                x1[q] = x2[q] = INF;
                if (base + 32 * q >= npairs) continue;
                const bool ok = base + 32 * q + lane < npairs;
                y[q] = low | (ok ? mine : 0u) | deposit_bits((base >> 5) + q, high);
                if (!ok) continue;
                x1[q] = a.table[(int64_t)y[q] * a.ld + v];
                x2[q] = a.table[(int64_t)(X ^ y[q]) * a.ld + v];
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const unsigned bal = __ballot_sync(FULL, x1[q] < INF && x2[q] < INF && x1[q] + x2[q] == D);
                if (bal) {
                    Y = __shfl_sync(FULL, y[q], __ffs(bal) - 1);
                    DY = __shfl_sync(FULL, x1[q], __ffs(bal) - 1);
                    return 1;
                }
            }
        }
    }
    for (int32_t e0 = beg;;) {
        const unsigned bal = __ballot_sync(FULL, du < INF && arc.y > 0 && du + arc.y == D);
        if (bal) {
            const int src = __ffs(bal) - 1;
            u = __shfl_sync(FULL, arc.x, src);
            wt = __shfl_sync(FULL, arc.y, src);
            if (WALK) {
                beg = __shfl_sync(FULL, ub, src);
                end = __shfl_sync(FULL, ue, src);
            }
            return 2;
        }
        e0 += 32;
        if (e0 >= end) return 3;
        head(e0 + lane);
    }
}

// A piece of the tree: the walk from (X, v) along arcs of row X to a leaf or to
// a split into kid (X \ Y) and kid + 1 (Y).
struct TbTask {
    uint32_t X;
    int32_t v, D;
    int32_t first, count;  // its edges
    int32_t kid;           // -1: a leaf
    int32_t ready;
};

// Tree recovery from the finished table (one block).  Starts at (C, q) and
// repeatedly explains d[X][v] by a leaf, a split into (Y, v) and (X\Y, v),
// or an arc (v, u) into (X, u) -- the decisions the reference records in b_v
// (R:2081-2084, R:2122-2128) and walks in backtrack() (R:1907-1932), found
// here by recomputation instead of a 2x-table predecessor store.  Every piece
// between two splits is walked by a warp of its own (one warp for the whole
// tree: 83 us at n = 4096, k = 10, a chain of 67 steps; the pieces together
// are as long as the longest way from the root), into its own edge list; the
// lists are then laid out in the order of the depth-first walk that visits
// X \ Y first.  A run of zero-weight arcs is resolved by a breadth-first
// search inside the set of vertices with the same value, so zero-weight
// cycles cannot loop; its arrays serve one warp at a time, and the others wait
// as long as that search goes on (each visits a vertex once, so it ends): it
// may take in the whole graph, a chain of dependent loads per vertex, and up to
// k - 2 pieces stand behind it.
__global__ void __launch_bounds__(32 * TB_WARPS) k_traceback(TbArgs a)
{
    __shared__ TbTask task[TB_TASKS];
    __shared__ int s_alloc, s_next, s_done, s_chunk, s_lock, s_walk, s_beat;
    __shared__ uint32_t s_status;
    __shared__ int32_t s_order[TB_TASKS], s_at[TB_TASKS], s_pieces;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if ((a.skip_err && *a.skip_err) || (a.skip_refused && *a.skip_refused)) {
        if (threadIdx.x < TB_HEAD) a.out[threadIdx.x] = 0;
        return;
    }
    unsigned long long t0 = 0;
    if (threadIdx.x == 0) {
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
        s_next = s_done = s_chunk = s_lock = s_walk = s_beat = 0;
        s_alloc = a.k >= 2;
        s_status = 0;
        if (a.k >= 2) {
            TbTask &t = task[0];
            t.X = (1u << (a.k - 1)) - 1;
            t.v = a.terms[a.k - 1];
            t.D = a.table[(int64_t)t.X * a.ld + t.v];
            t.ready = 1;
        }
        for (int i = a.k >= 2; i < TB_TASKS; i++) task[i].ready = 0;
    }
    __syncthreads();
    int32_t steps = 0;
    for (;;) {
        // claim a piece; a warp that finds none for long leaves the rest to the others
        int mine = -1;
        if (lane == 0)
            for (int spins = 0; spins < (1 << 20); spins++) {
                const int h = *(volatile int *)&s_next;
                if (h < min(*(volatile int *)&s_alloc, TB_TASKS) && *(volatile int *)&task[h].ready) {
                    if (atomicCAS(&s_next, h, h + 1) == h) {
                        mine = h;
                        break;
                    }
                } else if (*(volatile int *)&s_done >= *(volatile int *)&s_alloc || *(volatile uint32_t *)&s_status) {
                    break;
                }
            }
        mine = __shfl_sync(FULL, mine, 0);
        if (mine < 0) break;
        const uint32_t X = task[mine].X;
        int32_t v = task[mine].v, D = task[mine].D;
        int32_t beg = a.row_ptr[v], end = a.row_ptr[v + 1];
        int32_t count = 0, first = -1, chunk = -1, kid = -1;
        uint32_t fail = 0;
        auto add_edge = [&](int32_t x, int32_t y, int32_t w) {  // lane 0's arguments
            if (count % TB_CHUNK == 0) {
                int c = 0;
                if (lane == 0) c = atomicAdd(&s_chunk, 1);
                c = __shfl_sync(FULL, c, 0);
                if (c >= a.nchunks) {
                    fail = EMV_DEV_TB_OVERFLOW;
                    return;
                }
                if (lane == 0 && chunk >= 0) a.next[chunk] = c;
                if (first < 0) first = c;
                chunk = c;
            }
            if (lane == 0) {
                int32_t *e = a.chunks + ((int64_t)chunk * TB_CHUNK + count % TB_CHUNK) * 3;
                e[0] = x;
                e[1] = y;
                e[2] = w;
            }
            count++;
        };
        while (!fail) {
            if (++steps > a.max_steps) {
                fail = EMV_DEV_TB_STEPS;
                break;
            }
            uint32_t Y = 0;
            int32_t DY = 0, u = 0, wt = 0;
            const int kind = tb_witness<true>(a, X, v, D, beg, end, Y, DY, u, wt);
            if (kind == 0) break;
            if (kind == 1) {
                if (lane == 0) kid = atomicAdd(&s_alloc, 2);
                kid = __shfl_sync(FULL, kid, 0);
                if (kid + 2 > TB_TASKS) {
                    fail = EMV_DEV_TB_OVERFLOW;
                    break;
                }
                if (lane < 2) {
                    TbTask &t = task[kid + lane];
                    t.X = lane ? Y : X ^ Y;
                    t.v = v;
                    t.D = lane ? DY : D - DY;
                    __threadfence_block();
                    *(volatile int *)&t.ready = 1;
                }
                break;
            }
            if (kind == 2) {
                add_edge(v, u, wt);
                v = u;
                D -= wt;
                continue;
            }
            // Zero-weight run: BFS over arcs of weight 0 between vertices of value D.
            int walk = 0;
            if (lane == 0) {
                int beat = -1;
                for (int32_t spins = 0; spins < TB_WAIT;) {
                    if (atomicCAS(&s_lock, 0, 1) == 0) {
                        walk = ++s_walk;
                        break;
                    }
                    const int now = *(volatile int *)&s_beat;
                    spins = now == beat ? spins + 1 : 0;
                    beat = now;
                    __nanosleep(100);
                }
                if (!walk) walk = -1;
            }
            walk = __shfl_sync(FULL, walk, 0);
            if (walk < 0) {
                fail = EMV_DEV_TB_STEPS;
                break;
            }
            if (walk == 1)  // the first run of this launch clears the stamps
                for (int32_t i = lane; i < a.n; i += 32) a.stamp[i] = 0;
            __syncwarp();
            if (lane == 0) {
                a.queue[0] = v;
                a.parent[v] = -1;
                a.stamp[v] = walk;
            }
            __syncwarp();
            int32_t head = 0, tail = 1, target = -1;
            while (head < tail) {
                const int32_t x = *(volatile int32_t *)(a.queue + head);
                head++;
                if (lane == 0) ++*(volatile int *)&s_beat;
                if (x != v) {
                    uint32_t Y2;
                    int32_t d2, u2, w2, xb = a.row_ptr[x], xe = a.row_ptr[x + 1];
                    if (tb_witness<false>(a, X, x, D, xb, xe, Y2, d2, u2, w2) != 3) {
                        target = x;
                        break;
                    }
                }
                const int32_t xb = a.row_ptr[x], xe = a.row_ptr[x + 1];
                for (int32_t e0 = xb; e0 < xe; e0 += 32) {
                    const int32_t e = e0 + lane;
                    bool add = false;
                    int32_t y = 0;
                    if (e < xe) {
                        const int2 arc = a.adj[e];
                        y = arc.x;
                        if (arc.y == 0 && a.table[(int64_t)X * a.ld + y] == D) add = atomicExch(a.stamp + y, walk) != walk;
                    }
                    const unsigned bal = __ballot_sync(FULL, add);
                    if (add) {
                        const int pos = tail + __popc(bal & ((1u << lane) - 1));
                        a.queue[pos] = y;
                        a.parent[y] = x;
                    }
                    tail += __popc(bal);
                    __syncwarp();
                }
            }
            if (target < 0) fail = EMV_DEV_TB_NO_WITNESS;
            for (int32_t z = target; !fail && z != v;) {
                const int32_t p = *(volatile int32_t *)(a.parent + z);
                add_edge(z, p, 0);
                if (lane == 0) ++*(volatile int *)&s_beat;
                z = p;
            }
            if (!fail) {
                v = target;
                beg = a.row_ptr[v];
                end = a.row_ptr[v + 1];
            }
            __threadfence();
            __syncwarp();
            if (lane == 0) atomicExch(&s_lock, 0);
        }
        if (lane == 0) {
            task[mine].first = first;
            task[mine].count = count;
            task[mine].kid = kid;
            if (fail) atomicOr(&s_status, fail);
            __threadfence_block();
            atomicAdd(&s_done, 1);
        }
        __syncwarp();
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {  // the pieces in depth-first order and where their edges go
        int32_t total = 0, pieces = 0, sp = 0;
        int32_t stack[TB_TASKS];
        if (!s_status && s_done < s_alloc) s_status = EMV_DEV_TB_STEPS;
        if (!s_status && a.k >= 2) stack[sp++] = 0;
        while (sp > 0) {
            const int32_t t = stack[--sp];
            s_order[pieces] = t;
            s_at[pieces++] = total;
            total += task[t].count;
            if (task[t].kid >= 0) {
                stack[sp++] = task[t].kid + 1;
                stack[sp++] = task[t].kid;
            }
        }
        if (total > a.cap) {
            s_status |= EMV_DEV_TB_OVERFLOW;
            pieces = 0;
        }
        s_pieces = pieces;
        a.out[0] = s_status ? 0 : total;
        a.out[1] = (int32_t)s_status;
    }
    __syncthreads();
    for (int p = warp; p < s_pieces; p += TB_WARPS) {
        const TbTask &t = task[s_order[p]];
        int32_t *dst = a.out + TB_HEAD + (int64_t)s_at[p] * 3;
        for (int32_t i = 0, c = t.first; i < t.count; i += TB_CHUNK) {
            const int32_t words = min(TB_CHUNK, t.count - i) * 3;
            for (int32_t w = lane; w < words; w += 32)
                dst[(int64_t)i * 3 + w] = __ldcg(a.chunks + (int64_t)c * TB_CHUNK * 3 + w);
            c = __ldcg(a.next + c);
        }
    }
    if (threadIdx.x == 0) {
        unsigned long long t1;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t1));
        *reinterpret_cast<unsigned long long *>(a.out + 2) = t1 - t0;
    }
}

}  // namespace emv
