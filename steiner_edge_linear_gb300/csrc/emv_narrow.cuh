// emv_narrow.cuh -- closures of at most 32 rows on the whole GPU: the level-1
// single-source closures of the DP (reader/reader-el.c:1988-2031), the
// -dijkstra command's call and the allocation-free closure.
//
// Records hold 4 * LPV int32 rows of a vertex (16 to 128 bytes), four rows a
// lane, so a warp pulls 32 / LPV vertices at a time and has 8 gathers of each
// in flight.  One vertex a warp (a 128-byte record whatever the row count)
// left a sweep bound by the latency of about 30 vertices one after another: 17
// us at n = 2^17, degree 8, and 12 rows, 4 to 5 times the bytes' time.
// Bound now: L2 gathers in the dense sweeps, the grid barrier in the others.
#pragma once

#include <cmath>

#include "emv_common.cuh"
#include "emv_device_util.cuh"

namespace emv {

constexpr int NARROW_THREADS = 512;
constexpr int NARROW_AP1 = 4, NARROW_AP2 = 2, NARROW_AP4 = 2;
constexpr int NARROW_HUB = 64;  // a vertex of more arcs is pulled by the whole warp

// Arcs as packed pairs or as two arrays.
struct NarrowPacked {
    const int2 *adj;
    __device__ __forceinline__ int2 arc(int32_t e) const { return __ldg(adj + e); }
    __device__ __forceinline__ int32_t head(int32_t e) const { return __ldg(&adj[e].x); }
};
struct NarrowSplit {
    const int32_t *col, *w;
    __device__ __forceinline__ int2 arc(int32_t e) const { return make_int2(__ldg(col + e), __ldg(w + e)); }
    __device__ __forceinline__ int32_t head(int32_t e) const { return __ldg(col + e); }
};

struct NarrowArgs {
    const int32_t *row_ptr;
    int32_t n;
    int4 *rec;              // n * LPV
    uint8_t *act0, *act1;   // n flags each: vertices to take in the next even / odd sweep
    uint32_t *ctrl;         // C_WORDS words
    int32_t max_sweeps;
    int32_t dense_min;      // a sweep after one with more changed vertices takes every vertex
};

// Lanes that share the arcs of a vertex, for each of its LPV record lanes: a
// vertex's latency is then one gather for most degrees.
__host__ __device__ constexpr int narrow_arc_lanes(int lpv) { return lpv == 1 ? NARROW_AP1 : lpv == 2 ? NARROW_AP2 : lpv == 4 ? NARROW_AP4 : 1; }
// Vertices a warp pulls at a time.
__host__ __device__ constexpr int narrow_vertices(int lpv) { return 32 / (lpv * narrow_arc_lanes(lpv)); }

// One sweep over this warp's vertices [vbeg, vend): pulls the minimum over the
// arcs of every vertex (dense) or of the flagged ones; marks the neighbours of
// changed vertices in nxt when the next sweep is sparse.  list: this warp's 32
// bytes of shared memory.  Returns the number of changed vertices (the same in
// every lane).
template <int LPV, typename ARCS>
__device__ __forceinline__ int32_t narrow_pass(const NarrowArgs &a, const ARCS &arcs, int32_t vbeg, int32_t vend,
                                               bool dense, bool flags_next, uint8_t *cur, uint8_t *nxt,
                                               uint8_t *list)
{
    constexpr int AP = narrow_arc_lanes(LPV), GL = LPV * AP, VPW = 32 / GL;
    constexpr int U = AP == 1 ? 8 : 4;  // gathers of a lane in flight
    const int lane = threadIdx.x & 31, sub = lane % LPV, part = lane % GL / LPV, grp = lane / GL;
    const unsigned group = GL == 32 ? FULL : ((1u << GL) - 1) << (grp * GL);
    const int4 inf4 = make_int4(INF, INF, INF, INF);
    int32_t changed = 0;
    for (int32_t base = vbeg; base < vend; base += 32) {
        const int32_t mine = base + lane;
        const bool own = mine < vend, take = own && (dense || __ldcg(cur + mine) != 0);
        unsigned act = __ballot_sync(FULL, take);
        if (!act) continue;
        if (take) cur[mine] = 0;
        const int32_t rp0 = own ? __ldg(a.row_ptr + mine) : 0, rp1 = own ? __ldg(a.row_ptr + mine + 1) : 0;
        unsigned hubs = __ballot_sync(FULL, take && rp1 - rp0 > NARROW_HUB);
        act &= ~hubs;
        // stores vertex v's record where it went from old to x and marks the heads of its arcs
        auto finish = [&](int32_t v, int32_t beg, int32_t end, const int4 &old, const int4 &x, bool valid, int first,
                          int step, unsigned mask) {
            const bool dec = valid && vlt(x, old);
            if (dec) __stcg(a.rec + (int64_t)v * LPV + sub, x);
            const unsigned any = __ballot_sync(FULL, dec);
            if (flags_next && (any & mask))
                for (int32_t e = beg + first; e < end; e += step) nxt[arcs.head(e)] = 1;
            return any;
        };
        // minimum over the lanes that hold the same rows, from lane distance `from` on
        auto combine = [&](int4 x, int from, int to) {
#pragma unroll
            for (int o = from; o < to; o <<= 1) {
                x.x = min(x.x, __shfl_xor_sync(FULL, x.x, o));
                x.y = min(x.y, __shfl_xor_sync(FULL, x.y, o));
                x.z = min(x.z, __shfl_xor_sync(FULL, x.z, o));
                x.w = min(x.w, __shfl_xor_sync(FULL, x.w, o));
            }
            return x;
        };
        // VPW vertices at a time, a group of GL lanes each
        const int count = __popc(act);
        __syncwarp();
        if (act >> lane & 1u) list[__popc(act & ((1u << lane) - 1))] = (uint8_t)lane;
        __syncwarp();
        for (int i = grp; i - grp < count; i += VPW) {
            const bool valid = i < count;
            const int src = valid ? list[i] : 0;
            const int32_t beg = __shfl_sync(FULL, rp0, src), last = __shfl_sync(FULL, rp1, src);
            const int32_t end = valid ? last : beg;
            const int32_t v = base + src;
            const int4 old = valid ? __ldcg(a.rec + (int64_t)v * LPV + sub) : inf4;
            int4 x = old;
            for (int32_t e0 = beg; e0 < end; e0 += U * AP) {
                int4 val[U];
                int32_t w[U];
                if constexpr (AP == 1 && LPV == U) {  // the group's lanes load an arc each
                    const int2 arc = e0 + sub < end ? arcs.arc(e0 + sub) : make_int2(v, 0);  // itself: no gain
#pragma unroll
                    for (int q = 0; q < U; q++) {
                        const int32_t h = __shfl_sync(group, arc.x, q, LPV);
                        w[q] = __shfl_sync(group, arc.y, q, LPV);
                        val[q] = __ldcg(a.rec + (int64_t)h * LPV + sub);
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < U; q++) {
                        const int32_t e = e0 + part + q * AP;
                        const bool ok = e < end;
                        const int2 arc = ok ? arcs.arc(e) : make_int2(0, 0);
                        w[q] = arc.y;
                        val[q] = ok ? __ldcg(a.rec + (int64_t)arc.x * LPV + sub) : inf4;
                    }
                }
#pragma unroll
                for (int q = 0; q < U; q++) x = vaddmin(val[q], w[q], x);
            }
            __syncwarp();
            x = combine(x, LPV, GL);
            const unsigned any = finish(v, beg, end, old, x, valid && part == 0, lane % GL, GL, group);
            unsigned per_group = any;
#pragma unroll
            for (int o = 1; o < GL; o <<= 1) per_group |= per_group >> o;
            changed += __popc(per_group & (GL == 1   ? FULL
                                           : GL == 2 ? 0x55555555u
                                           : GL == 4 ? 0x11111111u
                                           : GL == 8 ? 0x01010101u
                                                     : 0x00010001u));
        }
        for (; hubs; hubs &= hubs - 1) {  // the groups share the arcs of a hub
            const int j = __ffs(hubs) - 1;
            const int32_t beg = __shfl_sync(FULL, rp0, j), end = __shfl_sync(FULL, rp1, j), v = base + j;
            constexpr int WAYS = 32 / LPV;
            const int4 old = __ldcg(a.rec + (int64_t)v * LPV + sub);
            int4 x = old;
            for (int32_t e0 = beg + lane / LPV; e0 < end; e0 += U * WAYS) {
                int4 val[U];
                int32_t w[U];
#pragma unroll
                for (int q = 0; q < U; q++) {
                    const bool ok = e0 + q * WAYS < end;
                    const int2 arc = ok ? arcs.arc(e0 + q * WAYS) : make_int2(0, 0);
                    w[q] = arc.y;
                    val[q] = ok ? __ldcg(a.rec + (int64_t)arc.x * LPV + sub) : inf4;
                }
#pragma unroll
                for (int q = 0; q < U; q++) x = vaddmin(val[q], w[q], x);
            }
            __syncwarp();
            x = combine(x, LPV, 32);
            changed += finish(v, beg, end, old, x, lane < LPV, lane, 32, FULL) != 0;
        }
    }
    return changed;
}

// Sweeps to convergence.  With sparse set the flags in act0 mark the vertices
// of sweep 0, else sweep 0 takes every vertex.  Returns the number of sweeps,
// or -1 after an error (recorded in the control words, or *err).
template <int LPV, typename ARCS>
__device__ int32_t narrow_sweeps(const NarrowArgs &a, const ARCS &arcs, bool sparse, uint32_t *err, int *s_ok)
{
    const int32_t gw = (int32_t)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    const int32_t nwg = (int32_t)((gridDim.x * blockDim.x) >> 5);
    const int32_t vbeg = (int32_t)((int64_t)a.n * gw / nwg), vend = (int32_t)((int64_t)a.n * (gw + 1) / nwg);
    volatile uint32_t *vctrl = a.ctrl;
    __shared__ uint8_t s_list[NARROW_THREADS];
    __shared__ unsigned s_chg;
    __shared__ uint32_t s_ctl[2];  // changed vertices of the last sweep, of the sweep before
    if (threadIdx.x == 0) {
        s_chg = 0;
        s_ctl[0] = s_ctl[1] = sparse ? 1u : (uint32_t)a.n;
    }
    __syncthreads();
    bool dense = !sparse;
    for (int32_t s = 0; s < a.max_sweeps; s++) {
        uint8_t *cur = (s & 1) ? a.act1 : a.act0, *nxt = (s & 1) ? a.act0 : a.act1;
        // the changed count of this sweep is not known yet: continue the last ratio
        const uint32_t last = s_ctl[0], before = s_ctl[1];
        const bool dense_next = min((uint64_t)a.n, (uint64_t)last * last / before) > (uint64_t)a.dense_min;
        if (blockIdx.x == 0 && threadIdx.x == 0) vctrl[C_CNT0 + (s + 1) % 4] = 0;
        const int32_t c = narrow_pass<LPV>(a, arcs, vbeg, vend, dense, !dense_next, cur, nxt,
                                          s_list + (threadIdx.x & ~31));
        if ((threadIdx.x & 31) == 0 && c) atomicAdd(&s_chg, (unsigned)c);
        __syncthreads();
        if (threadIdx.x == 0) {
            if (s_chg) atomicAdd(a.ctrl + C_CNT0 + s % 4, s_chg);
            s_chg = 0;
        }
        const bool ok = grid_barrier(a.ctrl, s_ok, [&] {
            s_ctl[1] = max(1u, s_ctl[0]);
            s_ctl[0] = vctrl[C_CNT0 + s % 4];
        });
        if (!ok) {
            if (threadIdx.x == 0) atomicOr(err, a.ctrl[C_ERR]);
            return -1;
        }
        if (s_ctl[0] == 0) return s + 1;
        dense = dense_next;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(err, (uint32_t)EMV_DEV_SWEEP_LIMIT);
    return -1;
}

// Threshold of the dense sweeps: with mean degree d and a fraction f of the
// vertices changed, a vertex has a changed neighbour with probability 1 - (1 -
// f)^d; from a half on, taking every vertex costs no more than marking.
inline int32_t narrow_dense_min(int64_t n, int64_t arcs)
{
    return arcs > 0 ? (int32_t)((double)n * (1.0 - std::pow(0.5, (double)n / (double)arcs))) : (int32_t)n;
}

}  // namespace emv
