// emv_resident.cuh -- the whole DP of one small instance in one launch.
//
// The multi-launch solver (emv_kernels.cuh) spends a small solve on launches,
// host reads and grid barriers: a relaxation sweep over a few thousand
// vertices is 10 us of barrier and latency, and a solve has 70-120 of them
// (n = 1024, k = 8: 1.03 ms of kernels; n = 4096, k = 10: 1.92 ms).  Here the
// rows of a level are dealt out to the CTAs: the closures of different rows
// are independent, so a CTA closes its rows in shared memory with CTA
// barriers only, and the grid meets twice a level (after the merge, after the
// relaxation).
//
// Phases of a level m (reader/reader-el.c:2033-2131):
//   merge  -- CTA = blocks of W vertices: the rows of sizes 1..m-1 of a block
//             are staged in shared memory, a lane computes 4 vertices of one
//             subset (R:2068-2107); few subsets split their pairs over lanes;
//   relax  -- CTA = a contiguous share of the level's rows, R at a time, as
//             states (row, vertex) with int32 distances in shared memory
//             (R:2109-2130): pull sweeps over all states while many change,
//             then rounds of pushes from the states that changed, marked in a
//             bitmap.  Dense sweeps alone would visit every arc 10-18 times a
//             row; pulls and pushes together visit 3 to 5 times.
// Arcs are kept in slices of 32 vertices, the j-th pair of arcs of the slice's
// vertices side by side: a warp that takes the 32 vertices reads them without
// bank conflicts (rows one after another, of regular degree, would fall into
// a few banks) and needs no row starts.
// Bound: instruction issue and bank conflicts of the arcs' random heads, and
// at k >= 10 the merge's shared loads.
#pragma once

#include "emv_common.cuh"
#include "emv_device_util.cuh"

namespace emv {

constexpr int RES_THREADS = 1024;
constexpr int RES_WARPS = RES_THREADS / 32;
constexpr int RES_KMAX = 11;             // most terminals whose subsets are solved
constexpr uint8_t RES_HUB_MARK = 255;    // its arc pairs in ResSmem::pairs
constexpr uint32_t RES_MAX_W = 1u << 14; // packed arcs hold smaller weights
constexpr float RES_PULL_SHARE = 0.2f;   // a round after one that changed more of the states pulls
constexpr uint32_t RES_SPIN_LIMIT = 1u << 22;  // least polls of an L2 word, over a second in all (res_spin_limit)
constexpr int RES_ACC_WORDS = 2 * RES_THREADS;  // merge minima of a level with at most half as many tasks as threads

// One instance as the device functions below take it.
struct ResInst {
    const int32_t *row_ptr;
    const int2 *adj;          // (head, weight) arcs
    void *slices;             // sliced arcs (written here)
    int32_t *table;           // 2^kt rows of stride ld
    int64_t *cost;            // d[C][t_{k-1}], INT64_MAX without a value
    uint32_t *unreached;      // if set: a level-1 closure left a vertex without a value
    uint32_t *rounds;         // if set: += rounds of the closures (pull sweeps, push rounds)
    unsigned long long *ns;   // if set: time of level 1, merges, relaxations (the first CTA's view)
    int64_t ld;
    int32_t n, k, kt;
    int32_t vec;              // table rows are 16-byte aligned
    int32_t want_rows;        // most rows of a closure
    int32_t mw;               // vertices of a merge block (multiple of 4)
    int32_t max_rounds;
    uint32_t inv_slices;      // ceil(2^32 / slices), for slices > 1
    int32_t hub_min;          // a vertex of more arcs is walked by a whole warp (res_hub_min)
};

// The CTAs that share an instance: all of them on the GPU at once.
struct ResTeam {
    uint32_t *bar;            // arrivals, on a line of its own, zero at first
    uint32_t *err;            // EMV_DEV_* bits
    int32_t rank, size;
    uint32_t epoch;           // barriers passed
    uint32_t limit;           // polls at a barrier (res_spin_limit)
};

// A CTA's static shared memory.
struct ResShared {
    int ok;                   // 1 until the team failed
    int32_t terms[EMV_MAX_K];
    int32_t hubs[RES_WARPS];
    int32_t lvl[RES_KMAX + 2];  // level m of the subset list: [lvl[m], lvl[m + 1])
};

// Control and result words of one k_resident launch (zeroed before it).
struct ResOut {
    uint32_t bar[32];
    uint32_t err;
    uint32_t unreached;
    uint32_t rounds;
    uint32_t refused;         // the CSR check found a fault: no row was filled
    GraphScan scan;
    unsigned long long ns[3];
    int64_t cost;
    int32_t terms[EMV_MAX_K];
};

struct ResArgs {
    ResInst inst;
    const int32_t *col, *w;   // the CSR as given
    int2 *adj;                // (head, weight) arcs (written here; also read by the traceback)
    const uint32_t *xs;       // subsets by level
    ResOut *out;
    int64_t arcs;
    int32_t check;            // leave after the CSR check found a fault
    int32_t smem;             // dynamic shared memory
    uint32_t spin_limit;
    int32_t lvl[RES_KMAX + 2];
    int32_t terms[EMV_MAX_K];
};

// The parts of the shared memory: subsets by level, the first arc pair of
// every slice, the arc pairs of every vertex, and the rest for the phases.
struct ResSmem {              // byte offsets
    int32_t xs;               // uint16
    int32_t slice;            // int32, slices + 1
    int32_t pairs;            // uint8, 32 * slices
    int32_t big, end;
};
__host__ __device__ inline int32_t res_fixed_smem(int32_t n, int32_t kt)
{
    const int32_t slices = (n + 31) / 32;
    return ((2 << kt) + 15) / 16 * 16 + (4 * (slices + 1) + 15) / 16 * 16 + 32 * slices;
}

extern __shared__ __align__(16) unsigned char res_smem[];
// Shared memory by byte offset: 32-bit addresses whatever the caller holds.
template <typename T> __device__ __forceinline__ T &res_at(int32_t off) { return *reinterpret_cast<T *>(res_smem + off); }
__device__ __forceinline__ volatile int32_t &res_i32(int32_t off)
{
    return *reinterpret_cast<volatile int32_t *>(res_smem + off);
}

constexpr uint32_t RES_FAILED = 1u << 31;  // set in the barrier word when a CTA failed

// Records an error and makes every CTA of the team leave at its next barrier.
__device__ __forceinline__ void res_fail(const ResTeam &t, uint32_t err, ResShared &sh)
{
    atomicOr(t.err, err);
    atomicOr(t.bar, RES_FAILED);
    *(volatile int *)&sh.ok = 0;
}

// Barrier over the team's CTAs.  Arrivals only count up, so no word is reset.
// Bounded: a CTA that waits longer than t.limit polls records the error; every
// CTA of the team leaves when it sees one.
__device__ __forceinline__ bool res_barrier(ResTeam &t, ResShared &sh)
{
    __syncthreads();
    t.epoch++;
    if (t.size > 1) {
        if (threadIdx.x == 0) {
            const uint32_t target = t.epoch * (uint32_t)t.size;
            uint32_t spins = 0, seen;
            __threadfence();
            atomicAdd(t.bar, 1u);
            for (;;) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(t.bar) : "memory");
                if ((seen & RES_FAILED) || (seen & ~RES_FAILED) >= target) break;
                if (++spins > t.limit) {
                    res_fail(t, EMV_DEV_BARRIER_TIMEOUT, sh);
                    break;
                }
            }
            if (seen & RES_FAILED) *(volatile int *)&sh.ok = 0;
        }
        __syncthreads();
    }
    return *(volatile int *)&sh.ok != 0;
}

__device__ __forceinline__ unsigned long long res_now()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// The p-th subset of mask in the order (s - mask) & mask steps through.
__device__ __forceinline__ uint32_t res_deposit(uint32_t p, uint32_t mask)
{
    uint32_t r = 0;
    for (; p && mask; p >>= 1) {
        const uint32_t low = mask & (0u - mask);
        if (p & 1u) r |= low;
        mask ^= low;
    }
    return r;
}

// ---------------------------------------------------------------- merge

__device__ __forceinline__ uint4 res_pairs(const uint4 *__restrict__ Sq, int32_t Q, uint32_t X, uint32_t p0, uint32_t p1)
{
    const uint32_t low = X & (0u - X), rest = X ^ low;
    uint4 a = make_uint4((uint32_t)INF, (uint32_t)INF, (uint32_t)INF, (uint32_t)INF);
    uint32_t sub = p0 ? res_deposit(p0, rest) : 0u;
#pragma unroll 2
    for (uint32_t p = p0; p < p1; p++) {
        const uint32_t Y = low | sub;
        const uint4 y = Sq[Y * Q], z = Sq[(X ^ Y) * Q];
        a.x = __viaddmin_u32(y.x, z.x, a.x);
        a.y = __viaddmin_u32(y.y, z.y, a.y);
        a.z = __viaddmin_u32(y.z, z.z, a.z);
        a.w = __viaddmin_u32(y.w, z.w, a.w);
        sub = (sub - rest) & rest;
    }
    return a;
}

// Bytes of the merge's staged rows and of the minima of split pair lists.
__host__ __device__ inline int32_t res_merge_bytes(int32_t mw, int32_t kt) { return ((4 * mw) << kt) + 4 * RES_ACC_WORDS; }

// Finishes 4 merged vertices from v on of subset X: the arcs of the virtual
// source (R:2099-2107; value(Y, d): vertex v + d of row Y) and the store.
template <typename F>
__device__ __forceinline__ void res_merged(const ResInst &a, const int32_t *terms, bool has_term, uint32_t X, int32_t v,
                                           uint4 r, F value)
{
    if (has_term)
        for (uint32_t bits = X; bits; bits &= bits - 1) {
            const int ti = __ffs(bits) - 1, d = terms[ti] - v;
            if (d < 0 || d >= 4) continue;
            const uint32_t o = value(X ^ (1u << ti), d);
            if (d == 0) r.x = o;
            else if (d == 1) r.y = o;
            else if (d == 2) r.z = o;
            else r.w = o;
        }
    int32_t *dst = a.table + (int64_t)X * a.ld + v;
    if (a.vec && v + 4 <= a.n) *reinterpret_cast<uint4 *>(dst) = r;
    else {
        if (v < a.n) dst[0] = (int32_t)r.x;
        if (v + 1 < a.n) dst[1] = (int32_t)r.y;
        if (v + 2 < a.n) dst[2] = (int32_t)r.z;
        if (v + 3 < a.n) dst[3] = (int32_t)r.w;
    }
}

// Four vertices of a table row from v on (INF past n).
__device__ __forceinline__ int4 res_row4(const ResInst &a, uint32_t X, int32_t v)
{
    const int32_t *src = a.table + (int64_t)X * a.ld + v;
    if (a.vec && v + 4 <= a.n) return __ldcg(reinterpret_cast<const int4 *>(src));
    return make_int4(v < a.n ? __ldcg(src) : INF, v + 1 < a.n ? __ldcg(src + 1) : INF, v + 2 < a.n ? __ldcg(src + 2) : INF,
                     v + 3 < a.n ? __ldcg(src + 3) : INF);
}

// Merge of level m for this CTA's vertex blocks, in the last res_merge_bytes
// of the shared memory: 2^kt rows of mw words (row Y at Y * mw) and, after
// them, the minima of split pair lists.  (Blocks of half the width in two
// halves of that space, the next staged while one is reduced: 280 against 212
// us at n = 4000, kt = 11, and 5 % more time for 4096 mixed instances; level 2
// read directly from the table, one pair a subset: the same.)
__device__ __forceinline__ void res_merge(const ResInst &a, const ResTeam &tm, const ResSmem &sm, const ResShared &sh,
                                          int32_t m)
{
    const uint16_t *xs = &res_at<uint16_t>(sm.xs);
    const int32_t *terms = sh.terms;
    const int32_t n = a.n, tid = threadIdx.x, kt = a.kt;
    const int32_t nlow = sh.lvl[m], cnt = sh.lvl[m + 1] - nlow;
    uint32_t *S = &res_at<uint32_t>(sm.end - res_merge_bytes(a.mw, kt));
    uint32_t *acc = S + ((size_t)a.mw << kt);
    const int32_t W = a.mw, Q = W / 4;
    const uint32_t npairs = (1u << (m - 1)) - 1;
    const int32_t tasks = cnt * Q;
    int32_t parts = 1;
    while (tasks * parts * 2 <= RES_THREADS && (uint32_t)parts * 2 <= npairs) parts *= 2;
    const uint4 *S4 = reinterpret_cast<const uint4 *>(S);
    for (int32_t v0 = tm.rank * W; v0 < n; v0 += tm.size * W) {
        for (int32_t i = tid; i < nlow * Q; i += RES_THREADS) {
            const int32_t r = i / Q, q = i - r * Q, v = v0 + 4 * q;
            const uint32_t Y = xs[r];
            int4 *to = reinterpret_cast<int4 *>(S) + Y * Q + q;
            // a row is ld >= n words: its last quad may hold words past n
            if (a.vec && v < n) cp_async16(to, a.table + (int64_t)Y * a.ld + v);
            else if (!a.vec) *to = res_row4(a, Y, v);
        }
        if (parts > 1)
            for (int32_t i = tid; i < cnt * W; i += RES_THREADS) acc[i] = (uint32_t)INF;
        cp_async_wait_all();
        __syncthreads();
        bool has_term = false;
        for (int32_t t = 0; t < kt; t++) has_term |= terms[t] >= v0 && terms[t] < v0 + W;
        if (parts > 1) {
            for (int32_t t = tid; t < tasks * parts; t += RES_THREADS) {
                const int32_t part = t / tasks, u = t - part * tasks, xi = u / Q, q = u - xi * Q;
                const uint4 r = res_pairs(S4 + q, Q, xs[nlow + xi], npairs * (uint32_t)part / (uint32_t)parts,
                                          npairs * (uint32_t)(part + 1) / (uint32_t)parts);
                uint32_t *A = acc + 4 * u;
                atomicMin(A + 0, r.x);
                atomicMin(A + 1, r.y);
                atomicMin(A + 2, r.z);
                atomicMin(A + 3, r.w);
            }
            __syncthreads();
        }
        for (int32_t t = tid; t < tasks; t += RES_THREADS) {
            const int32_t xi = t / Q, q = t - xi * Q;
            const uint32_t X = xs[nlow + xi];
            const uint4 r = parts > 1 ? reinterpret_cast<const uint4 *>(acc)[t] : res_pairs(S4 + q, Q, X, 0, npairs);
            res_merged(a, terms, has_term, X, v0 + 4 * q, r,
                       [&](uint32_t Y, int d) { return S[Y * W + 4 * q + d]; });
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- relax

// Sliced arcs, a pair of arcs per element: packed words (head * 4 | weight <<
// 18, the head as a byte offset) in shared or global memory, or both arcs as
// (head * 4, weight) in global memory, for weights of 2^14 and more.  Element
// j of the vertex at lane l of slice i: (slice[i] + j) * 32 + l.  A vertex
// with fewer pairs than its slice's widest (and the second arc of an odd
// last pair) is padded with an arc to itself that improves nothing; vertices
// of more than hub_min arcs have no pairs here and are read from adj.
enum ResArcs { ARCS_SMEM, ARCS_PACKED, ARCS_WIDE };

template <ResArcs SRC> struct ResElem {
    using T = uint2;
};
template <> struct ResElem<ARCS_WIDE> {
    using T = int4;
};

template <ResArcs SRC> struct ResGraph {
    using T = typename ResElem<SRC>::T;
    const T *el;              // global memory
    int32_t el_off;           // ARCS_SMEM: byte offset in shared memory
    int32_t slice, pairs;     // byte offsets (ResSmem)
    __device__ __forceinline__ T elem(int32_t i) const
    {
        if constexpr (SRC == ARCS_SMEM) return res_at<T>(el_off + i * (int32_t)sizeof(T));
        else return el[i];
    }
    // Adds the two arcs of an element to a minimum (row: byte offset of the
    // row's distances).
    __device__ __forceinline__ int32_t pull(const T &x, int32_t row, int32_t acc) const
    {
        int32_t off[2], w[2];
        unpack(x, off, w);
        const int32_t p = res_i32(row + off[0]), q = res_i32(row + off[1]);
        return __viaddmin_s32(q, w[1], __viaddmin_s32(p, w[0], acc));
    }
    static __device__ __forceinline__ void unpack(const T &x, int32_t (&off)[2], int32_t (&w)[2])
    {
        if constexpr (SRC == ARCS_WIDE) {
            off[0] = x.x;
            w[0] = x.y;
            off[1] = x.z;
            w[1] = x.w;
        } else {
            off[0] = (int32_t)(x.x & 0x3ffffu);
            w[0] = (int32_t)(x.x >> 18);
            off[1] = (int32_t)(x.y & 0x3ffffu);
            w[1] = (int32_t)(x.y >> 18);
        }
    }
};

// wd / slices for a word index below 2^16 (inv: ResInst::inv_slices).
__device__ __forceinline__ int32_t res_div(uint32_t inv, int32_t wd, int32_t slices)
{
    return slices == 1 ? wd : (int32_t)__umulhi((uint32_t)wd, inv);
}

// Closure of R rows in shared memory: states s = r * 32 * slices + v,
// distances at byte offset d + 4 * s (INF for v >= n).  A warp owns the states
// of a contiguous run of bitmap words, a word being one row's states of one
// slice.
//
// Closures of at most a word a warp and four arc pairs a vertex keep the arcs
// in registers and pull three times between barriers until nothing changes
// (one pull a barrier: 40 % more time at n = 1024, degree 4).
//
// Others switch between two kinds of rounds.  A pull sweep takes every state:
// no atomics and few instructions an arc, for rounds in which many states
// change; it leaves the marks (bitmap bits) of the states it changed.  A push
// round takes the marked states: a warp lists its own and pushes from them
// (taking marks again before the barrier, as they arrive: 8 % more time at n =
// 20 000, the pushes of not yet settled distances cost more than the barriers
// they save).  A mark is taken by an exchange before its state's distance is
// read and set after a distance was lowered, so none is lost; it is set
// whenever a value looked improvable, and a lost race costs a visit.
//
// Graphs with vertices of more than hub_min arcs list those apart (from the
// far end of the warp's part), and after a barrier all warps share them, a
// warp per vertex: one warp would otherwise walk all hubs of its run.
// Returns false when max_rounds ran out; `rounds` counts barriers passed.
template <ResArcs SRC>
__device__ bool res_close(const ResInst &a, const ResGraph<SRC> &g, bool has_hubs, int32_t R, bool level1, int32_t d,
                          int32_t list, int32_t bm, int32_t *hub_cnt, int32_t &rounds)
{
    using G = ResGraph<SRC>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1;
    const int32_t slices = (a.n + 31) >> 5, words = R * slices, max_rounds = a.max_rounds;
    const uint32_t inv = a.inv_slices;
    auto row_of = [&](int32_t wd) -> int32_t { return R == 1 ? 0 : res_div(inv, wd, slices); };
    // this warp's words; its list holds at most their states
    const int32_t per = (words + RES_WARPS - 1) / RES_WARPS;
    const int32_t w0 = min(words, warp * per), w1 = min(words, w0 + per);
    rounds = 0;

    if (per == 1 && !has_hubs) {
        const int32_t wd = min(w0, words - 1), r = row_of(wd), sl = wd - r * slices, row = d + r * slices * 128;
        const int32_t first = res_i32(g.slice + 4 * sl), width = res_i32(g.slice + 4 * sl + 4) - first;
        if (__syncthreads_and(width <= 4)) {
            const int32_t own = d + (wd * 32 + lane) * 4;
            typename G::T x[4];
#pragma unroll
            for (int j = 0; j < 4; j++) x[j] = g.elem((first + min(j, max(width - 1, 0))) * 32 + lane);
            bool changed = false;
            do {
                if (++rounds > max_rounds) return false;
                changed = false;
                if (w0 < words && width > 0)
#pragma unroll
                    for (int pass = 0; pass < 3; pass++) {
                        const int32_t old = res_i32(own);
                        int32_t y = old;
#pragma unroll
                        for (int j = 0; j < 4; j++)
                            if (j < width) y = g.pull(x[j], row, y);
                        if (y < old) {
                            res_i32(own) = y;
                            changed = true;
                        }
                    }
            } while (__syncthreads_or(changed));
            return true;
        }
    }

    const int32_t mylist = list + w0 * 64, myend = list + w1 * 64;  // byte offsets of 16-bit entries
    // index j of all warps' hubs -> its state (every warp, uniform j)
    int32_t hub_all = 0, hub_pre = 0;
    auto hub_count = [&]() {
        hub_pre = hub_cnt[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(FULL, hub_pre, o);
            if (lane >= o) hub_pre += t;
        }
        hub_all = __shfl_sync(FULL, hub_pre, 31);
    };
    auto hub_state = [&](int32_t j) -> int32_t {
        const int w = __popc(__ballot_sync(FULL, hub_pre <= j));
        const int32_t before = __shfl_sync(FULL, hub_pre, max(w - 1, 0));
        const int32_t end = min(words, (w + 1) * per) * 32;
        return res_at<uint16_t>(list + 2 * (end - 1 - (j - (w ? before : 0))));
    };
    auto is_hub = [&](int32_t v) -> bool { return res_at<uint8_t>(g.pairs + v) == RES_HUB_MARK; };
    // threads with a change among their `per` states when RES_PULL_SHARE of all states change
    float same = 1.0f;
    for (int32_t i = 0; i < per && i < 16; i++) same *= 1.0f - RES_PULL_SHARE;
    const int many = (int)(RES_THREADS * (1.0f - same));
    bool pull = !level1, any = true;
    for (;;) {
        if (++rounds > max_rounds) return false;
        if (pull) {
            int32_t hubs = 0;
            any = false;
            for (int32_t wd = w0; wd < w1; wd++) {
                const int32_t r = row_of(wd), sl = wd - r * slices, s = wd * 32 + lane, row = d + r * slices * 128;
                const int32_t old = res_i32(d + 4 * s);
                int32_t x = old;
                if (has_hubs) {
                    const bool hub = is_hub(sl * 32 + lane);
                    const unsigned hb = __ballot_sync(FULL, hub);
                    if (hub) res_at<uint16_t>(myend - 2 - 2 * (hubs + __popc(hb & lt))) = (uint16_t)s;
                    hubs += __popc(hb);
                }
                int32_t e = res_i32(g.slice + 4 * sl);
                int32_t left = res_i32(g.slice + 4 * sl + 4) - e;
                e = e * 32 + lane;
                for (; left >= 2; left -= 2, e += 64) {
                    const typename G::T x0 = g.elem(e), x1 = g.elem(e + 32);
                    x = g.pull(x0, row, x);
                    x = g.pull(x1, row, x);
                }
                if (left) x = g.pull(g.elem(e), row, x);
                const bool dec = x < old;
                if (dec) res_i32(d + 4 * s) = x;
                any |= dec;
                const unsigned bal = __ballot_sync(FULL, dec);
                if (lane == 0) res_at<uint32_t>(bm + 4 * wd) = bal;
            }
            if (has_hubs) {
                if (lane == 0) hub_cnt[warp] = hubs;
                __syncthreads();
                hub_count();
                for (int32_t j = warp; j < hub_all; j += RES_WARPS) {
                    const int32_t s = hub_state(j), r = row_of(s >> 5), v = s - r * slices * 32, row = d + r * slices * 128;
                    const int32_t beg = __ldg(a.row_ptr + v), end = __ldg(a.row_ptr + v + 1);
                    int32_t x = INF;
#pragma unroll 4
                    for (int32_t q = beg + lane; q < end; q += 32) {
                        const int2 arc = a.adj[q];
                        x = min(x, res_i32(row + 4 * arc.x) + arc.y);
                    }
                    x = __reduce_min_sync(FULL, x);
                    const bool dec = x < res_i32(d + 4 * s);
                    __syncwarp();
                    if (dec && lane == 0) {
                        res_i32(d + 4 * s) = x;
                        atomicOr(&res_at<uint32_t>(bm + 4 * (s >> 5)), 1u << (s & 31));
                    }
                    any |= dec;
                }
            }
        } else {
            any = false;
            auto push = [&](int32_t row, int32_t off, int32_t nd) {
                const int32_t t = (row - d + off) >> 2;
                atomicMin(&res_at<int32_t>(row + off), nd);
                atomicOr(&res_at<uint32_t>(bm + 4 * (t >> 5)), 1u << (t & 31));
                any = true;
            };
            // list this warp's marked states, taking their marks
            int32_t total = 0, hubs = 0;
            for (int32_t wb = w0; wb < w1; wb += 32) {
                const int32_t mine = wb + lane;
                uint32_t word = mine < w1 ? (uint32_t)res_i32(bm + 4 * mine) : 0u;
                if (word) word = atomicExch(&res_at<uint32_t>(bm + 4 * mine), 0u);
                for (unsigned some = __ballot_sync(FULL, word != 0); some; some &= some - 1) {
                    const int j = __ffs(some) - 1;
                    uint32_t bits = __shfl_sync(FULL, word, j);
                    const int32_t wd = wb + j, s = wd * 32 + lane;
                    if (has_hubs) {
                        const unsigned hb = __ballot_sync(
                            FULL, (bits >> lane & 1u) && is_hub((wd - row_of(wd) * slices) * 32 + lane));
                        if (hb >> lane & 1u)
                            res_at<uint16_t>(myend - 2 - 2 * (hubs + __popc(hb & lt))) = (uint16_t)s;
                        hubs += __popc(hb);
                        bits &= ~hb;
                    }
                    if (bits >> lane & 1u) res_at<uint16_t>(mylist + 2 * (total + __popc(bits & lt))) = (uint16_t)s;
                    total += __popc(bits);
                }
            }
            __syncwarp();
            // fewer states than lanes: several lanes share a state's arcs
            const int sh = total == 0 || total > 16 ? 0 : 5 - (32 - __clz(total - 1));
            const int L = 1 << sh, sub = lane & (L - 1);
            for (int32_t i = lane >> sh; i < total; i += 32 >> sh) {
                const int32_t s = res_at<uint16_t>(mylist + 2 * i), wd = s >> 5, r = row_of(wd), sl = wd - r * slices;
                const int32_t row = d + r * slices * 128, ds = res_i32(d + 4 * s);
                const int32_t np = res_at<uint8_t>(g.pairs + sl * 32 + (s & 31));
                const int32_t e = res_i32(g.slice + 4 * sl) * 32 + (s & 31);
                for (int32_t p = sub; p < np; p += 2 * L) {
                    const bool two = p + L < np;
                    int32_t o0[2], w0_[2], o1[2], w1_[2];
                    const typename G::T x0 = g.elem(e + p * 32), x1 = g.elem(e + (two ? p + L : p) * 32);
                    G::unpack(x0, o0, w0_);
                    G::unpack(x1, o1, w1_);
                    const int32_t h0 = res_i32(row + o0[0]), h1 = res_i32(row + o0[1]), h2 = res_i32(row + o1[0]),
                                  h3 = res_i32(row + o1[1]);
                    if (ds + w0_[0] < h0) push(row, o0[0], ds + w0_[0]);
                    if (ds + w0_[1] < h1) push(row, o0[1], ds + w0_[1]);
                    if (two && ds + w1_[0] < h2) push(row, o1[0], ds + w1_[0]);
                    if (two && ds + w1_[1] < h3) push(row, o1[1], ds + w1_[1]);
                }
            }
            if (has_hubs) {
                if (lane == 0) hub_cnt[warp] = hubs;
                __syncthreads();
                hub_count();
                for (int32_t j = warp; j < hub_all; j += RES_WARPS) {
                    const int32_t s = hub_state(j), r = row_of(s >> 5), v = s - r * slices * 32, ds = res_i32(d + 4 * s);
                    const int32_t row = d + r * slices * 128;
                    const int32_t beg = __ldg(a.row_ptr + v), end = __ldg(a.row_ptr + v + 1);
#pragma unroll 4
                    for (int32_t q = beg + lane; q < end; q += 32) {
                        const int2 arc = a.adj[q];
                        if (ds + arc.y < res_i32(row + 4 * arc.x)) push(row, 4 * arc.x, ds + arc.y);
                    }
                }
            }
        }
        const int all = __syncthreads_count(any);
        if (all == 0) return true;
        pull = all > many;
    }
}

// Bytes of the states of R rows: distances, lists, the bitmap.
__host__ __device__ inline int64_t res_state_bytes(int32_t n, int64_t R) { return (n + 31) / 32 * R * 196; }

// Closure of nr <= R rows (R = 8, 16, .. 128) kept vertex by vertex: the R
// distances of a vertex side by side, four to a lane, so that an arc is
// decoded once for four rows and its head is read with 16-byte loads, which
// meet the fewer bank conflicts the more rows lie together (none from 32 on,
// where a quarter-warp reads 128 bytes).  A sweep takes every vertex, but for
// a row and arc it needs a third of res_close's instructions, which outweighs
// that res_close takes fewer states; used for shares of at least
// RES_WIDE_MIN rows.  From 32 rows on, 16 bytes of padding per vertex keep the
// transposing copies free of conflicts.  Returns false when max_rounds ran out.
constexpr int RES_WIDE_SMALL = 8192;  // states
constexpr int RES_WIDE_MIN = 6;
constexpr int RES_WIDE_SMEM = 8;   // arcs stay in shared memory when this many rows fit beside them

__host__ __device__ inline int32_t res_wide_words(int32_t R) { return R < 32 ? R : R + 4; }
__host__ __device__ inline int64_t res_wide_bytes(int32_t n, int32_t R) { return (int64_t)n * res_wide_words(R) * 4; }

template <ResArcs SRC>
__device__ bool res_wide(const ResInst &a, const ResGraph<SRC> &g, int32_t R, int32_t nr, const uint16_t *xs, int32_t d,
                         int32_t &rounds)
{
    using G = ResGraph<SRC>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t n = a.n, slices = (n + 31) >> 5, scale = res_wide_words(R), stride = scale * 4, max_rounds = a.max_rounds;
    const uint32_t inv = a.inv_slices;
    const int64_t ld = a.ld;
    int32_t *table = a.table;
    // a warp moves four rows of one slice
    auto each = [&](auto f) {
#pragma unroll 2
        for (int32_t i = warp; i < R / 4 * slices; i += RES_WARPS) {
            const int32_t q = res_div(inv, i, slices), v = (i - q * slices) * 32 + lane;
            if (v < n) f(4 * q, v, res_at<int4>(d + v * stride + 16 * q));
        }
    };
    each([&](int32_t r, int32_t v, int4 &x) {
        x.x = r < nr ? __ldcg(table + xs[r] * ld + v) : INF;
        x.y = r + 1 < nr ? __ldcg(table + xs[r + 1] * ld + v) : INF;
        x.z = r + 2 < nr ? __ldcg(table + xs[r + 2] * ld + v) : INF;
        x.w = r + 3 < nr ? __ldcg(table + xs[r + 3] * ld + v) : INF;
    });
    __syncthreads();
    const int lpv = R / 4, vpw = 32 / lpv;  // lanes of a vertex, vertices of a warp
    const int32_t mine = d + (lane & (lpv - 1)) * 16, sub = lane / lpv;
    bool changed;
    rounds = 0;
    do {
        if (++rounds > max_rounds) return false;
        changed = false;
        for (int32_t v0 = warp * vpw; v0 < n; v0 += RES_WARPS * vpw) {
            const int32_t v = v0 + sub, sl = v0 >> 5;
            if (v >= n) continue;
            int4 &own = res_at<int4>(mine + v * stride);
            const int4 old = own;
            int4 x = old;
            int32_t e = res_i32(g.slice + 4 * sl);
            const int32_t width = res_i32(g.slice + 4 * sl + 4) - e;
            e = e * 32 + (v & 31);
#pragma unroll 2
            for (int32_t j = 0; j < width; j++) {
                int32_t off[2], w[2];
                G::unpack(g.elem(e + 32 * j), off, w);
                const int4 p = res_at<int4>(mine + off[0] * scale), q = res_at<int4>(mine + off[1] * scale);
                x = vaddmin(p, w[0], x);  // off counts 4 bytes a vertex, a record has 4 * scale
                x = vaddmin(q, w[1], x);
            }
            if (vlt(x, old)) {
                own = x;
                changed = true;
            }
        }
    } while (__syncthreads_or(changed));
    each([&](int32_t r, int32_t v, int4 &x) {
        if (r < nr) table[xs[r] * ld + v] = x.x;
        if (r + 1 < nr) table[xs[r + 1] * ld + v] = x.y;
        if (r + 2 < nr) table[xs[r + 2] * ld + v] = x.z;
        if (r + 3 < nr) table[xs[r + 3] * ld + v] = x.w;
    });
    return true;
}

// Records of the next closure of a share with `left` rows: R rows vertex by
// vertex (R <= cap), or 0 for res_close.
__device__ __forceinline__ int32_t res_wide_rows(int32_t n, int32_t left, int32_t cap)
{
    if (cap < 8 || left < RES_WIDE_MIN) return 0;
    int32_t R = 8;
    while (R < cap && left > R) R *= 2;
    // a quarter of the rows may be idle, more where latency outweighs the work
    if (R > 8 && left * 4 < R * 3 && n * R > RES_WIDE_SMALL) R /= 2;
    return R;
}

// Relaxation of this CTA's rows of level m, at most `rows` at a time, from
// byte offset dyn of the shared memory.
template <ResArcs SRC>
__device__ void res_relax(const ResInst &a, const ResTeam &tm, const ResGraph<SRC> &g, const ResSmem &sm, ResShared &sh,
                          bool has_hubs, int32_t m, int32_t dyn, int32_t rows, int32_t wide_cap)
{
    const int32_t *terms = sh.terms;
    const int32_t n = a.n, slices = (n + 31) >> 5, np = slices * 32, cnt = sh.lvl[m + 1] - sh.lvl[m];
    const int32_t rb = (int32_t)((int64_t)cnt * tm.rank / tm.size),
                  re = (int32_t)((int64_t)cnt * (tm.rank + 1) / tm.size);
    const uint32_t C = (1u << (a.k - 1)) - 1;
    uint32_t rounds = 0;
    for (int32_t r0 = rb, R; r0 < re; r0 += R) {
        const uint16_t *xs = &res_at<uint16_t>(sm.xs) + sh.lvl[m] + r0;
        const int32_t wide = m > 1 ? res_wide_rows(n, re - r0, wide_cap) : 0;
        if (wide) {
            R = min(wide, re - r0);
            int32_t did = 0;
            const bool ok = res_wide<SRC>(a, g, wide, R, xs, dyn, did);
            rounds += did;
            if (!ok) {
                if (threadIdx.x == 0) res_fail(tm, EMV_DEV_SWEEP_LIMIT, sh);
                __syncthreads();
                break;
            }
            if (m == a.k - 1)
                for (int32_t r = threadIdx.x; r < R; r += RES_THREADS)
                    if (xs[r] == C) {
                        const int32_t x = res_i32(dyn + (terms[a.k - 1] * res_wide_words(wide) + r) * 4);
                        *a.cost = x < INF ? (int64_t)x : INT64_MAX;
                    }
            __syncthreads();
            continue;
        }
        R = min(rows, re - r0);
        const int32_t words = R * slices;
        int32_t *d = &res_at<int32_t>(dyn);
        uint32_t *bm = &res_at<uint32_t>(dyn + words * 128);
        // four states of a row at a time
        auto quads = [&](auto f) {
#pragma unroll 2
            for (int32_t i = threadIdx.x; i < words * 8; i += RES_THREADS) {
                const int32_t r = R == 1 ? 0 : res_div(a.inv_slices, i >> 3, slices);
                const int32_t v = i * 4 - r * np;
                f(i, v, a.table + (int64_t)xs[r] * a.ld + v);
            }
        };
        if (m == 1)
            for (int32_t i = threadIdx.x; i < words * 8; i += RES_THREADS)
                reinterpret_cast<int4 *>(d)[i] = make_int4(INF, INF, INF, INF);
        else
            quads([&](int32_t i, int32_t v, const int32_t *src) {
                int4 x;
                if (a.vec && v + 4 <= n) x = __ldcg(reinterpret_cast<const int4 *>(src));
                else
                    x = make_int4(v < n ? __ldcg(src) : INF, v + 1 < n ? __ldcg(src + 1) : INF,
                                  v + 2 < n ? __ldcg(src + 2) : INF, v + 3 < n ? __ldcg(src + 3) : INF);
                reinterpret_cast<int4 *>(d)[i] = x;
            });
        for (int32_t i = threadIdx.x; i < words; i += RES_THREADS) bm[i] = 0;
        __syncthreads();
        if (m == 1) {
            for (int32_t r = threadIdx.x; r < R; r += RES_THREADS) {
                const int32_t s = r * np + terms[__ffs(xs[r]) - 1];
                d[s] = 0;
                atomicOr(bm + (s >> 5), 1u << (s & 31));
            }
            __syncthreads();
        }
        int32_t did = 0;
        const bool ok = res_close<SRC>(a, g, has_hubs, R, m == 1, dyn, dyn + words * 132, dyn + words * 128, sh.hubs, did);
        rounds += did;
        if (!ok && threadIdx.x == 0) res_fail(tm, EMV_DEV_SWEEP_LIMIT, sh);
        bool unreached = false;
        quads([&](int32_t i, int32_t v, int32_t *dst) {
            const int4 x = reinterpret_cast<const int4 *>(d)[i];
            if (a.vec && v + 4 <= n) {
                *reinterpret_cast<int4 *>(dst) = x;
                unreached |= max(max(x.x, x.y), max(x.z, x.w)) >= INF;
                return;
            }
            const int32_t y[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (v + q < n) {
                    dst[q] = y[q];
                    unreached |= y[q] >= INF;
                }
        });
        if (m == 1 && unreached && a.unreached) *a.unreached = 1;
        if (m == a.k - 1)
            for (int32_t r = threadIdx.x; r < R; r += RES_THREADS)
                if (xs[r] == C) {
                    const int32_t x = d[r * np + terms[a.k - 1]];
                    *a.cost = x < INF ? (int64_t)x : INT64_MAX;
                }
        __syncthreads();
        if (!ok) break;
    }
    if (threadIdx.x == 0 && rounds && a.rounds) atomicAdd(a.rounds, rounds);
}

// Levels lo..hi.  Arcs that the closures keep in shared memory are copied there
// again for every level as far as the merge's staging overlaps them, between
// the merge and the barrier after it.
template <ResArcs SRC>
__device__ void res_levels(const ResInst &a, ResTeam &tm, const ResSmem &sm, ResShared &sh, bool has_hubs, int32_t lo,
                           int32_t hi)
{
    using T = typename ResElem<SRC>::T;
    const bool clock = a.ns && tm.rank == 0 && threadIdx.x == 0;
    unsigned long long t0 = clock ? res_now() : 0;
    const int32_t slices = (a.n + 31) >> 5;
    const int32_t arc_bytes = SRC == ARCS_SMEM ? res_i32(sm.slice + 4 * slices) * 32 * (int32_t)sizeof(T) : 0;
    const ResGraph<SRC> g{reinterpret_cast<const T *>(a.slices), sm.big, sm.slice, sm.pairs};
    const int32_t dyn = sm.big + arc_bytes;
    // the merge's part of the shared memory ends at sm.end: arcs below stay
    const int32_t keep = max(0, sm.end - res_merge_bytes(a.mw, a.kt) - sm.big) / 16 * 16;
    // rows of a closure: what fits, and their states must fit 16 bits
    const int32_t rows = (int32_t)min(min((int64_t)a.want_rows, (int64_t)(65535 / (32 * slices))),
                                      (sm.end - dyn) / res_state_bytes(a.n, 1));
    int32_t wide_cap = has_hubs ? 0 : 128;
    while (wide_cap >= 8 && (wide_cap > 2 * a.want_rows || res_wide_bytes(a.n, wide_cap) > sm.end - dyn)) wide_cap /= 2;
    for (int32_t m = lo; m <= hi; m++) {
        if (m > 1) res_merge(a, tm, sm, sh, m);
        for (int32_t i = (m == lo ? 0 : keep) + threadIdx.x * 16; i < arc_bytes; i += RES_THREADS * 16)
            cp_async16(&res_at<int4>(sm.big + i), (const char *)a.slices + i);
        if (m > 1) {
            if (!res_barrier(tm, sh)) break;
            if (clock) {
                const unsigned long long t = res_now();
                a.ns[1] += t - t0;
                t0 = t;
            }
        }
        cp_async_wait_all();  // made visible to the CTA by the barrier before the closure
        res_relax<SRC>(a, tm, g, sm, sh, has_hubs, m, dyn, rows, wide_cap);
        if (m < hi && !res_barrier(tm, sh)) break;
        if (clock) {
            const unsigned long long t = res_now();
            a.ns[m == 1 ? 0 : 2] += t - t0;
            t0 = t;
        }
    }
    cp_async_wait_all();
}

// Widths of the slices in arc pairs, their prefix sums (sm.slice) and the
// pairs of every vertex; needs at most RES_THREADS slices.  Returns whether a
// vertex has more than hub_min arcs.
__device__ __forceinline__ bool res_slice_starts(const ResInst &a, const ResSmem &sm, int32_t *warp_sums)
{
    bool hub = false;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t slices = (a.n + 31) >> 5;
    int32_t *slice = &res_at<int32_t>(sm.slice);
    for (int32_t i = warp; i < slices; i += RES_WARPS) {
        const int32_t v = i * 32 + lane;
        const int32_t deg = v < a.n ? __ldg(a.row_ptr + v + 1) - __ldg(a.row_ptr + v) : 0;
        const bool big = deg > a.hub_min;
        const int32_t np = big ? 0 : (deg + 1) / 2;
        hub |= big;
        res_at<uint8_t>(sm.pairs + v) = big ? RES_HUB_MARK : (uint8_t)np;
        const int32_t width = __reduce_max_sync(FULL, np);
        if (lane == 0) slice[i] = width;
    }
    __syncthreads();
    const int32_t own = threadIdx.x < slices ? slice[threadIdx.x] : 0;
    int32_t pre = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t t = __shfl_up_sync(FULL, pre, o);
        if (lane >= o) pre += t;
    }
    if (lane == 31) warp_sums[warp] = pre;
    __syncthreads();
    int32_t before = lane < warp ? warp_sums[lane] : 0;
    before = __reduce_add_sync(FULL, before);
    if (threadIdx.x <= slices) slice[threadIdx.x] = before + pre - own;
    if (slices == RES_THREADS && threadIdx.x == RES_THREADS - 1) slice[slices] = before + pre;
    return __syncthreads_or(hub) != 0;
}

// Writes the sliced arcs (a warp per slice, the team's warps sharing them).
template <ResArcs SRC> __device__ void res_pack(const ResInst &a, const ResTeam &tm, const ResSmem &sm)
{
    const int lane = threadIdx.x & 31;
    const int32_t slices = (a.n + 31) >> 5;
    const int32_t *slice = &res_at<int32_t>(sm.slice);
    for (int32_t i = tm.rank * RES_WARPS + (threadIdx.x >> 5); i < slices; i += tm.size * RES_WARPS) {
        const int32_t v = i * 32 + lane, p = res_at<uint8_t>(sm.pairs + v), np = p == RES_HUB_MARK ? 0 : p, width = slice[i + 1] - slice[i];
        const int32_t beg = np ? __ldg(a.row_ptr + v) : 0, deg = np ? __ldg(a.row_ptr + v + 1) - beg : 0;
        for (int32_t j = 0; j < width; j++) {
            int2 x[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                // a distance of at most INF plus INF - 1 stays below 2^31
                x[q] = make_int2(v, SRC == ARCS_WIDE ? INF - 1 : (int32_t)RES_MAX_W - 1);
                if (2 * j + q < deg) x[q] = __ldcg(a.adj + beg + 2 * j + q);
            }
            const size_t at = (size_t)(slice[i] + j) * 32 + lane;
            if constexpr (SRC == ARCS_WIDE)
                reinterpret_cast<int4 *>(a.slices)[at] = make_int4(4 * x[0].x, x[0].y, 4 * x[1].x, x[1].y);
            else
                reinterpret_cast<uint2 *>(a.slices)[at] =
                    make_uint2((uint32_t)x[0].x << 2 | (uint32_t)x[0].y << 18, (uint32_t)x[1].x << 2 | (uint32_t)x[1].y << 18);
        }
    }
}

// The parts of `smem` bytes of dynamic shared memory, and the subset list in
// its part (xs: the first level's; lvl[kt + 1] entries).
__device__ __forceinline__ ResSmem res_layout(int32_t n, int32_t kt, int32_t smem, const uint32_t *xs, int32_t count)
{
    ResSmem sm;
    sm.xs = 0;
    sm.slice = ((2 << kt) + 15) / 16 * 16;
    sm.pairs = sm.slice + (4 * ((n + 31) / 32 + 1) + 15) / 16 * 16;
    sm.big = res_fixed_smem(n, kt);
    sm.end = smem;
    for (int32_t i = threadIdx.x; i < count; i += RES_THREADS)
        res_at<uint16_t>(sm.xs + 2 * i) = (uint16_t)__ldg(xs + i);
    return sm;
}

// Slices the arcs (narrow: every weight is below RES_MAX_W) and solves levels
// lo..hi; returns when the CTA's part is done or the team failed.
__device__ __forceinline__ void res_solve(const ResInst &a, ResTeam &tm, const ResSmem &sm, ResShared &sh, bool narrow,
                                          int32_t lo, int32_t hi)
{
    const bool has_hubs = res_slice_starts(a, sm, sh.hubs);
    const int64_t arc_bytes = (int64_t)res_i32(sm.slice + 4 * ((a.n + 31) >> 5)) * 32 * sizeof(uint2);
    // arcs in shared memory, unless they would keep records of RES_WIDE_SMEM rows out of it
    int64_t states = res_state_bytes(a.n, 1);
    if (a.want_rows * 4 >= RES_WIDE_SMEM * 3 && !has_hubs && res_wide_bytes(a.n, RES_WIDE_SMEM) <= sm.end - sm.big)
        states = max(states, res_wide_bytes(a.n, RES_WIDE_SMEM));
    const bool in_smem = narrow && arc_bytes + states <= sm.end - sm.big;
    if (narrow) res_pack<ARCS_PACKED>(a, tm, sm);
    else res_pack<ARCS_WIDE>(a, tm, sm);
    if (!res_barrier(tm, sh)) return;
    if (in_smem) res_levels<ARCS_SMEM>(a, tm, sm, sh, has_hubs, lo, hi);
    else if (narrow) res_levels<ARCS_PACKED>(a, tm, sm, sh, has_hubs, lo, hi);
    else res_levels<ARCS_WIDE>(a, tm, sm, sh, has_hubs, lo, hi);
}

}  // namespace emv
