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
constexpr int RES_HUB = 64;              // a vertex of more arcs is walked by a whole warp
constexpr uint8_t RES_HUB_MARK = 255;    // its arc pairs in ResSmem::pairs
constexpr uint32_t RES_MAX_W = 1u << 14; // packed arcs hold smaller weights
constexpr float RES_PULL_SHARE = 0.2f;   // a round after one that changed more of the states pulls
constexpr uint32_t RES_SPIN_LIMIT = 1u << 22;  // polls of an L2 word, over a second in all
constexpr int RES_ACC_WORDS = 2 * RES_THREADS;  // merge minima of a level with at most half as many tasks as threads

// Control and result words of one launch (zeroed before it).
struct ResOut {
    uint32_t bar[32];        // arrivals of the grid barrier, on a line of its own
    uint32_t err;            // EMV_DEV_* bits
    uint32_t unreached;      // a level-1 closure left a vertex without a value
    uint32_t hubs;           // a vertex has more than RES_HUB arcs
    uint32_t rounds;         // pull sweeps and push rounds, summed over the CTAs' chunks
    GraphScan scan;
    unsigned long long ns[3];  // level 1, merges, relaxations (CTA 0's view)
    int32_t cost;            // d[C][t_{k-1}]
    int32_t terms[EMV_MAX_K];
};

struct ResArgs {
    const int32_t *row_ptr, *col, *w;  // the CSR as given
    int2 *adj;                // (head, weight) arcs (written here; read for hubs and by the traceback)
    void *slices;             // sliced arcs (written here)
    int32_t *table;           // 2^kt rows of stride ld
    const uint32_t *xs;       // subsets by level
    ResOut *out;
    int64_t ld, arcs;
    int32_t n, k, kt;
    int32_t check;            // leave after the CSR check found a fault
    int32_t vec;              // table rows are 16-byte aligned
    int32_t want_rows;        // rows of the widest level's largest share
    int32_t mw;               // vertices of a merge block (multiple of 4)
    int32_t smem;             // dynamic shared memory
    int32_t max_rounds;
    uint32_t inv_slices;      // ceil(2^32 / slices), for slices > 1
    int32_t xs_off[RES_KMAX + 2];
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

// Records an error and makes every CTA leave at its next barrier.
__device__ __forceinline__ void res_fail(ResOut *out, uint32_t err, int *s_ok)
{
    atomicOr(&out->err, err);
    atomicOr(out->bar, RES_FAILED);
    *(volatile int *)s_ok = 0;
}

// Barrier over the grid's CTAs (all resident: a cooperative launch, or one
// CTA).  Arrivals only count up, so no word is reset.  Bounded: a CTA that
// waits longer than RES_SPIN_LIMIT polls records the error; every CTA leaves
// when it sees one (*s_ok is 1 until then).
__device__ __forceinline__ bool res_barrier(ResOut *out, uint32_t &epoch, int *s_ok)
{
    __syncthreads();
    epoch++;
    if (gridDim.x > 1) {
        if (threadIdx.x == 0) {
            const uint32_t target = epoch * gridDim.x;
            uint32_t spins = 0, seen;
            __threadfence();
            atomicAdd(out->bar, 1u);
            for (;;) {
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(out->bar) : "memory");
                if ((seen & RES_FAILED) || (seen & ~RES_FAILED) >= target) break;
                if (++spins > RES_SPIN_LIMIT) {
                    res_fail(out, EMV_DEV_BARRIER_TIMEOUT, s_ok);
                    break;
                }
            }
            if (seen & RES_FAILED) *(volatile int *)s_ok = 0;
        }
        __syncthreads();
    }
    return *(volatile int *)s_ok != 0;
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
        a.x = min(a.x, y.x + z.x);
        a.y = min(a.y, y.y + z.y);
        a.z = min(a.z, y.z + z.z);
        a.w = min(a.w, y.w + z.w);
        sub = (sub - rest) & rest;
    }
    return a;
}

// Bytes of the merge's staged rows and of the minima of split pair lists.
__host__ __device__ inline int32_t res_merge_bytes(int32_t mw, int32_t kt) { return ((4 * mw) << kt) + 4 * RES_ACC_WORDS; }

// Merge of level m for this CTA's vertex blocks, in the last res_merge_bytes
// of the shared memory: 2^kt rows of mw words (row Y at Y * mw) and, after
// them, the minima of split pair lists.
__device__ void res_merge(const ResArgs &a, const ResSmem &sm, int32_t m, const int32_t *terms)
{
    uint32_t *S = &res_at<uint32_t>(sm.end - res_merge_bytes(a.mw, a.kt));
    const uint16_t *xs = &res_at<uint16_t>(sm.xs);
    const int32_t n = a.n, W = a.mw, Q = W / 4, tid = threadIdx.x;
    const int32_t nlow = a.xs_off[m], cnt = a.xs_off[m + 1] - nlow;
    const uint32_t npairs = (1u << (m - 1)) - 1;
    const int32_t tasks = cnt * Q;
    int32_t parts = 1;
    while (tasks * parts * 2 <= RES_THREADS && (uint32_t)parts * 2 <= npairs) parts *= 2;
    uint32_t *acc = S + ((size_t)W << a.kt);
    const uint4 *S4 = reinterpret_cast<const uint4 *>(S);
    for (int32_t v0 = blockIdx.x * W; v0 < n; v0 += gridDim.x * W) {
        bool has_term = false;
        for (int32_t t = 0; t < a.kt; t++) has_term |= terms[t] >= v0 && terms[t] < v0 + W;
        for (int32_t i = tid; i < nlow * Q; i += RES_THREADS) {
            const int32_t r = i / Q, q = i - r * Q;
            const uint32_t Y = xs[r];
            const int32_t v = v0 + 4 * q;
            const int32_t *src = a.table + (int64_t)Y * a.ld + v;
            int4 x;
            if (a.vec && v + 4 <= n) x = __ldcg(reinterpret_cast<const int4 *>(src));
            else
                x = make_int4(v < n ? __ldcg(src) : INF, v + 1 < n ? __ldcg(src + 1) : INF,
                              v + 2 < n ? __ldcg(src + 2) : INF, v + 3 < n ? __ldcg(src + 3) : INF);
            reinterpret_cast<int4 *>(S)[Y * Q + q] = x;
        }
        if (parts > 1)
            for (int32_t i = tid; i < cnt * W; i += RES_THREADS) acc[i] = (uint32_t)INF;
        __syncthreads();
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
            uint4 r = parts > 1 ? reinterpret_cast<const uint4 *>(acc)[t] : res_pairs(S4 + q, Q, X, 0, npairs);
            const int32_t v = v0 + 4 * q;
            if (has_term)  // arcs of the virtual source (R:2099-2107)
                for (uint32_t bits = X; bits; bits &= bits - 1) {
                    const int ti = __ffs(bits) - 1, d = terms[ti] - v;
                    if (d < 0 || d >= 4) continue;
                    const uint32_t o = S[(X ^ (1u << ti)) * W + 4 * q + d];
                    if (d == 0) r.x = o;
                    else if (d == 1) r.y = o;
                    else if (d == 2) r.z = o;
                    else r.w = o;
                }
            int32_t *dst = a.table + (int64_t)X * a.ld + v;
            if (a.vec && v + 4 <= n) *reinterpret_cast<uint4 *>(dst) = r;
            else {
                if (v < n) dst[0] = (int32_t)r.x;
                if (v + 1 < n) dst[1] = (int32_t)r.y;
                if (v + 2 < n) dst[2] = (int32_t)r.z;
                if (v + 3 < n) dst[3] = (int32_t)r.w;
            }
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
// of more than RES_HUB arcs have no pairs here and are read from adj.
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
        return min(min(acc, p + w[0]), q + w[1]);
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

// wd / slices for a word index below 2^16.
__device__ __forceinline__ int32_t res_div(const ResArgs &a, int32_t wd, int32_t slices)
{
    return slices == 1 ? wd : (int32_t)__umulhi((uint32_t)wd, a.inv_slices);
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
// Graphs with vertices of more than RES_HUB arcs list those apart (from the
// far end of the warp's part), and after a barrier all warps share them, a
// warp per vertex: one warp would otherwise walk all hubs of its run.
// Returns false when max_rounds ran out; `rounds` counts barriers passed.
template <ResArcs SRC>
__device__ bool res_close(const ResArgs &a, const ResGraph<SRC> &g, bool has_hubs, int32_t R, bool level1, int32_t d,
                          int32_t list, int32_t bm, int32_t *hub_cnt, int32_t &rounds)
{
    using G = ResGraph<SRC>;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1;
    const int32_t slices = (a.n + 31) >> 5, words = R * slices;
    auto row_of = [&](int32_t wd) -> int32_t { return R == 1 ? 0 : res_div(a, wd, slices); };
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
                if (++rounds > a.max_rounds) return false;
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
    // threads with a change among their `per` states when half of all states change
    float same = 1.0f;
    for (int32_t i = 0; i < per && i < 16; i++) same *= 1.0f - RES_PULL_SHARE;
    const int many = (int)(RES_THREADS * (1.0f - same));
    bool pull = !level1, any = true;
    for (;;) {
        if (++rounds > a.max_rounds) return false;
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

// Relaxation of this CTA's rows of level m, at most `rows` at a time, from
// byte offset dyn of the shared memory.
template <ResArcs SRC>
__device__ void res_relax(const ResArgs &a, const ResGraph<SRC> &g, const ResSmem &sm, bool has_hubs, int32_t m,
                          int32_t dyn, int32_t rows, const int32_t *terms, int32_t *hub_cnt, int *s_ok)
{
    const int32_t n = a.n, slices = (n + 31) >> 5, np = slices * 32, cnt = a.xs_off[m + 1] - a.xs_off[m];
    const int32_t rb = (int32_t)((int64_t)cnt * blockIdx.x / gridDim.x),
                  re = (int32_t)((int64_t)cnt * (blockIdx.x + 1) / gridDim.x);
    const uint32_t C = (1u << (a.k - 1)) - 1;
    uint32_t rounds = 0;
    for (int32_t r0 = rb; r0 < re; r0 += rows) {
        const int32_t R = min(rows, re - r0), words = R * slices;
        const uint16_t *xs = &res_at<uint16_t>(sm.xs) + a.xs_off[m] + r0;
        int32_t *d = &res_at<int32_t>(dyn);
        uint32_t *bm = &res_at<uint32_t>(dyn + words * 128);
        // four states of a row at a time
        auto quads = [&](auto f) {
#pragma unroll 2
            for (int32_t i = threadIdx.x; i < words * 8; i += RES_THREADS) {
                const int32_t r = R == 1 ? 0 : res_div(a, i >> 3, slices);
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
        const bool ok = res_close<SRC>(a, g, has_hubs, R, m == 1, dyn, dyn + words * 132, dyn + words * 128, hub_cnt, did);
        rounds += did;
        if (!ok && threadIdx.x == 0) res_fail(a.out, EMV_DEV_SWEEP_LIMIT, s_ok);
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
        if (m == 1 && unreached) a.out->unreached = 1;
        if (m == a.k - 1)
            for (int32_t r = threadIdx.x; r < R; r += RES_THREADS)
                if (xs[r] == C) a.out->cost = d[r * np + terms[a.k - 1]];
        __syncthreads();
        if (!ok) break;
    }
    if (threadIdx.x == 0 && rounds) atomicAdd(&a.out->rounds, rounds);
}

// Levels 1..kt.  Arcs that the closures keep in shared memory are copied there
// again for every level as far as the merge's staging overlaps them, between
// the merge and the barrier after it.
template <ResArcs SRC>
__device__ void res_levels(const ResArgs &a, const ResSmem &sm, bool has_hubs, const int32_t *terms, int32_t *hub_cnt,
                           uint32_t &epoch, int *s_ok)
{
    using T = typename ResElem<SRC>::T;
    const bool clock = blockIdx.x == 0 && threadIdx.x == 0;
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
    auto load_arcs = [&](int32_t from) {
        for (int32_t i = from + threadIdx.x * 16; i < arc_bytes; i += RES_THREADS * 16)
            cp_async16(&res_at<int4>(sm.big + i), (const char *)a.slices + i);
    };
    for (int32_t m = 1; m <= a.kt; m++) {
        if (m > 1) res_merge(a, sm, m, terms);
        load_arcs(m > 1 ? keep : 0);
        if (m > 1) {
            if (!res_barrier(a.out, epoch, s_ok)) break;
            if (clock) {
                const unsigned long long t = res_now();
                a.out->ns[1] += t - t0;
                t0 = t;
            }
        }
        cp_async_wait_all();  // made visible to the CTA by the barrier before the closure
        res_relax<SRC>(a, g, sm, has_hubs, m, dyn, rows, terms, hub_cnt, s_ok);
        if (m < a.kt && !res_barrier(a.out, epoch, s_ok)) break;
        if (clock) {
            const unsigned long long t = res_now();
            a.out->ns[m == 1 ? 0 : 2] += t - t0;
            t0 = t;
        }
    }
    cp_async_wait_all();
}

// Widths of the slices in arc pairs, their prefix sums (sm.slice) and the
// pairs of every vertex; needs at most RES_THREADS slices.
__device__ void res_slice_starts(const ResArgs &a, const ResSmem &sm, int32_t *warp_sums)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int32_t slices = (a.n + 31) >> 5;
    int32_t *slice = &res_at<int32_t>(sm.slice);
    for (int32_t i = warp; i < slices; i += RES_WARPS) {
        const int32_t v = i * 32 + lane;
        const int32_t deg = v < a.n ? __ldg(a.row_ptr + v + 1) - __ldg(a.row_ptr + v) : 0;
        const int32_t np = deg > RES_HUB ? 0 : (deg + 1) / 2;
        res_at<uint8_t>(sm.pairs + v) = deg > RES_HUB ? RES_HUB_MARK : (uint8_t)np;
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
    __syncthreads();
}

// Writes the sliced arcs (a warp per slice, the grid's warps sharing them).
template <ResArcs SRC> __device__ void res_pack(const ResArgs &a, const ResSmem &sm)
{
    const int lane = threadIdx.x & 31;
    const int32_t slices = (a.n + 31) >> 5;
    const int32_t *slice = &res_at<int32_t>(sm.slice);
    for (int32_t i = blockIdx.x * RES_WARPS + (threadIdx.x >> 5); i < slices; i += gridDim.x * RES_WARPS) {
        const int32_t v = i * 32 + lane, p = res_at<uint8_t>(sm.pairs + v), np = p == RES_HUB_MARK ? 0 : p, width = slice[i + 1] - slice[i];
        const int32_t beg = np ? __ldg(a.row_ptr + v) : 0, deg = np ? __ldg(a.row_ptr + v + 1) - beg : 0;
        for (int32_t j = 0; j < width; j++) {
            int32_t h[2], w[2];
#pragma unroll
            for (int q = 0; q < 2; q++) {
                const bool ok = 2 * j + q < deg;
                h[q] = ok ? __ldg(a.col + beg + 2 * j + q) : v;
                // a distance of at most INF plus INF - 1 stays below 2^31
                w[q] = ok ? __ldg(a.w + beg + 2 * j + q) : SRC == ARCS_WIDE ? INF - 1 : (int32_t)RES_MAX_W - 1;
            }
            const size_t at = (size_t)(slice[i] + j) * 32 + lane;
            if constexpr (SRC == ARCS_WIDE)
                reinterpret_cast<int4 *>(a.slices)[at] = make_int4(4 * h[0], w[0], 4 * h[1], w[1]);
            else
                reinterpret_cast<uint2 *>(a.slices)[at] =
                    make_uint2((uint32_t)h[0] << 2 | (uint32_t)w[0] << 18, (uint32_t)h[1] << 2 | (uint32_t)w[1] << 18);
        }
    }
}

// The whole solve: CSR check and arc slices, then levels 1..kt.
__global__ void __launch_bounds__(RES_THREADS, 1) k_resident(ResArgs a)
{
    __shared__ int s_ok;
    __shared__ int32_t s_terms[EMV_MAX_K];
    __shared__ int32_t s_hubs[RES_WARPS];
    uint32_t epoch = 0;
    const int32_t slices = (a.n + 31) >> 5;
    const int64_t first = (int64_t)blockIdx.x * RES_THREADS + threadIdx.x, stride = (int64_t)gridDim.x * RES_THREADS;
    ResSmem sm;
    sm.xs = 0;
    sm.slice = ((2 << a.kt) + 15) / 16 * 16;
    sm.pairs = sm.slice + (4 * (slices + 1) + 15) / 16 * 16;
    sm.big = res_fixed_smem(a.n, a.kt);
    sm.end = a.smem;
    if (threadIdx.x == 0) s_ok = 1;  // before the barrier that first reads it
    for (int32_t i = threadIdx.x; i < a.xs_off[a.kt + 1]; i += RES_THREADS)
        res_at<uint16_t>(sm.xs + 2 * i) = (uint16_t)__ldg(a.xs + i);
    if (threadIdx.x < EMV_MAX_K) s_terms[threadIdx.x] = a.terms[threadIdx.x];
    if (blockIdx.x == 0 && threadIdx.x < a.k) a.out->terms[threadIdx.x] = a.terms[threadIdx.x];
    scan_csr(a.row_ptr, a.n, a.col, a.w, a.adj, a.arcs, &a.out->scan);
    bool hub = false;
    for (int64_t v = first; v < a.n; v += stride) {
        a.table[v] = INF;  // row 0 (R:2243-2259)
        hub |= a.row_ptr[v + 1] - a.row_ptr[v] > RES_HUB;
    }
    if (hub) a.out->hubs = 1;
    if (!res_barrier(a.out, epoch, &s_ok)) return;
    const uint32_t bad = __ldcg(&a.out->scan.bad), maxw = __ldcg(&a.out->scan.maxw);
    if (a.check) {  // the host reads the same words and names the fault
        if (bad) return;
        const long long bound =
            min((long long)(a.n - 1) * (long long)maxw, (long long)(__ldcg(&a.out->scan.sumw) / 2));
        if (bound >= INF) return;
    }
    const bool has_hubs = __ldcg(&a.out->hubs) != 0;
    res_slice_starts(a, sm, s_hubs);
    const int64_t arc_bytes = (int64_t)res_i32(sm.slice + 4 * slices) * 32 * sizeof(uint2);
    const bool narrow = maxw < RES_MAX_W && !(bad & SCAN_BAD_WEIGHT);
    const bool in_smem = narrow && arc_bytes + res_state_bytes(a.n, 1) <= sm.end - sm.big;
    if (narrow) res_pack<ARCS_PACKED>(a, sm);
    else res_pack<ARCS_WIDE>(a, sm);
    if (!res_barrier(a.out, epoch, &s_ok)) return;
    if (in_smem) res_levels<ARCS_SMEM>(a, sm, has_hubs, s_terms, s_hubs, epoch, &s_ok);
    else if (narrow) res_levels<ARCS_PACKED>(a, sm, has_hubs, s_terms, s_hubs, epoch, &s_ok);
    else res_levels<ARCS_WIDE>(a, sm, has_hubs, s_terms, s_hubs, epoch, &s_ok);
}

}  // namespace emv
