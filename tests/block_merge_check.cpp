// block_merge_check.cpp -- checks the block merge plan of emv_plan.cpp for one
// k and split of the terminals (host only, built by tests/test_block_merge.py):
// replays every phase's units as the kernel walks them.  Staged positions and
// minima stay in bounds, every pair formed is a split of its subset, every
// unordered pair {Y, X \ Y} of every subset is formed, and without shared
// minima a unit's subsets belong to one warp of the phase.
#include "emv_plan.h"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <set>
#include <utility>

using namespace emv;

static std::vector<uint32_t> of_bits(int32_t low, int32_t a)
{
    std::vector<uint32_t> r;
    for (uint32_t s = 0; s < 1u << low; s++)
        if (__builtin_popcount(s) == a) r.push_back(s);
    return r;
}

int main(int argc, char **argv)
{
    const int32_t k = std::atoi(argv[1]), low = argc > 3 ? std::atoi(argv[3]) : BLOCK_LOW;
    const int64_t smem = std::atoll(argv[2]);
    std::vector<uint32_t> xs, data;
    std::vector<int64_t> off;
    subset_levels(k, xs, off);
    std::vector<HostBlockLevel> plan;
    plan_block_levels(k, low, xs, off, smem, data, plan);
    int levels = 0;
    auto fail = [&](const char *what, int m) {
        std::printf("FAIL k=%d m=%d: %s\n", k, m, what);
        return 1;
    };
    for (int32_t m = 3; m <= k; m++) {
        const HostBlockLevel &L = plan[(size_t)m];
        if (L.phases.empty()) continue;
        levels++;
        const int64_t x0 = off[(size_t)m], cnt = off[(size_t)m + 1] - x0;
        if (((L.split ? 2 : 1) * cnt + L.rows) * 128 > smem) return fail("shared memory", m);
        std::vector<std::set<uint32_t>> have((size_t)cnt);
        for (const HostBlockPhase &P : L.phases) {
            if (P.units_at % 4) return fail("alignment", m);
            if (P.ny + P.nz > L.rows) return fail("rows", m);
            std::vector<int> owner((size_t)cnt, -1);
            auto row = [&](int64_t i) { return xs[(size_t)(i < P.ny ? P.y0 + i : P.z0 + i - P.ny)]; };
            for (int w = 0; w < BLOCK_WARPS; w++)
                for (uint32_t u = data[P.warps_at + (size_t)w]; u < data[P.warps_at + (size_t)w + 1]; u++) {
                    const uint32_t *h = &data[P.units_at + 8 * u];
                    const int64_t acc = h[0] & 0xffffu;
                    const int32_t q = (int32_t)(h[0] >> 16);
                    if (q > low) return fail("bits", m);
                    const std::vector<uint32_t> qs = of_bits(low, q);
                    if (acc + (int64_t)qs.size() > cnt) return fail("minima", m);
                    for (size_t o = 0; o < qs.size(); o++) {
                        int &own = owner[(size_t)acc + o];
                        if (own >= 0 && own != w && !L.split) return fail("owner", m);
                        own = w;
                    }
                    const uint32_t *word = &data[P.words_at] + h[1];
                    for (int32_t a = 0; a <= q; a++) {
                        const uint32_t n2 = h[2 + a / 2], n = a % 2 ? n2 >> 16 : n2 & 0xffffu;
                        const std::vector<uint32_t> ya = of_bits(low, a), zc = of_bits(low, q - a);
                        for (uint32_t i = 0; i < n; i++, word++) {
                            const int64_t y0 = *word & 0xffffu, z0 = *word >> 16;
                            if (y0 + (int64_t)ya.size() > P.ny + P.nz || z0 + (int64_t)zc.size() > P.ny + P.nz)
                                return fail("staged position", m);
                            for (size_t y = 0; y < ya.size(); y++)
                                for (size_t z = 0; z < zc.size(); z++) {
                                    if (ya[y] & zc[z]) continue;
                                    const auto o = std::find(qs.begin(), qs.end(), ya[y] | zc[z]) - qs.begin();
                                    const uint32_t Y = row(y0 + (int64_t)y), Z = row(z0 + (int64_t)z);
                                    if ((Y & Z) || (Y | Z) != xs[(size_t)(x0 + acc + o)]) return fail("pair", m);
                                    have[(size_t)acc + (size_t)o].insert(std::min(Y, Z));
                                }
                        }
                    }
                }
        }
        for (int64_t i = 0; i < cnt; i++)
            if (have[(size_t)i].size() != (1u << (m - 1)) - 1) return fail("missing pairs", m);
    }
    std::printf("ok k=%d block_levels=%d\n", k, levels);
    return 0;
}
