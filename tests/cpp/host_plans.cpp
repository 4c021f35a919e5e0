// Checks of the host-side plans in pink_b200/csrc that need no GPU; prints what is wrong and returns 1, or returns 0.
#include "../../pink_b200/csrc/dot_plan.hpp"

#include <cstdio>

using namespace pinkb;

static int failures = 0;
#define CHECK(cond, ...) do { if (!(cond)) { ++failures; std::printf("%s: ", #cond); std::printf(__VA_ARGS__); std::printf("\n"); } } while (0)

// The cheapest split by trying every tile count and every number of ranges.
static uint64_t cheapest(uint32_t n, uint32_t T, uint32_t slices, const DotPlan& p, uint32_t max_splits, uint32_t sms, uint64_t* of_plan)
{
    const uint32_t rows = p.swap ? T : n, columns = p.swap ? n : T;
    uint32_t m_tiles = (rows + 127) / 128;
    if (p.pair) m_tiles = (m_tiles + 1) / 2 * 2;
    uint64_t lowest = ~0ull;
    *of_plan = 0;
    for (uint32_t count = (columns + 255) / 256; count <= std::max((columns + 255) / 256, columns / 32); ++count) {
        const uint32_t width = std::min(256u, ((columns + count - 1) / count + 15) / 16 * 16), tiles = (columns + width - 1) / width;
        for (uint32_t s = 1; s <= max_splits; ++s) {
            const uint32_t len = (slices + s - 1) / s;
            if (s > 1 && (2 * s > slices || (s - 1) * len >= slices)) continue;
            const uint64_t waves = ((uint64_t)m_tiles * tiles * s + sms - 1) / sms;
            const uint64_t cost = waves * len * (128 + (p.pair ? width / 2 : width)) * 128 * 2 + (uint64_t)s * n * T * 8 / sms;
            lowest = std::min(lowest, cost);
            if (width == p.n_tile && s == p.splits) *of_plan = cost;
        }
    }
    return lowest;
}

static void check_dot_plans()
{
    for (uint32_t n : { 1u, 15u, 100u, 129u, 257u, 400u, 2791u, 9000u })
        for (uint32_t T : { 1u, 8u, 33u, 720u, 1440u, 12800u })
            for (uint32_t slices : { 1u, 2u, 3u, 7u, 32u, 65u, 259u })
                for (uint32_t max_splits : { 1u, 3u, 16u })
                    for (bool single : { false, true }) {
                        const DotPlan p = plan_dots(n, T, slices, single, max_splits, 148);
                        const uint32_t rows = p.swap ? T : n;
                        uint64_t cost = 0;
                        const uint64_t lowest = cheapest(n, T, slices, p, max_splits, 148, &cost);
                        CHECK(cost == lowest, "n %u T %u slices %u splits %u: %llu, lowest %llu", n, T, slices, max_splits,
                              (unsigned long long)cost, (unsigned long long)lowest);
                        CHECK(p.pair == (rows > 128 && !single), "n %u T %u", n, T);
                        CHECK(p.n_tile >= 16 && p.n_tile <= 256 && p.n_tile % 16 == 0, "n %u T %u: %u columns", n, T, p.n_tile);
                        CHECK(p.splits >= 1 && p.splits <= max_splits, "n %u T %u: %u ranges", n, T, p.splits);
                        // the ranges cover K, none is empty, all but the last have at least two slices
                        CHECK(p.splits * p.kb_split >= slices && (p.splits - 1) * p.kb_split < slices, "slices %u: %u x %u", slices, p.splits, p.kb_split);
                        CHECK(p.splits == 1 || p.kb_split >= 2, "slices %u: %u x %u", slices, p.splits, p.kb_split);
                    }
}

int main()
{
    check_dot_plans();
    return failures != 0;
}
