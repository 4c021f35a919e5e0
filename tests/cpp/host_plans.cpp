// Checks of the host-side plans in pink_b200/csrc that need no GPU; prints what is wrong and returns 1, or returns 0.
#include "../../pink_b200/csrc/dot_plan.hpp"
#include "../../pink_b200/csrc/owners.hpp"

#include <chrono>
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

struct Map { std::vector<int16_t> at; bool hex; uint32_t dim0, dim1, dim2; };

static Map cartesian(uint32_t dim0, uint32_t dim1, uint32_t dim2)
{
    Map m{ {}, false, dim0, dim1, dim2 };
    for (uint32_t z = 0; z < dim2; ++z)
        for (uint32_t y = 0; y < dim0; ++y)
            for (uint32_t x = 0; x < dim1; ++x) for (uint32_t v : { x, y, z, 0u }) m.at.push_back((int16_t)v);
    return m;
}

static Map hexagonal(int dim)
{
    Map m{ {}, true, (uint32_t)dim, (uint32_t)dim, 1 };
    const int radius = (dim - 1) / 2;
    for (int r = -radius; r <= radius; ++r)
        for (int q = std::max(-radius, -radius - r); q <= std::min(radius, radius - r); ++q) for (int v : { q, r, 0, 0 }) m.at.push_back((int16_t)v);
    return m;
}

// Factor of every distance class: a Gaussian of the distance.
static std::vector<float> gaussian(const Map& m, double sigma)
{
    std::vector<float> lut;
    if (m.hex) for (uint32_t d = 0; d < m.dim0; ++d) lut.push_back((float)std::exp(-0.5 * d * d / (sigma * sigma)));
    else
        for (uint32_t z = 0; z < m.dim2; ++z)
            for (uint32_t y = 0; y < m.dim0; ++y)
                for (uint32_t x = 0; x < m.dim1; ++x) lut.push_back((float)std::exp(-0.5 * (x * x + y * y + z * z) / (sigma * sigma)));
    return lut;
}

// Most neurons of one block among those that a best matching unit's neighbourhood (factor above 1e-3) touches, over all units.
static uint32_t crowding(const std::vector<uint32_t>& owners, uint32_t blocks, uint32_t per_block, const NearNeurons& pairs, const float* lut,
                         uint32_t first, uint32_t stride, uint32_t neurons)
{
    uint32_t worst = 0;
    for (uint32_t unit = 0; unit < neurons; unit += 7)
        for (uint32_t b = 0; b < blocks; ++b) {
            uint32_t touched = 0;
            for (uint32_t j = 0; j < per_block; ++j) {
                const uint32_t o = owners[(size_t)b * per_block + j];
                if (o != ~0u && std::fabs(lut[pairs.distance_class(unit, first + o * stride)]) > 1e-3f) ++touched;
            }
            worst = std::max(worst, touched);
        }
    return worst;
}

static double seconds()
{
    return std::chrono::duration<double>(std::chrono::steady_clock::now().time_since_epoch()).count();
}

static void check_owners()
{
    const Map maps[] = { cartesian(10, 10, 1), cartesian(1, 300, 1), cartesian(300, 1, 1), cartesian(40, 40, 1), cartesian(6, 7, 8), hexagonal(3),
                         hexagonal(21), hexagonal(61) };
    for (const Map& map : maps)
        for (double sigma : { 0.3, 1.1, 3.0, 100.0 })
            for (uint32_t stride : { 1u, 3u }) {
                const uint32_t neurons = (uint32_t)map.at.size() / 4, first = stride - 1, n = neurons > first ? (neurons - first + stride - 1) / stride : 0u;
                const uint32_t blocks = std::min(148u, n), per_block = (n + blocks - 1) / blocks;
                std::vector<float> lut = gaussian(map, sigma);
                const NearNeurons near(map.at.data(), neurons, map.hex, map.dim0, map.dim1, lut.data(), (uint32_t)lut.size(), first, stride);
                auto all = [&](uint32_t i, auto add) {
                    for (uint32_t m = 0; m < i; ++m) add(m, lut[near.distance_class(first + i * stride, first + m * stride)]);
                };
                // the pairs that are left out are the ones with (almost) no factor, and none comes twice
                std::vector<uint32_t> seen(n, ~0u);
                for (uint32_t i = 0; i < n; ++i) {
                    near(i, [&](uint32_t m, float f) {
                        CHECK(m < i && seen[m] != i, "%u neurons: pair %u %u", neurons, i, m);
                        CHECK(f == lut[near.distance_class(first + i * stride, first + m * stride)], "%u neurons: pair %u %u", neurons, i, m);
                        if (m < i) seen[m] = i;
                    });
                    all(i, [&](uint32_t m, float f) { CHECK(seen[m] == i || f <= 1.01e-8f, "%u neurons: pair %u %u left out", neurons, i, m); });
                }
                std::vector<uint32_t> owners((size_t)blocks * per_block), full(owners.size()), times(n, 0);
                assign_owners(n, blocks, per_block, owners.data(), near);
                assign_owners(n, blocks, per_block, full.data(), all);
                for (uint32_t o : owners) if (o != ~0u) { CHECK(o < n, "owner of %u", o); if (o < n) ++times[o]; }
                for (uint32_t i = 0; i < n; ++i) CHECK(times[i] == 1, "%u neurons: %u owned %u times", neurons, i, times[i]);
                // as even as with all pairs
                CHECK(crowding(owners, blocks, per_block, near, lut.data(), first, stride, neurons)
                      <= crowding(full, blocks, per_block, near, lut.data(), first, stride, neurons) + 1, "%u neurons, sigma %g", neurons, sigma);
            }
    // setting a neighbourhood of a large map is quick
    const Map map = hexagonal(61);
    const std::vector<float> lut = gaussian(map, 1.1);
    const uint32_t n = (uint32_t)map.at.size() / 4, per_block = (n + 147) / 148;
    std::vector<uint32_t> owners(148 * per_block);
    double near_s = 1e9, all_s = 1e9;
    for (int k = 0; k < 5; ++k) {
        const double t0 = seconds();
        const NearNeurons near(map.at.data(), n, true, 61, 61, lut.data(), (uint32_t)lut.size(), 0, 1);
        assign_owners(n, 148, per_block, owners.data(), near);
        const double t1 = seconds();
        assign_owners(n, 148, per_block, owners.data(), [&](uint32_t i, auto add) { for (uint32_t m = 0; m < i; ++m) add(m, lut[near.distance_class(i, m)]); });
        near_s = std::min(near_s, t1 - t0);
        all_s = std::min(all_s, seconds() - t1);
    }
    CHECK(near_s < 0.5 * all_s, "%.2f ms against %.2f of all pairs", near_s * 1e3, all_s * 1e3);
    std::printf("owners of 2791 neurons: %.2f ms, all pairs %.2f ms\n", near_s * 1e3, all_s * 1e3);
}

int main()
{
    check_dot_plans();
    check_owners();
    return failures != 0;
}
