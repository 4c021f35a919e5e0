// Which block of the persistent training kernel rewrites which neuron (host code only, so that it can be checked without a GPU).
#ifndef PINK_B200_OWNERS_HPP
#define PINK_B200_OWNERS_HPP
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <vector>

namespace pinkb {

// Greedy assignment in index order: a neuron goes to the block (with room left) whose neurons so far are
// farthest from it, closeness measured by the update factors themselves -- the factor of (i, m) is large exactly when
// i and m are rewritten together.  The neighbourhood of any best matching unit then spreads over the
// blocks almost evenly (measured on a hexagonal map of 2791 neurons, sigma 3: at most 5-7 neurons of a
// block among the ~700-1000 neurons an image rewrites, against 7-9 for a round-robin assignment).
// owners[block * per_block + slot] = local neuron, ~0u where a slot stays empty.  near(i, add) calls add(m, closeness) for
// local neurons m < i; pairs that it leaves out count as far apart.
template <class Near>
void assign_owners(uint32_t count, uint32_t blocks, uint32_t per_block, uint32_t* owners, const Near& near)
{
    std::fill(owners, owners + (size_t)blocks * per_block, ~0u);
    std::vector<uint32_t> color(count), load(blocks, 0);
    std::vector<double> score(blocks);
    for (uint32_t i = 0; i < count; ++i) {
        std::fill(score.begin(), score.end(), 0.0);
        near(i, [&](uint32_t m, float closeness) { score[color[m]] += std::fabs((double)closeness); });
        uint32_t best = blocks;
        for (uint32_t c = 0; c < blocks; ++c) {
            if (load[c] >= per_block) continue;
            if (best == blocks || score[c] < score[best] || (score[c] == score[best] && load[c] < load[best])) best = c;
        }
        color[i] = best;
        owners[(size_t)best * per_block + load[best]++] = i;
    }
}

// The pairs of a map whose update factor depends on the distance class of the two neurons, that is on the difference of their
// coordinates: one table of it, walked along the rows of neurons within reach (2791 neurons, sigma 1.1 and 3: 1.4 and 2.7 ms; all
// pairs, classified one by one: 12 ms, in every call that sets a neighbourhood).  Two neurons are rewritten together when
// some unit is near both, so the reach is twice as far as any factor goes that can change a value (1e-8 of the
// largest).  (Once the largest distance with a factor above 1e-4 is
// too short: 331 neurons then trained 4 % slower.)
class NearNeurons
{
public:
    // coords: x, y, z, 0 of every neuron of the map; lut: factor of every distance class, as pink_b200_distance_classes numbers
    // them; local neuron j is neuron first + j * stride
    NearNeurons(const int16_t* coords, uint32_t neurons, bool hexagonal, uint32_t dim0, uint32_t dim1, const float* lut, uint32_t classes,
                uint32_t first, uint32_t stride)
        : at_(coords), hex_(hexagonal), dim0_(dim0), dim1_(dim1), first_(first), stride_(stride)
    {
        for (uint32_t i = 0; i < neurons; ++i) {
            if (i == 0 || x(i) != x(i - 1) + 1 || y(i) != y(i - 1) || z(i) != z(i - 1)) rows_.push_back({ i, 0 });
            rows_.back().length += 1;
        }
        float most = 0.0f;
        for (uint32_t c = 0; c < classes; ++c) most = std::max(most, std::fabs(lut[c]));
        int far[3] = { 0, 0, 0 };
        for (uint32_t c = 0; c < classes; ++c) {
            if (!(std::fabs(lut[c]) > 1e-8f * most)) continue;
            far[0] = std::max<int>(far[0], hex_ ? c : c % dim1);
            far[1] = std::max<int>(far[1], hex_ ? c : c / dim1 % dim0);
            far[2] = std::max<int>(far[2], hex_ ? 0 : c / dim1 / dim0);
        }
        int lo[3] = { x(0), y(0), z(0) }, hi[3] = { x(0), y(0), z(0) };
        for (uint32_t i = 0; i < neurons; ++i)
            for (int a = 0; a < 3; ++a) { lo[a] = std::min<int>(lo[a], at_[4 * (size_t)i + a]); hi[a] = std::max<int>(hi[a], at_[4 * (size_t)i + a]); }
        for (int a = 0; a < 3; ++a) { reach_[a] = std::min(2 * far[a], hi[a] - lo[a]); width_[a] = 2 * (size_t)reach_[a] + 1; }
        factor_.resize(width_[0] * width_[1] * width_[2]);
        size_t k = 0;
        for (int dz = -reach_[2]; dz <= reach_[2]; ++dz)
            for (int dy = -reach_[1]; dy <= reach_[1]; ++dy)
                for (int dx = -reach_[0]; dx <= reach_[0]; ++dx) {
                    const uint32_t c = class_of(dx, dy, dz);
                    factor_[k++] = c < classes ? lut[c] : 0.0f;        // (a corner of the box may lie outside a hexagon)
                }
    }

    uint32_t distance_class(uint32_t i, uint32_t m) const { return class_of(x(i) - x(m), y(i) - y(m), z(i) - z(m)); }

    template <class Add>
    void operator()(uint32_t local, const Add& add) const
    {
        const uint32_t i = first_ + local * stride_;
        for (const Row& r : rows_) {
            if (r.start >= i) break;
            const int dy = y(r.start) - y(i), dz = z(r.start) - z(i), dx = x(r.start) - x(i);
            if (std::abs(dy) > reach_[1] || std::abs(dz) > reach_[2]) continue;
            // this shard's neurons among start + [lo, hi), those within reach along x and before neuron i
            const int64_t lo = std::max(0, -reach_[0] - dx), hi = std::min<int64_t>(std::min<int64_t>(r.length, (int64_t)reach_[0] - dx + 1), (int64_t)i - r.start);
            int64_t m = (int64_t)r.start + lo <= first_ ? 0 : ((int64_t)r.start + lo - first_ + stride_ - 1) / stride_;
            // (neuron start + k lies at factor_[row + k]; row alone may point in front of the table)
            const int64_t row = ((int64_t)(dz + reach_[2]) * (int64_t)width_[1] + (dy + reach_[1])) * (int64_t)width_[0] + reach_[0] + dx;
            for (int64_t k = (int64_t)first_ + m * stride_ - r.start; k < hi; k += stride_, ++m) add((uint32_t)m, factor_[(size_t)(row + k)]);
        }
    }

private:
    struct Row { uint32_t start, length; };      // neurons start, start + 1, .. lie side by side in x
    int x(uint32_t i) const { return at_[4 * (size_t)i]; }
    int y(uint32_t i) const { return at_[4 * (size_t)i + 1]; }
    int z(uint32_t i) const { return at_[4 * (size_t)i + 2]; }
    uint32_t class_of(int dx, int dy, int dz) const
    {
        if (hex_) return (uint32_t)std::max(std::max(std::abs(dx), std::abs(dy)), std::abs(dx + dy));
        return ((uint32_t)std::abs(dz) * dim0_ + (uint32_t)std::abs(dy)) * dim1_ + (uint32_t)std::abs(dx);
    }
    const int16_t* at_;
    bool hex_;
    uint32_t dim0_, dim1_, first_, stride_;
    int reach_[3];
    size_t width_[3];
    std::vector<float> factor_;                  // by dz, dy, dx, each from -reach_ to reach_
    std::vector<Row> rows_;
};

} // namespace pinkb
#endif
