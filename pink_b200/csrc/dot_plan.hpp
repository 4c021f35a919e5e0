// How the tensor-core estimate of one image's float32 distances is split over the GPU (training; host code only, so that it
// can be checked without a GPU).
#ifndef PINK_B200_DOT_PLAN_HPP
#define PINK_B200_DOT_PLAN_HPP
#include <algorithm>
#include <cstdint>

namespace pinkb {

constexpr uint32_t kMaxDotSplits = 16;

struct DotPlan
{
    uint32_t swap;               // the transforms are the tile rows (M side), the neurons its columns
    uint32_t pair;               // two CTAs share a tile pair of 256 rows
    uint32_t n_tile;             // tile columns
    uint32_t splits, kb_split;   // ranges of K, and 128-byte slices of K per range; 0 splits: not planned yet
};

// Orientation of the estimate: the one whose padded tile grid (rows to 128, or 256 for block pairs; columns to balanced tiles
// of at most 256, multiples of 16) computes fewer pairs that do not exist.
inline bool estimate_swapped(uint32_t n, uint32_t T)
{
    auto padded = [](uint32_t rows, uint32_t columns) -> uint64_t {
        const uint32_t mp = rows > 128 ? (rows + 255) / 256 * 256 : 128;
        const uint32_t tiles = (columns + 255) / 256, nt = (((columns + tiles - 1) / tiles) + 15) & ~15u;
        return (uint64_t)mp * ((columns + nt - 1) / nt) * nt;
    };
    return padded(T, n) < padded(n, T);
}

// One image's tiles alone leave most SMs idle or, narrow, make every SM pull the whole row tile (400 x 720 x 4096:
// 54 blocks of 5 MB, 40.6 us; with K split 16.6).  So K is split too: the choice of column tiles and K ranges that
// moves the fewest bytes per SM, operand slices in, partial products out and in again.  Every range but the last has at least
// two slices.  The choice depends on the context only and is made once: the search takes about as long on the host as a
// launch (two operand planes of n x `slices` and T x `slices` slices, `sms` SMs).
inline DotPlan plan_dots(uint32_t n, uint32_t T, uint32_t slices, bool single_cta, uint32_t max_splits, uint32_t sms)
{
    constexpr uint32_t row_tile = 128, slice_bytes = 128, planes = 2, max_n = 256;
    DotPlan best{};
    best.swap = estimate_swapped(n, T);
    const uint32_t rows = best.swap ? T : n, columns = best.swap ? n : T;
    best.pair = rows > row_tile && !single_cta;
    uint32_t m_tiles = (rows + row_tile - 1) / row_tile;
    if (best.pair) m_tiles = (m_tiles + 1) & ~1u;
    const uint64_t wave = sms ? sms : 148;
    max_splits = std::min(std::max(max_splits, 1u), kMaxDotSplits);
    const uint32_t fewest = (columns + max_n - 1) / max_n, most = std::max(fewest, columns / 32);
    uint64_t lowest = ~0ull;
    uint32_t last = 0;
    for (uint32_t count = fewest; count <= most; ++count) {
        const uint32_t width = std::min(max_n, ((columns + count - 1) / count + 15) & ~15u);
        if (width == last) continue;                              // (rounding up gives most counts the same width)
        last = width;
        const uint32_t tiles = (columns + width - 1) / width, b = best.pair ? width / 2 : width;
        for (uint32_t s = 1; s <= max_splits && (s == 1 || 2 * s <= slices); ++s) {
            const uint32_t len = (slices + s - 1) / s;
            if ((s - 1) * len >= slices) continue;                // (the last range would be empty)
            const uint64_t waves = ((uint64_t)m_tiles * tiles * s + wave - 1) / wave;
            const uint64_t cost = waves * len * (row_tile + b) * slice_bytes * planes + (uint64_t)s * n * T * 8 / wave;
            if (cost < lowest) { lowest = cost; best.n_tile = width; best.splits = s; best.kb_split = len; }
        }
    }
    return best;
}

} // namespace pinkb
#endif
