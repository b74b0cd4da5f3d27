// kvb_chunk_shape.hpp -- how the chunk kernels cut a call into CTAs, and the workspace that takes.  Host only, no CUDA.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace kvb {

constexpr int kRowTile = 128;       // rows per row tile of the partials
constexpr int kMaxKeyRanges = 128;  // what the merge kernel holds
constexpr int kWaves = 4;           // at most four waves of CTAs, one CTA per SM

// What a rule weighs: waves x (fixed + step x key steps of a range) for r key ranges of `ctas` CTAs each.
struct ShapeCost {
    int fixed, step;   // of a CTA
    int min_steps;     // key steps a range has at least (one range always goes)
    int parts;         // partials a row gets per range
};
// head_dim 128, in fifths of the time a row tile takes for a key tile with two row tiles a CTA (1.15 us, measured at 1,024 tokens over
// 262,144; with split keys 1.7 us): a step of two row tiles costs 10, one with split keys 7, set-up and epilogue about 17 and 12 us.
// Measured, the kernel alone: 1,024 tokens over 262,144 3.06 ms with two row tiles, 4.49 ms with split keys; 777 tokens alone 35.6 and
// 23.9 us (their append included 36.8 and 29.2).  The costs are those of ranges that are merged: that one range writes no partials and
// needs no merge kernel is not in them.
constexpr ShapeCost kTwoTiles{70, 10, 2, 1}, kSplitKeys{50, 7, 2, 2};
// head_dim 256: a CTA costs its pages plus about six pages' worth of set-up and epilogue.
constexpr ShapeCost kPages256{6, 1, 4, 1};

inline int64_t shape_cost(const ShapeCost& c, int64_t ctas, int64_t r, int64_t steps, int sms) {
    return (ctas * r + sms - 1) / sms * (c.fixed + c.step * ((steps + r - 1) / r));
}
inline bool range_count_goes(const ShapeCost& c, int64_t ctas, int64_t r, int64_t steps, int sms) {
    return c.parts * r <= kMaxKeyRanges && (r == 1 || (c.min_steps * r <= steps && ctas * r <= static_cast<int64_t>(kWaves) * sms));
}

struct ChunkShape {
    bool split;             // 128 dims: one row tile per CTA, its streams split the keys
    int mtiles, ksplit;     // row tiles; partials per row
    int ranges;             // key ranges (grid z)
};
inline int row_tiles(int q_heads, int kv_heads, int tokens) { return (tokens * (q_heads / kv_heads) + kRowTile - 1) / kRowTile; }

// The cheapest of two row tiles a CTA and split keys, and of the numbers of key ranges.
inline ChunkShape chunk_shape_128(int kv_len_max, int kv_heads, int q_heads, int tokens, int sms) {
    const int mtiles = row_tiles(q_heads, kv_heads, tokens), steps = (kv_len_max + 127) / 128;
    ChunkShape best{};
    int64_t best_cost = INT64_MAX;
    for (int split = mtiles == 1 ? 1 : 0; split < 2; ++split) {
        const ShapeCost& c = split ? kSplitKeys : kTwoTiles;
        const int ctas = (split ? mtiles : (mtiles + 1) / 2) * kv_heads;
        for (int r = 1; range_count_goes(c, ctas, r, steps, sms); ++r) {
            const int64_t cost = shape_cost(c, ctas, r, steps, sms);
            if (cost < best_cost) {
                best_cost = cost;
                best = {split != 0, mtiles, c.parts * r, r};
            }
        }
    }
    return best;
}
inline ChunkShape chunk_shape_256(int kv_len_max, int kv_heads, int q_heads, int tokens, int sms) {
    const int mtiles = row_tiles(q_heads, kv_heads, tokens), steps = (kv_len_max + 63) / 64, ctas = mtiles * kv_heads;
    ChunkShape best{};
    int64_t best_cost = INT64_MAX;
    for (int r = 1; range_count_goes(kPages256, ctas, r, steps, sms); ++r) {
        const int64_t cost = shape_cost(kPages256, ctas, r, steps, sms);
        if (cost < best_cost) {
            best_cost = cost;
            best = {false, mtiles, r, r};
        }
    }
    return best;
}

// The most key ranges the rule can take for `ctas` CTAs a range at any number of key steps up to `steps`.  More ranges in more
// waves win only where their cost, without the rounding of the steps, is below that of the most ranges of fewer waves, with it;
// both sides are linear in the steps, so the two ends decide.
inline int64_t most_ranges(const ShapeCost& c, int64_t ctas, int64_t steps, int sms) {
    auto waves = [&](int64_t r) { return (ctas * r + sms - 1) / sms; };
    int64_t r = std::min<int64_t>({kMaxKeyRanges / c.parts, steps / c.min_steps, static_cast<int64_t>(kWaves) * sms / ctas});
    for (; r > 1; --r) {
        const int64_t w = waves(r);
        bool wins = true;
        for (int64_t v = 1; v < w && wins; ++v) {
            const int64_t q = v * sms / ctas;  // the most ranges of v waves, if any
            if (q < 1) continue;
            auto below = [&](int64_t n) {  // w (fixed + step n / r) < v (fixed + step (n + q - 1) / q), times r q
                return r * q * c.fixed * (w - v) + c.step * n * (w * q - v * r) - c.step * v * r * (q - 1) < 0;
            };
            wins = below(c.min_steps * r) || below(steps);
        }
        if (wins) break;
    }
    return std::max<int64_t>(r, 1);
}

// The most partials (tiles of 128 rows) a call of up to `tokens` tokens and `kv_len_max` keys can have: a shorter call may be cut
// into more ranges.  Row tiles beyond four waves always go with one range.
inline int64_t most_partials(int head_dim, int kv_len_max, int kv_heads, int q_heads, int tokens, int sms) {
    const int64_t mtiles = row_tiles(q_heads, kv_heads, tokens), few = std::min<int64_t>(mtiles, 2 * static_cast<int64_t>(kWaves) * sms / kv_heads + 2);
    const int64_t steps = head_dim == 128 ? (kv_len_max + 127) / 128 : (kv_len_max + 63) / 64;
    int64_t most = mtiles * kv_heads * (head_dim == 128 ? 2 : 1);
    for (int64_t m = 1; m <= few; ++m) {
        if (head_dim != 128) {
            most = std::max(most, m * kv_heads * most_ranges(kPages256, m * kv_heads, steps, sms));
            continue;
        }
        most = std::max(most, m * kv_heads * 2 * most_ranges(kSplitKeys, m * kv_heads, steps, sms));
        if (m > 1) most = std::max(most, m * kv_heads * most_ranges(kTwoTiles, (m + 1) / 2 * kv_heads, steps, sms));
    }
    return most;
}
inline size_t partials_bytes(int64_t partials, int head_dim) { return static_cast<size_t>(partials) * kRowTile * (head_dim + 2) * sizeof(float); }

}  // namespace kvb
