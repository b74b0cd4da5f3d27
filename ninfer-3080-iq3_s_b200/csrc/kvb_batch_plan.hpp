// kvb_batch_plan.hpp -- how the caches of a batched decode are cut into parts.  Host only, no CUDA.
#pragma once

#include <algorithm>
#include <cstdint>

namespace kvb {

// Parts (splits over the sealed tiles; the last one also reads the open tile) of every sequence from the host's
// bounds of their lengths: chunks of at least 4 tiles, at most 64 splits per sequence.  A CTA of 8 warps takes `fixed` (set-up,
// first fetch, merge) and `round` per 8 pages; `beside` of them share an SM, so that one's set-up and end lie beside the
// others' work.  Chunk sizes that make about 1/2 .. 4 waves of CTAs are costed by the work per place plus 0.45 of what the last CTA
// ends later than that, the CTAs of a head taken in order by its share of the places (a CTA left alone on its SM runs faster, hence not
// all of it: fitted to sweeps of the chunk size over six batches).  Measured on B200, calls in a row, one CTA of 16 warps an SM with 2 ..
// 12 CTAs per SM in total against this, us: 32 sequences of up to 131,072 tokens (24 / 4 heads) 317 -> 286, 8 of them 117 -> 84, 48 of
// 30,000 130 -> 124, 40 of 4,096 34.4 -> 31.5, 24 of 100,000 (32 / 8) 353 -> 342, 20 of 60,000 (16 / 2) 73.5 -> 52.8.
struct BatchCost {
    int beside;
    int fixed, round;  // tenths of a microsecond
};
constexpr int kBatchMost = 64;     // sequences of a call
constexpr int kBatchParts = 64;    // of a sequence: what the merge kernel holds
constexpr int kBatchLeast = 4;     // tiles of a chunk: a page for each of the 8 warps
constexpr int kBatchPlaces = 512;  // the most places of a head that are modelled
constexpr int kBatchTimes = 16384; // the most points of time that are modelled; longer calls in coarser units

inline int batch_parts(int tiles, int chunk) { return std::min(std::max((tiles + chunk - 1) / chunk, 1), kBatchParts); }

// When the last of the CTAs ends: parts[b] of them that take us[b] each, in order, each on the place that is free first.  Places are counted by
// the time they are free at, and a sequence's CTAs that begin at one time are taken together.  `bound`: no end lies beyond it.
inline int last_end(const int* us, const int* parts, int batch, int places, int bound) {
    uint16_t free_at[kBatchTimes];
    uint64_t any[kBatchTimes / 64];
    std::fill_n(free_at, bound + 1, uint16_t{0});
    std::fill_n(any, bound / 64 + 1, uint64_t{0});
    free_at[0] = static_cast<uint16_t>(places);
    any[0] = 1;
    int now = 0, end = 0;
    for (int b = 0; b < batch; ++b)
        for (int left = parts[b]; left > 0;) {
            if (free_at[now] == 0) {
                int w = now / 64;
                uint64_t bits = any[w] & (~uint64_t{0} << (now % 64));
                while (bits == 0) bits = any[++w];
                now = 64 * w + __builtin_ctzll(bits);
            }
            const int n = std::min<int>(left, free_at[now]), then = now + us[b];
            left -= n;
            free_at[now] = static_cast<uint16_t>(free_at[now] - n);
            if (free_at[now] == 0) any[now / 64] &= ~(uint64_t{1} << (now % 64));
            free_at[then] = static_cast<uint16_t>(free_at[then] + n);
            any[then / 64] |= uint64_t{1} << (then % 64);
            end = std::max(end, then);
        }
    return end;
}

// The modelled time with this chunk size, in tenths of a microsecond.
inline float batch_time(const int32_t* tiles, int batch, int chunk, const BatchCost& cost, int places) {
    int us[kBatchMost], parts[kBatchMost];
    int64_t work = 0, longest = 0;
    for (int b = 0; b < batch; ++b) {
        parts[b] = batch_parts(tiles[b], chunk);
        us[b] = cost.fixed + cost.round * (((tiles[b] + parts[b] - 1) / parts[b] + 3) / 4);
        work += static_cast<int64_t>(us[b]) * parts[b];
        longest = std::max<int64_t>(longest, us[b]);
    }
    // a CTA begins when all places are taken, at the latest at their mean end
    int64_t unit = 1;
    auto bound = [&] { return (work / unit + kBatchMost * kBatchParts) / places + longest / unit + 2; };
    while (bound() >= kBatchTimes) unit *= 2;
    if (unit > 1)
        for (int b = 0; b < batch; ++b) us[b] = static_cast<int>((us[b] + unit - 1) / unit);
    const float per_place = static_cast<float>(work) / static_cast<float>(places), end = static_cast<float>(unit * last_end(us, parts, batch, places, static_cast<int>(bound())));
    return per_place + 0.45f * (end - per_place);
}

// Tiles of a chunk for sequences of so many sealed tiles.
inline int plan_batch_chunk(const int32_t* tiles, int batch, int kv_heads, int sms, const BatchCost& cost) {
    int64_t total = 0;
    int most = 0;
    for (int b = 0; b < batch; ++b) {
        total += tiles[b];
        most = std::max(most, tiles[b]);
    }
    const int places = std::min(std::max(1, cost.beside * sms / kv_heads), kBatchPlaces);  // of a head
    int best_chunk = kBatchLeast, last_chunk = 0;
    float best = 1e30f;
    static const float kWaves[] = {0.5f, 0.98f, 1.48f, 1.95f, 2.45f, 2.9f, 3.9f};
    for (float waves : kWaves) {
        const int want = static_cast<int>(static_cast<float>(total) / (waves * static_cast<float>(places))) + 1;
        const int chunk = (std::max({kBatchLeast, want, (most + kBatchParts - 1) / kBatchParts}) + 3) / 4 * 4;
        if (chunk == last_chunk) continue;
        last_chunk = chunk;
        const float time = batch_time(tiles, batch, chunk, cost, places);
        if (time < best) {
            best = time;
            best_chunk = chunk;
        }
    }
    return best_chunk;
}

// How a batch runs: tiles of a chunk, and whether its CTAs (up to 8 merged rows) are `alone` on their SMs, with 16 warps.  They are where chunks
// of 4 or 8 tiles, no more than a page a warp, give every CTA an SM of its own: nothing beside it would hide a longer round.  Not where
// the CTAs of the merge, one a row, find SMs that had none of the attention's: 8 warps merge sooner.  Measured on B200 in graph replay, us a call,
// two CTAs of 8 warps an SM / one of 16: 6 sequences of up to 500 / 1,500 / 4,788 tokens (24 / 4 heads) 11.0 11.8 12.3 / 9.2 9.5 9.9, 2 of 10,000
// and 20,000 12.0 13.1 / 9.8 12.1; 2 of 1,500 and 4,788 9.2 8.5 / 9.5 9.0; in chunks of 16 tiles, alone too, 3 of 30,000 15.4 / 16.0.
struct BatchChoice {
    int chunk;
    bool alone;
};
inline BatchChoice choose_batch(const int32_t* tiles, int batch, int kv_heads, int group, int sms, const BatchCost& cost) {
    for (int chunk = kBatchLeast; chunk <= 2 * kBatchLeast && group <= 8; chunk *= 2) {
        int parts = 0;
        bool whole = true;  // no sequence has more chunks than splits
        for (int b = 0; b < batch; ++b) {
            parts += batch_parts(tiles[b], chunk);
            whole = whole && tiles[b] <= chunk * kBatchParts;
        }
        if (whole && parts * kv_heads <= sms) {
            if ((parts + batch * group) * kv_heads <= sms) break;
            return {chunk, true};
        }
    }
    return {plan_batch_chunk(tiles, batch, kv_heads, sms, cost), false};
}

// A thread's last choice, with what it follows from: a serving loop asks for the same one at every step until a sequence
// enters its next tile.  Modelling it takes a host core 2 .. 13 us for 8 .. 64 sequences (10 .. 47 with a heap of places).
struct LastBatch {
    int32_t tiles[kBatchMost];
    int batch = 0, kv_heads = 0, group = 0, sms = 0;
    BatchChoice choice{kBatchLeast, false};

    BatchChoice of(const int32_t* now, int n, int heads, int rows, int processors, const BatchCost& cost) {
        if (batch != n || kv_heads != heads || group != rows || sms != processors || !std::equal(now, now + n, tiles)) {
            choice = choose_batch(now, n, heads, rows, processors, cost);
            std::copy(now, now + n, tiles);
            batch = n;
            kv_heads = heads;
            group = rows;
            sms = processors;
        }
        return choice;
    }
};

}  // namespace kvb
