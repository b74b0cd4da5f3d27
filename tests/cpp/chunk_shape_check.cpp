// The workspace bound of the chunk kernels against the shapes their rules take: a workspace for `tokens` and `keys` serves every
// call of up to that many, and is what one of them can use, not a multiple of it.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "kvb_chunk_shape.hpp"

using namespace kvb;

int main() {
    const int heads[][2] = {{4, 24}, {8, 32}, {2, 16}, {1, 7}, {8, 8}, {1, 1}, {3, 9}, {8, 64}};
    int bad = 0;
    for (int sms : {148, 132, 20})
        for (int D : {128, 256})
            for (const auto& h : heads) {
                std::vector<int> keys;
                for (int n = 1; n <= 270000; n += n < 9000 ? 64 : n < 70000 ? 640 : 6400) keys.push_back(n);
                std::vector<int64_t> most(keys.size(), 0);  // of all calls of up to t tokens and keys[i] keys
                const int G = h[1] / h[0];
                for (int t = 1; t <= 4096; t += t < 1024 ? (128 + G - 1) / G : 128) {
                    int64_t run = 0;
                    for (size_t i = 0; i < keys.size(); ++i) {
                        const ChunkShape s = D == 128 ? chunk_shape_128(keys[i], h[0], h[1], t, sms) : chunk_shape_256(keys[i], h[0], h[1], t, sms);
                        if (s.ranges < 1 || s.ksplit > kMaxKeyRanges || s.ksplit != s.ranges * (s.split ? 2 : 1)) ++bad;
                        const int64_t need = static_cast<int64_t>(s.mtiles) * s.ksplit * h[0];
                        run = run > need ? run : need;
                        if (most[i] < run) most[i] = run;
                        const int64_t bound = most_partials(D, keys[i], h[0], h[1], t, sms);
                        if (bound < most[i] && bad++ < 5)
                            std::printf("D %d heads %d/%d sms %d tokens %d keys %d: bound %ld, needed %ld\n", D, h[0], h[1], sms, t, keys[i], static_cast<long>(bound), static_cast<long>(most[i]));
                        if (bound > 5 * most[i] && bad++ < 5)
                            std::printf("D %d heads %d/%d sms %d tokens %d keys %d: bound %ld for %ld\n", D, h[0], h[1], sms, t, keys[i], static_cast<long>(bound), static_cast<long>(most[i]));
                    }
                }
            }
    // the calls of tests/test_gpu_chunk_finish.py: one key range, and the walk they are there for
    const struct { int kv_heads, q_heads, ctx, tokens; bool split; } one_range[] = {
        {4, 24, 0, 780, true}, {8, 64, 0, 128, true}, {1, 3, 0, 20, true}, {2, 16, 0, 8, true}, {8, 64, 250, 8, true}, {4, 24, 300, 40, true}, {4, 24, 192, 8, true}, {4, 32, 125, 5, true}, {8, 64, 56, 4, true},
        {8, 64, 0, 290, false}, {4, 28, 5, 680, false}, {4, 24, 0, 1024, false}, {8, 24, 130, 1000, false}, {8, 64, 0, 1023, false}, {8, 64, 140, 290, false}};
    for (const auto& c : one_range) {
        const ChunkShape s = chunk_shape_128(c.ctx + c.tokens, c.kv_heads, c.q_heads, c.tokens, 148);
        if (s.ranges == 1 && s.split == c.split) continue;
        std::printf("heads %d/%d ctx %d tokens %d: %d ranges, split %d\n", c.kv_heads, c.q_heads, c.ctx, c.tokens, s.ranges, s.split);
        ++bad;
    }
    std::printf(bad ? "chunk shapes: %d wrong\n" : "chunk shapes: ok\n", bad);
    return bad != 0;
}
