// The pages of a head, dealt to splits and warps: each page once, in order, whatever the open tile; no split has a round more than with equal
// shares; quotients exact.
#include <cstdint>
#include <cstdio>
#include <initializer_list>

#include "kvb_shares.hpp"

using namespace kvb;

static int bad = 0;
static void wrong(const char* what, int n, int open, int nsplit, int at) {
    if (bad++ < 10) std::printf("%s: %d pages, open tile %d, %d splits, at %d\n", what, n, open, nsplit, at);
}

template <int W, int kSlices> static void deal(int n, int open, int nsplit) {
    const SplitBy by{SplitBy::inverse(nsplit), SplitBy::inverse(nsplit - 1)};
    const int rounds = ((n + nsplit - 1) / nsplit + W - 1) / W;
    int next = 0;
    for (int s = 0; s < nsplit; ++s) {
        int begin, end;
        split_pages<W, kSlices>(n, open, s, nsplit, by, begin, end);
        if (begin != next || end < begin || end > n) return wrong("split", n, open, nsplit, s);
        if (end - begin > rounds * W) return wrong("rounds", n, open, nsplit, s);
        next = end;
        for (int last_first = 0; last_first < 2; ++last_first) {
            if (warp_pages<W>(end - begin, 0, last_first) != 0 || warp_pages<W>(end - begin, W, last_first) != end - begin) return wrong("warps", n, open, nsplit, s);
            for (int w = 0; w < W; ++w) {
                const int mine = warp_pages<W>(end - begin, w + 1, last_first) - warp_pages<W>(end - begin, w, last_first);
                if (mine < 0 || mine > (end - begin + W - 1) / W) return wrong("warp", n, open, nsplit, w);
            }
        }
    }
    if (next != n) wrong("all", n, open, nsplit, next);
}

int main() {
    // a newest position below 0 leaves a remainder below 0: no key is there
    static const int kOpen[] = {0, 1, 15, 16, 17, 33, 64, 100, 127, -1, -46, -47, -50, -71, -127};
    for (int nsplit = 1; nsplit <= 64; ++nsplit)
        for (int open : kOpen)
            for (int k = 0; k < 300; ++k) {
                const int n = k < 200 ? k : k < 260 ? 37 * (k - 190) : 911 * (k - 250) + nsplit;
                deal<8, 1>(n, open, nsplit);
                deal<12, 1>(n, open, nsplit);
                deal<16, 1>(n, open, nsplit);
                deal<8, 2>(n, open, nsplit);
            }
    for (int d = 2; d <= 64; ++d)
        for (int64_t n = 0; n < (1 << 26); n += n < 5000 ? 1 : 77777) {
            const int m = static_cast<int>(n), multiple = m / d * d;
            for (int x : {m, multiple, multiple > 0 ? multiple - 1 : 0})
                if (SplitBy::divide(x, SplitBy::inverse(d)) != x / d) wrong("quotient", x, 0, d, 0);
        }
    std::printf(bad ? "shares: %d wrong\n" : "shares: ok\n", bad);
    return bad != 0;
}
