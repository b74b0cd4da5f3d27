// kvb_shares.hpp -- how the pages of a head are dealt to the splits of a decode or verify step and to their warps.  Host and device, no CUDA.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define KVB_SHARES __host__ __device__ __forceinline__
#else
#define KVB_SHARES inline
#endif

namespace kvb {

KVB_SHARES int smaller(int a, int b) { return a < b ? a : b; }
KVB_SHARES int larger(int a, int b) { return a > b ? a : b; }

// Division by a number of splits as a multiplication; exact from 0 to below 2^26.
struct SplitBy {
    uint32_t all, others;  // 2^32 / nsplit, / (nsplit - 1), rounded up (0: by one)
    KVB_SHARES static uint32_t inverse(int d) { return d > 1 ? 0xFFFFFFFFu / static_cast<uint32_t>(d) + 1u : 0u; }
    KVB_SHARES static int divide(int n, uint32_t inv) { return inv != 0u ? static_cast<int>((static_cast<uint64_t>(static_cast<uint32_t>(n)) * inv) >> 32) : n; }
};

// Pages of split `split` of `n` pages, which its CTA walks W at a time.  The last split has the open tile as well, whose 16-key groups (a
// warp or pair each) count as 3/4 of a page; it takes no page that would be a round more for those with a group.  Neither may cost the
// other splits a round.  A CTA with the open tile was some 2,000 cycles behind the others.
// Measured on B200 in graph replay, append and attention, us a layer, equal shares (by 64-bit divisions, the first position read behind the
// newest, the next kernel's start by every warp) / this:
//   decode at 300, 1,500, 8,000, 32,768, 65,536, 378,944 tokens   8.6  9.1 10.2 12.6 17.8 49.4 / 8.1  7.8  8.7 12.6 17.6 49.1
//   decode of 256 dims at 1,500, 4,000, 30,011                    14.2 13.2 23.1 / 11.5 11.6 21.0
//   4 rows at 1,500, 8,000, 131,072                               9.2 11.6 52.0 / 7.8 10.7 52.2
//   5 rows of 256 dims at 20,000                                  35.9 / 35.3
// From eight rounds on (128 dims) the pages alone are shared, evenly; with the open tile counted / without:
//   4 rows at 126,000, 127,526, 129,000                           49.0 51.1 51.4 / 48.3 48.9 52.0
//   decode at 378,944                                             45.7 / 46.1
//   256 dims at 45,000 (not there)                                62.0 / 63.5
constexpr int kManyRounds = 8;
template <int W, int kSlices> KVB_SHARES void split_pages(int n, int open_keys, int split, int nsplit, SplitBy by, int& begin, int& end) {
    const int groups = larger(open_keys + 15, 0) / 16, weighted = n + groups * 3 / 4;
    int share = SplitBy::divide(n, by.all), more = n - share * nsplit;  // `more` splits have a page more
    const int rounds = (share + (more != 0) + W - 1) / W, keep = rounds * W - groups;
    if (kSlices == 1 && rounds >= kManyRounds) {
        begin = share * split + SplitBy::divide(more * split, by.all);
        end = share * (split + 1) + SplitBy::divide(more * (split + 1), by.all);
        return;
    }
    if (weighted <= rounds * W * nsplit) {
        share = SplitBy::divide(weighted, by.all);
        more = weighted - share * nsplit;
    }
    if (nsplit > 1 && n - share * (nsplit - 1) - more > keep && n - keep <= rounds * W * (nsplit - 1)) {
        share = SplitBy::divide(n - keep, by.others);
        more = n - keep - share * (nsplit - 1);
    }
    begin = smaller(share * split + smaller(split, more), n);
    end = split == nsplit - 1 ? n : smaller(begin + share + (split < more), n);
}
// Pages of warp (or pair) w of the W of a CTA with n.  Over few rounds, and beside the open tile, whose groups the first ones have, the last
// ones take a page more (the first ones rotate the query before they begin); over many, every so many-th.
template <int W> KVB_SHARES int warp_pages(int n, int w, bool last_first) {
    const int share = n / W;
    return last_first ? share * w + larger(w - (W - (n - share * W)), 0) : n * w / W;
}

}  // namespace kvb
