// The batched decode's schedule against one that hands every CTA to the earliest place, and the plan a thread keeps.
#include <cmath>
#include <cstdio>
#include <functional>
#include <queue>
#include <random>
#include <vector>

#include "kvb_batch_plan.hpp"

using namespace kvb;

static int64_t one_by_one(const int* us, const int* parts, int batch, int places) {
    std::priority_queue<int64_t, std::vector<int64_t>, std::greater<int64_t>> free_at(std::greater<int64_t>(), std::vector<int64_t>(places, 0));
    int64_t end = 0;
    for (int b = 0; b < batch; ++b)
        for (int i = 0; i < parts[b]; ++i) {
            const int64_t t = free_at.top() + us[b];
            free_at.pop();
            free_at.push(t);
            end = std::max(end, t);
        }
    return end;
}

int main() {
    int bad = 0;
    std::mt19937 rng(7);
    auto between = [&](int lo, int hi) { return lo + static_cast<int>(rng() % static_cast<unsigned>(hi - lo + 1)); };
    for (int round = 0; round < 4000 && bad < 5; ++round) {
        const int batch = between(1, kBatchMost), places = round % 50 == 0 ? 1 : between(1, kBatchPlaces), longest = 1 << between(2, 17), shortest = between(0, 1) ? longest : longest / 8;
        const int chunk = 4 * between(1, std::max(1, longest / 16));
        const BatchCost cost{1, 30, 43};
        int32_t tiles[kBatchMost];
        int us[kBatchMost], parts[kBatchMost];
        int64_t work = 0;
        for (int b = 0; b < batch; ++b) {
            tiles[b] = between(shortest, longest);
            parts[b] = batch_parts(tiles[b], chunk);
            us[b] = cost.fixed + cost.round * (((tiles[b] + parts[b] - 1) / parts[b] + 3) / 4);
            work += static_cast<int64_t>(us[b]) * parts[b];
        }
        const float per_place = static_cast<float>(work) / static_cast<float>(places), got = batch_time(tiles, batch, chunk, cost, places);
        const double end = per_place + (static_cast<double>(got) - per_place) / 0.45, want = static_cast<double>(one_by_one(us, parts, batch, places));
        // in units of 1 (what fits the points of time): the same; in coarser ones every CTA is rounded up by less than a unit
        const double unit = want < kBatchTimes / 4 ? 0.0 : 64.0 * kBatchParts * 4.0 * want / kBatchTimes / places + 8.0 * want / kBatchTimes;
        if (std::fabs(end - want) > 2e-5 * (want + per_place) + unit) {
            std::printf("%d sequences, %d places, chunks of %d: ends at %.1f, one by one %.1f\n", batch, places, chunk, end, want);
            ++bad;
        }
    }
    // a thread's last plan serves the same numbers and no others
    LastBatch last;
    int32_t tiles[3] = {100, 700, 1000};
    for (int i = 0; i < 200; ++i) {
        const int n = between(1, 3), heads = 1 << between(0, 3), sms = between(0, 1) ? 148 : 74;
        const int group = between(1, 16);
        const BatchCost cost = group > 8 ? BatchCost{1, 61, 44} : BatchCost{2, 30, 43};
        if (between(0, 2) == 0) tiles[between(0, 2)] = between(1, 3000);
        for (int again = 0; again < 2; ++again)
            {
                const BatchChoice kept = last.of(tiles, n, heads, group, sms, cost), made = choose_batch(tiles, n, heads, group, sms, cost);
                if (kept.chunk != made.chunk || kept.alone != made.alone) {
                    std::printf("a plan of other numbers\n");
                    ++bad;
                }
            }
    }
    // CTAs that are alone on their SMs: no more of them than SMs, no more than 16 pages each
    for (int i = 0; i < 2000 && bad < 5; ++i) {
        const int n = between(1, kBatchMost), heads = 1 << between(0, 3), most = 1 << between(0, 12);
        int32_t t[kBatchMost];
        for (int b = 0; b < n; ++b) t[b] = between(0, most);
        const BatchChoice c = choose_batch(t, n, heads, between(1, 8), 148, {2, 30, 43});
        int all = 0, pages = 0;
        for (int b = 0; b < n; ++b) {
            const int parts = batch_parts(t[b], c.chunk);
            all += parts * heads;
            pages = std::max(pages, (2 * t[b] + parts - 1) / parts);
        }
        if ((c.alone && (all > 148 || pages > 16)) || choose_batch(t, n, heads, 9, 148, {1, 61, 44}).alone) {
            std::printf("alone: %d CTAs, %d pages\n", all, pages);
            ++bad;
        }
    }
    std::printf(bad ? "batch plan: %d wrong\n" : "batch plan: ok\n", bad);
    return bad != 0;
}
