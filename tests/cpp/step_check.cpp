// What of a step may run beside what: by the memory its buffers share.
#include <cstdio>
#include <initializer_list>

#include "kvb_step.hpp"

using namespace kvb;

int main() {
    int bad = 0;
    auto expect = [&](bool got, bool want, const char* what) {
        if (got != want) { std::printf("%s: %d\n", what, got); ++bad; }
    };
    char m[4096];
    const auto at = [&](int begin, int end) { return span_of(m + begin, end - begin); };
    expect(overlap(at(0, 10), at(10, 20)), false, "neighbours");
    expect(overlap(at(0, 11), at(10, 20)) && overlap(at(10, 20), at(0, 11)), true, "one byte");
    expect(overlap(at(0, 100), at(40, 50)) && overlap(at(40, 50), at(0, 100)), true, "inside");
    expect(overlap(at(5, 5), at(5, 5)), false, "nothing");

    const StepAppend step{true, at(1000, 1512), at(2000, 2512), at(3000, 3032)};
    expect(starts_beside(nullptr, at(0, 10)), false, "no append");
    expect(starts_beside(&step, at(0, 1000)) && starts_beside(&step, at(1512, 2000)) && starts_beside(&step, at(2512, 3000)) && starts_beside(&step, at(3032, 4096)), true, "beside what the append reads");
    expect(starts_beside(&step, at(0, 1001)), false, "first byte of k");
    expect(starts_beside(&step, at(1511, 1600)), false, "last byte of k");
    expect(starts_beside(&step, at(2511, 2600)), false, "last byte of v");
    expect(starts_beside(&step, at(3028, 3100)), false, "last position");
    expect(starts_beside(&step, at(0, 4096)), false, "all of them");

    const StepAppend alone{false, step.k, step.v, step.positions};
    expect(starts_beside(&alone, at(0, 10)), false, "an append that does not let it start");
    for (int tokens : {1, 2, 8, 9, 1024}) expect(append_starts_next(128, tokens), true, "128 dims");
    for (int tokens : {1, 2, 8, 9, 1024}) expect(append_starts_next(256, tokens), tokens == 1 || tokens > 8, "256 dims");

    const Span q = at(0, 1024), pos = at(2000, 2032), total = at(3000, 3004);
    expect(stores_beside(at(1024, 2000), q, pos, total), true, "an output of its own");
    expect(stores_beside(q, q, pos, total), true, "in the place of q");
    expect(stores_beside(at(256, 1280), q, pos, total), false, "a token further than q");
    expect(stores_beside(at(1031, 2055), q, pos, total), false, "over the positions");
    expect(stores_beside(at(2500, 3524), q, pos, total), false, "over the newest position");
    std::printf(bad ? "step: %d wrong\n" : "step: ok\n", bad);
    return bad != 0;
}
