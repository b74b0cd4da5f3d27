// Two warps that share rows walk the parts of their key tiles and give up at every wait they have, alike or not: each meeting has both.
#include <condition_variable>
#include <cstdio>
#include <mutex>
#include <thread>

#include "kvb_walk.hpp"

namespace {

enum Kind { kNone, kVerdict, kEnd };  // no meeting, the one of a part, the one behind the walk

// The two warps' barrier: a meeting is sound if both come to the same one; a warp that comes alone finds the other gone.
struct Barrier {
    std::mutex m;
    std::condition_variable cv;
    Kind at[2] = {kNone, kNone};
    bool flag[2] = {false, false}, gone[2] = {false, false}, any = false, sound = true;
    int met = 0;

    bool come(int who, Kind kind, bool mine) {
        std::unique_lock<std::mutex> lock(m);
        if (at[who ^ 1] == kNone && !gone[who ^ 1]) {
            at[who] = kind;
            flag[who] = mine;
            const int before = met;
            cv.wait(lock, [&] { return met != before || gone[who ^ 1]; });
            if (met == before) sound = false;  // left alone
            return any;
        }
        if (gone[who ^ 1] || at[who ^ 1] != kind) sound = false;
        any = mine || flag[who ^ 1];
        at[who ^ 1] = kNone;
        ++met;
        cv.notify_all();
        return any;
    }
    void leave(int who) {
        std::lock_guard<std::mutex> lock(m);
        gone[who] = true;
        cv.notify_all();
    }
};

// A warp gives up at its wait number `first` (none if it never gets there); what it waits for behind that, it gets or does not.
struct Warp {
    int first;
    bool again;
};

// The softmax warps' walk: a part is waited for, two warps that share its rows meet, and before the sums are scaled the products before them
// are waited for.  Returns the parts that were worked on.
template <bool kMeets, typename Meet> int walk(int steps, bool rows, Warp w, bool& failed, Meet meet) {
    int waits = 0, parts = 0;
    auto wait = [&] { return waits++ < w.first || (waits - 1 > w.first && !w.again); };
    kvb::Walk<kMeets> walk;
    for (int i = 0; i < steps; ++i)
        for (int h = 0; h < 2; ++h) {
            walk.waited(wait());
            if (walk.leaves_alone(rows)) { i = steps; break; }
            if (kMeets && walk.leaves_together(meet(walk.failed))) { i = steps; break; }
            ++parts;
            if (i + h > 0) walk.waited(wait());
        }
    failed = walk.failed;
    return parts;
}

bool two_warps(int steps, Warp a, Warp b) {
    Barrier barrier;
    auto run = [&](int who, Warp w) {
        bool failed;
        walk<true>(steps, true, w, failed, [&](bool mine) { return barrier.come(who, kVerdict, mine); });
        barrier.come(who, kEnd, failed);
        barrier.leave(who);
    };
    std::thread other(run, 1, b);
    run(0, a);
    other.join();
    return barrier.sound;
}

}  // namespace

int main() {
    int bad = 0;
    for (int steps = 1; steps <= 3; ++steps) {
        const int waits = 2 * 2 * steps - 1;  // of a whole walk
        for (int x = 0; x <= waits; ++x)
            for (int y = 0; y <= waits; ++y)
                for (int again = 0; again < 4; ++again)
                    if (!two_warps(steps, {x, (again & 1) != 0}, {y, (again & 2) != 0})) {
                        if (bad++ < 5) std::printf("%d steps, given up at waits %d and %d (%d): a warp is left alone\n", steps, x, y, again);
                    }
    }
    // a warp that shares no rows leaves behind the first wait for a part that finds it given up
    for (int at = 0; at <= 7; ++at) {
        bool failed;
        const int parts = walk<false>(2, true, {at, true}, failed, [](bool) { return false; });
        if (parts != (at == 0 ? 0 : at / 2 + 1) || failed != (at < 7)) { std::printf("alone, given up at %d: %d parts\n", at, parts); ++bad; }
    }
    std::printf(bad ? "walk: %d wrong\n" : "walk: ok\n", bad);
    return bad != 0;
}
