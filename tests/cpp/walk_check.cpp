// Two warps that share rows walk the parts of their key tiles and give up at every wait they have, alike or not: each meeting has both.
#include <atomic>
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
// are waited for.  A wait that is given up raises the abort flag.  Returns the parts that were worked on.
template <typename Meet> int walk(int steps, Warp w, bool& failed, std::atomic<bool>& abort, Meet meet) {
    int waits = 0, parts = 0;
    auto wait = [&] {
        const bool whole = waits++ < w.first || (waits - 1 > w.first && !w.again);
        if (!whole) abort = true;
        return whole;
    };
    failed = false;
    for (int i = 0; i < steps && !failed; ++i)
        for (int h = 0; h < 2; ++h) {
            if (kvb::leaves_alone<true>(failed, wait(), true)) break;
            if (kvb::leaves_together(failed, meet(failed))) break;
            ++parts;
            if (i + h > 0) wait();
        }
    return parts;
}

// Whether no warp is left alone, and both know in the end if either has given up.
bool two_warps(int steps, Warp a, Warp b) {
    Barrier barrier;
    std::atomic<bool> abort{false};
    bool known[2];
    auto run = [&](int who, Warp w) {
        bool failed;
        walk(steps, w, failed, abort, [&](bool mine) { return barrier.come(who, kVerdict, mine); });
        barrier.come(who, kEnd, failed);
        known[who] = failed || abort;
        barrier.leave(who);
    };
    std::thread other(run, 1, b);
    run(0, a);
    other.join();
    return barrier.sound && known[0] == abort && known[1] == abort;
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
                        if (bad++ < 5) std::printf("%d steps, given up at waits %d and %d (%d): a warp is left alone, or does not know\n", steps, x, y, again);
                    }
    }
    // a warp that shares no rows leaves behind the first wait for a part that is given up (it has no others)
    for (int at = 0; at <= 4; ++at) {
        int waits = 0, parts = 0;
        bool failed = false;
        for (int i = 0; i < 2 && !failed; ++i)
            for (int h = 0; h < 2; ++h) {
                if (at & 1 ? kvb::leaves_alone<false>(failed, waits++ != at, true) : kvb::leaves_alone<true>(failed, waits++ != at, false)) break;
                ++parts;
            }
        if (parts != at || failed != (at < 4)) { std::printf("alone, given up at %d: %d parts\n", at, parts); ++bad; }
    }
    std::printf(bad ? "walk: %d wrong\n" : "walk: ok\n", bad);
    return bad != 0;
}
