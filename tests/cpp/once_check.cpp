// OncePerDevice under threads: whoever returns finds the set-up of its device done; a set-up that failed is made again.
#include <atomic>
#include <chrono>
#include <cstdio>
#include <thread>
#include <vector>

#include "kvb_once.hpp"

int main() {
    int bad = 0;
    for (int round = 0; round < 20; ++round) {
        kvb::OncePerDevice once;
        std::atomic<int> go{0}, missed{0};
        std::atomic<bool> ready[3] = {};
        std::vector<std::thread> threads;
        for (int i = 0; i < 6; ++i)
            threads.emplace_back([&, i] {
                while (go.load() == 0) {}
                if (i >= 3) std::this_thread::sleep_for(std::chrono::microseconds(300));  // in the middle of another thread's set-up
                const int dev = i % 3;
                const int st = once.run(dev, [&] {
                    std::this_thread::sleep_for(std::chrono::milliseconds(1));
                    ready[dev] = true;
                    return 0;
                });
                if (st != 0 || !ready[dev]) ++missed;
            });
        go = 1;
        for (auto& t : threads) t.join();
        int again = 0;
        for (int dev = 0; dev < 3; ++dev) once.run(dev, [&] { return ++again, 0; });
        bad += missed + again;
    }
    kvb::OncePerDevice once;
    int calls = 0;
    bad += once.run(5, [&] { return ++calls, 7; }) != 7;
    bad += once.run(5, [&] { return ++calls, 0; }) != 0 || once.run(5, [&] { return ++calls, 9; }) != 0 || calls != 2;
    bad += once.run(-1, [&] { return ++calls, 0; }) != 0 || once.run(-1, [&] { return ++calls, 3; }) != 3 || calls != 4;
    std::printf(bad ? "once per device: %d wrong\n" : "once per device: ok\n", bad);
    return bad != 0;
}
