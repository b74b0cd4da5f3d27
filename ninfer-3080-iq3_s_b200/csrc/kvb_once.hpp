// kvb_once.hpp -- set-up that CUDA keeps per device and a library makes once.  Host only, no CUDA.
#pragma once

#include <atomic>
#include <cstdint>

namespace kvb {

// run(device, setup): `setup` (which returns 0 when it succeeded) has been run for `device` when this returns 0.  Threads that make
// the first call at once each run it -- it must bear that --, so that none goes on before the set-up is done; one that failed is
// run again by the next call.  Devices from 64 on, and a negative one (unknown), run it every time.
class OncePerDevice {
    std::atomic<uint64_t> done_{0};

public:
    template <typename F> auto run(int device, F setup) -> decltype(setup()) {
        const uint64_t bit = device >= 0 && device < 64 ? uint64_t{1} << device : 0;
        if ((done_.load(std::memory_order_acquire) & bit) != 0) return decltype(setup())(0);
        const auto status = setup();
        if (status == decltype(setup())(0)) done_.fetch_or(bit, std::memory_order_release);
        return status;
    }
};

}  // namespace kvb
