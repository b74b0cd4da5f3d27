// kvb_walk.hpp -- when a softmax warp of a chunk kernel that has given up leaves the walk over its key tiles.  Host and device, no CUDA.
#pragma once

#ifdef __CUDACC__
#define KVB_WALK __host__ __device__ __forceinline__
#else
#define KVB_WALK inline
#endif

namespace kvb {

// Two warps that share rows (`kMeets`, and their rows are real) meet once in every part of a key tile, with one verdict for both: whether
// either has given up a wait.  Such a warp leaves at a meeting and nowhere else, even if it gave up long before: its partner waits for
// it at the next one.  Other warps leave behind their next wait for a part.
template <bool kMeets> struct Walk {
    bool failed = false;

    KVB_WALK void waited(bool whole) { if (!whole) failed = true; }
    // Behind the wait for a part: whether the warp leaves.
    KVB_WALK bool leaves_alone(bool rows) const { return failed && !(kMeets && rows); }
    // Behind the meeting in it, which the warp came to with `failed`: whether both leave.
    KVB_WALK bool leaves_together(bool verdict) {
        if (verdict) failed = true;
        return verdict;
    }
};

}  // namespace kvb
