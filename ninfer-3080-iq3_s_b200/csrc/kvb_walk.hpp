// kvb_walk.hpp -- when a softmax warp of a chunk kernel that has given up leaves the walk over its key tiles.  Host and device, no CUDA.
#pragma once

#ifdef __CUDACC__
#define KVB_WALK __host__ __device__ __forceinline__
#else
#define KVB_WALK inline
#endif

namespace kvb {

// Two warps that share rows (`kMeets`, and their rows are real) meet once in every part of a key tile, with one verdict for both: whether
// either has given up the wait for the part.  They leave at a meeting and nowhere else; other warps leave behind that wait.  The
// walk goes on while nobody has failed: for (..; i < steps && !failed; ..).  A wait behind the meeting that is given up must not end
// the walk of one of the two: it raises the CTA's abort flag alone, which both look at behind the walk, with the last sums there.

// Behind the wait for a part: whether the warp leaves.
template <bool kMeets> KVB_WALK bool leaves_alone(bool& failed, bool whole, bool rows) {
    if (!whole) failed = true;
    return failed && (!kMeets || !rows);
}
// Behind the meeting in it, which the warp came to with `failed`: whether both leave.
KVB_WALK bool leaves_together(bool& failed, bool verdict) {
    if (verdict) failed = true;
    return verdict;
}

}  // namespace kvb
