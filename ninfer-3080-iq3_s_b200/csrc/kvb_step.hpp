// kvb_step.hpp -- which parts of a step (append, attention, merge) may run beside each other.  Host only, no CUDA.
#pragma once

#include <cstddef>
#include <cstdint>

namespace kvb {

struct Span {
    uintptr_t begin, end;
};
inline Span span_of(const void* p, size_t bytes) {
    const uintptr_t at = reinterpret_cast<uintptr_t>(p);
    return {at, at + bytes};
}
inline bool overlap(Span a, Span b) { return a.begin < b.end && b.begin < a.end; }

// Whether the attention of a step starts its work beside the append (whose trigger lets every kernel behind it be launched), and only what
// of it reads the rows written there waits for the append's end.  Measured on B200, a layer of a step launched one by one: 32,768 tokens 13.8 ->
// 13.4 us, 8-row verify of 100,003 67.6 -> 63.6, a prompt of 777 35.9 -> 33.0.  Several rows of a verify step at 256 dims are launched early
// and wait (2 / 4 / 5 / 8 rows at 20,000 tokens, graph replay, 25.2 / 29.8 / 35.3 / 46.6 -> 24.6 / 29.5 / 34.7 / 46.2).  The kernel with one warp a
// page lost by starting beside the append (5 rows 41.2 -> 42.5); the one with two, which is there now, would gain (34.7 -> 33.9): the line is
// older than it.
inline bool append_starts_next(int head_dim, int tokens) { return head_dim == 128 || tokens == 1 || tokens > 8; }

// An append right before the attention: whether the attention starts its work beside it, and what it reads.
struct StepAppend {
    bool starts_next;
    Span k, v, positions;
};

// An attention that starts beside its append (after_append in the kernels' parameters) reads q, the positions and the pages the append
// leaves alone, and writes, without waiting for it.  That is sound because
//   - the append is the launch right before it in the stream and waits for all before it ahead of its trigger;
//   - the CTAs and warps that read what the append writes (the stage, tiles from that of its first row on) wait for its end first;
//   - what the attention writes shares no memory with what the append reads: checked here;
//   - every thread waits for the append before it leaves, so that whatever waits for the attention finds both over.
inline bool starts_beside(const StepAppend* step, Span written) {
    return step != nullptr && step->starts_next && !overlap(written, step->k) && !overlap(written, step->v) && !overlap(written, step->positions);
}

// Whether the CTAs of a chunk may store finished rows while others still read q and the positions.  Rows of an output that is q
// itself are read by the CTA that stores them, before it does.
inline bool stores_beside(Span out, Span q, Span positions, Span total_pos) {
    return (out.begin == q.begin || !overlap(out, q)) && !overlap(out, positions) && !overlap(out, total_pos);
}

}  // namespace kvb
