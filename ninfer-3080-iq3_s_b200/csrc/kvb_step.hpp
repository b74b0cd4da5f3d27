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

// What an append right before the attention reads.
struct StepAppend {
    Span k, v, positions;
};

// The attention writes (partials, or finished rows) while the append may still read: it starts beside the append unless what it writes
// shares memory with what the append reads.
inline bool starts_beside(const StepAppend* step, Span written) {
    return step != nullptr && !overlap(written, step->k) && !overlap(written, step->v) && !overlap(written, step->positions);
}

// Whether the CTAs of a chunk may store finished rows while others still read q and the positions.  Rows of an output that is q
// itself are read by the CTA that stores them, before it does.
inline bool stores_beside(Span out, Span q, Span positions, Span total_pos) {
    return (out.begin == q.begin || !overlap(out, q)) && !overlap(out, positions) && !overlap(out, total_pos);
}

}  // namespace kvb
