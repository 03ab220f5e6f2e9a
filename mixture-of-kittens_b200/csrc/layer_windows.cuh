// How a layer call cuts its schedule rows: windows of the activation ring, and the chunks of a window that are handed from
// dispatch to the GEMMs to combine.  Host code only.
#pragma once

#include <cstdlib>

#include "../../include/mok_b200.h"

namespace mok {

constexpr int kMinibatchesPerChunk = 8;

// Schedule rows that the call runs over.  The capacity is at least twice the routes of a rank, so launches sized for it find
// nothing to do in half of the windows and chunks (each costs the host about 5 us and the GPU 2 to 3).  How far an expert is
// padded is the schedule's own business, so only the caller can promise fewer rows; dispatch_kernel and the gathering quantizer
// report a schedule that claims more.
inline int covered_rows(const mok_layer_args* a) {
    return a->schedule_rows > 0 && a->schedule_rows < a->schedule_capacity ? a->schedule_rows : a->schedule_capacity;
}

inline int num_windows(const mok_layer_args* a) { return (covered_rows(a) + a->macrobatch_size - 1) / a->macrobatch_size; }

// rows [begin, end) of the schedule; `base` is the schedule row held by row 0 of the activation buffers
struct Span {
    int begin, end, base;
};

inline Span window_span(const mok_layer_args* a, int w) {
    Span s;
    s.begin = s.base = w * a->macrobatch_size;
    s.end = s.begin + a->macrobatch_size;
    if (s.end > covered_rows(a)) s.end = covered_rows(a);
    return s;
}

// Rows handed from dispatch to the GEMMs to combine in one piece: kMinibatchesPerChunk minibatches, so the caller's
// minibatch_size sets the hand-over granularity (the default 4096 gives 32768-row chunks, the size that measured best
// on the DeepSeek-V3-shaped layer).  MOK_CHUNK_ROWS overrides the row count (rounded up to whole minibatches).
// One rank: a window is cut into equal chunks of about that size; one that holds less than one and a half of them stays whole,
// and without anything to hand over (`whole`) every one does: each further launch adds a nearly empty last wave of tiles.
// Several ranks: chunks of exactly that size, as they were measured, and what is left.  The second chunk of a window between one and
// one and a half of them is what the first one's NVLink stores run beside.
inline int chunk_rows_for(const mok_layer_args* a, int window_rows, bool whole) {
    long long rows = whole ? window_rows : static_cast<long long>(kMinibatchesPerChunk) * a->minibatch_size;
    if (const char* v = std::getenv("MOK_CHUNK_ROWS")) {
        const int r = std::atoi(v);
        if (r > 0) rows = r;
    }
    if (a->ep_size == 1) {
        const long long n = (window_rows + rows / 2) / rows;
        if (n <= 1) return window_rows;
        rows = (window_rows + n - 1) / n;
    }
    rows = (rows + a->minibatch_size - 1) / a->minibatch_size * a->minibatch_size;
    // never more than ~100 chunks per window: events and launches stay bounded
    const long long min_rows = (a->macrobatch_size / 100 + a->minibatch_size) / a->minibatch_size * a->minibatch_size;
    if (rows < min_rows) rows = min_rows;
    return static_cast<int>(rows < window_rows ? rows : window_rows);
}

}  // namespace mok
