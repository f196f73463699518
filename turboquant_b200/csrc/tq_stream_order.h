// Which of the library's kernels was launched last on a stream, and what may begin before it has finished.  Plain C++.
//
// Several kernels let the launch behind them begin before they have finished (programmatic dependent launch) and do part of
// their work before they wait for the launch ahead; that is only safe when the launch still in flight cannot be writing what is
// read early:
//   * the tensor-core store kernels fetch their key / value rows before the wait.  The decode family appends the new token to
//     the ring - rows a flush then reads - so a store behind a decode launch only asks for its constant operands early, waits in
//     front of its first row and lets its own dependents begin after that;
//   * the decode family and the scores of the cache object read sequence lengths, block tables and the first pool records before
//     the wait.  The tensor-core store kernels write the pool and let their dependents begin at once.  The query preparation
//     reads nothing that they write and may start under them; the kernel behind it is then told to wait before its first record
//     (and to let its own dependents begin only after that, so that no later kernel's early reads reach back to the store).
//     A decode kernel directly behind a store is launched in plain stream order.  The fp32 store and the planes' converter let
//     nobody begin, but a launch that begins when they have finished has not waited for them either, and only the wait makes
//     what they wrote visible: the same holds behind them.
// Kernels of other libraries between two of ours never start early and only make the order stricter.  Of a stream that has no
// note - the library has not seen it, or other streams' notes took its place - anything may be in flight.
#pragma once

#include <mutex>

enum TqLaunchKind {
    TQ_LAUNCH_UNKNOWN = 0,             // no note
    TQ_LAUNCH_DECODE = 1,              // decode family, ring writes: may write rows, and lets nobody begin while a store may be in flight
    TQ_LAUNCH_STORE_EARLY = 2,         // writes the pool and lets its dependents begin at once
    TQ_LAUNCH_NEUTRAL = 3,             // in plain stream order, writes neither rows nor pool
    TQ_LAUNCH_PREP_BEHIND_STORE = 4,   // prepares a call, a store may still be in flight
    TQ_LAUNCH_WAITED = 5,              // writes no pool (rows perhaps), and waits before it lets anyone begin
    TQ_LAUNCH_STORE_PLAIN = 6,         // writes the pool, in plain stream order, and lets nobody begin before it has finished
};

// what a launch is noted as that prepares a call (and neither reads nor writes the pool) and lets its dependents begin at once
inline int tq_kind_of_prep(int ahead) {
    return ahead == TQ_LAUNCH_DECODE || ahead == TQ_LAUNCH_NEUTRAL || ahead == TQ_LAUNCH_WAITED ? TQ_LAUNCH_DECODE : TQ_LAUNCH_PREP_BEHIND_STORE;
}
// whether a kernel that reads the pool early may be launched as a programmatic dependent (else: plain stream order) ...
inline bool tq_reader_may_overlap(int ahead) {
    return ahead != TQ_LAUNCH_STORE_EARLY && ahead != TQ_LAUNCH_STORE_PLAIN && ahead != TQ_LAUNCH_UNKNOWN;
}
// ... and whether it then has to wait before its first record
inline bool tq_pool_is_late(int ahead) { return ahead == TQ_LAUNCH_PREP_BEHIND_STORE || !tq_reader_may_overlap(ahead); }
// whether a store may read its rows early
inline bool tq_rows_are_at_rest(int ahead) {
    return ahead == TQ_LAUNCH_STORE_EARLY || ahead == TQ_LAUNCH_STORE_PLAIN || ahead == TQ_LAUNCH_NEUTRAL;
}

// The notes of one device: the streams noted last, up to eight.
class TqStreamNotes {
    struct Note {
        const void* stream;
        int kind;
    };
    std::mutex mu_;
    Note notes_[8];
    int count_ = 0, next_ = 0;

public:
    void note(const void* stream, int kind) {
        std::lock_guard<std::mutex> lock(mu_);
        for (int i = 0; i < count_; ++i)
            if (notes_[i].stream == stream) {
                notes_[i].kind = kind;
                return;
            }
        notes_[next_] = Note{stream, kind};
        next_ = (next_ + 1) % 8;
        if (count_ < 8) ++count_;
    }
    int last(const void* stream) {
        std::lock_guard<std::mutex> lock(mu_);
        for (int i = 0; i < count_; ++i)
            if (notes_[i].stream == stream) return notes_[i].kind;
        return TQ_LAUNCH_UNKNOWN;
    }
};
