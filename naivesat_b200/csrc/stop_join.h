// stop_join.h -- SATOSTOP doubling of a table of 32-bit entries (n <= 31).
#pragma once
#include <stdint.h>

#include <functional>

#include "internal.h"
#include "stop_kernels.h"

namespace nsat {

struct StopRun {
    // in: the table built (next | STOP << n) in `a`; `b` has the same size
    uint32_t n = 0, unknowns = 0, mode = 0;
    uint32_t* a = nullptr;
    uint32_t* b = nullptr;
    bool steps = false;            // distances wanted
    uint32_t* dist = nullptr;      // steps: 2^n words, or null to take them from the context's pool
    cudaEvent_t begin = nullptr;   // recorded before the first kernel (null: not wanted)
    cudaEvent_t done = nullptr;    // and behind the last
    uint64_t* out64 = nullptr;     // steps: the 64-bit table after the last round (null: not wanted)
    // where scratch buffers come from, null when there is no room; the caller
    // has them back after the call (not set: the context's pool)
    std::function<void*(size_t)> scratch;
    // out
    uint32_t rounds = 0;
    bool found = false;
    uint32_t start = 0, entry = 0, steps_of = 0;   // entry: halting state | STOP << n
    uint32_t* table = nullptr;     // a or b: the table after the last round (not written when out64 was)
    uint32_t launches = 0;
    bool polled = false;           // one short kernel: no events, its own time is in ms
    double ms = 0;
};

// Runs the rounds on the context's stream and waits for the answer.
// NSAT_ENOMEM (and nothing done) when the distances cannot be allocated.
int stop_run(nsat_ctx* ctx, StopRun* x);

}  // namespace nsat
