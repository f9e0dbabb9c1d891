// Contexts for tests of batch.cpp: a context does nothing but count the work
// that is queued on its memory.
#pragma once
#include <atomic>
#include <thread>

#include "gnss_b200.h"

struct gnss_ctx {
    gnss_config cfg{};
    std::atomic<int> queued{0};   // steps and clears queued and not yet run
};

namespace fake {
extern std::atomic<int> live;                 // contexts created and not destroyed
extern std::atomic<int> recycled;             // contexts taken over by gnss_recycle
extern std::atomic<int> recycled_busy;        // ... with work still queued
extern std::atomic<int> destroyed_elsewhere;  // gnss_destroy calls from other threads than main
extern std::atomic<int> fail_after;           // steps of a stream that succeed before one fails (-1: all do)
extern std::thread::id main_thread;
}  // namespace fake
