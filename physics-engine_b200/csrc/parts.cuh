// A call's work in parts, each by a thread of its own. Plain C++.
#pragma once

#include <thread>

namespace pe {

// Calls run(0) .. run(parts - 1), parts <= MAX, the first on the caller's thread, and
// returns when all have. A part no thread could be had for (no thread, or no memory
// for one: either is an exception, with threads running that have to be joined) is
// the caller's. run must not throw.
template <int MAX, class F>
void run_parts(int parts, F& run) noexcept {
    std::thread pool[MAX];
    for (int t = 1; t < parts; ++t) {
        try {
            pool[t] = std::thread([&run, t] { run(t); });
        } catch (...) {
        }
    }
    run(0);
    for (int t = 1; t < parts; ++t) {
        if (pool[t].joinable()) pool[t].join();
        else run(t);
    }
}

}  // namespace pe
