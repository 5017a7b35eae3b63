// gd_workers.h -- host work shared out to threads, without an exception leaving it.
#pragma once

#include <atomic>
#include <thread>
#include <vector>

namespace gd {

// Runs work(k) for every k in [0, n): k = 0 on the caller's thread, the others on
// threads of their own, or on the caller's where no thread can be started.  Returns
// once all have ended; false when one of them threw (out of memory).
template <typename Thread = std::thread, typename F>
bool run_workers(int n, F &&work)
{
    std::atomic<bool> ok{true};
    auto guarded = [&ok, &work](int k) {
        try {
            work(k);
        } catch (...) {
            ok = false;
        }
    };
    std::vector<Thread> threads;
    int started = 1;
    try {
        threads.reserve(n);
        for (; started < n; started++) threads.emplace_back(guarded, started);
    } catch (...) {
    }
    guarded(0);
    for (int k = started; k < n; k++) guarded(k);
    for (Thread &t : threads) t.join();
    return ok;
}

}  // namespace gd
