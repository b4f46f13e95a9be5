// ss_shares.h -- a job cut over a few host threads.
#pragma once

#include <thread>

namespace ssb {

// f(0) .. f(n - 1), n <= Most: the first on this thread, the others on threads
// of their own; a thread that cannot be had (or the memory for it) leaves its
// and the later ones to this thread.  Nothing is thrown: the callers run under
// C entry points, and a thread must be joined whatever happens.  f must not
// throw either.
template <int Most, class Thread = std::thread, class F>
void run_shares(int n, F f) noexcept {
    Thread threads[Most];
    int started = 1;
    try {
        for (; started < n; ++started) threads[started] = Thread(f, started);
    } catch (...) {
    }
    f(0);
    for (int i = started; i < n; ++i) f(i);
    for (int i = 1; i < started && i < n; ++i) threads[i].join();
}

}  // namespace ssb
