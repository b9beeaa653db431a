// Work dealt out to a few threads that end with the call.
#pragma once
#include <exception>
#include <thread>

namespace ma {

// work(0 .. N-1), work(0) on the calling thread and the others on threads of their own.  A thread that cannot be
// had (std::system_error from the system, std::bad_alloc for its state) has its part done on the calling
// thread: nothing leaves here while a thread still runs, and callers are C functions.
template <int N, class Thread = std::thread, class F>
void on_threads(const F& work) {
    Thread pool[N];
    for (int i = 1; i < N; ++i) {
        try {
            pool[i] = Thread(work, i);
        } catch (const std::exception&) {
            work(i);
        }
    }
    work(0);
    for (int i = 1; i < N; ++i)
        if (pool[i].joinable()) pool[i].join();
}

}  // namespace ma
