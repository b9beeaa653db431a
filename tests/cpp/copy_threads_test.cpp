// on_threads when threads cannot be had: every part is done once, and nothing is thrown.
#include <atomic>
#include <cstdio>
#include <new>
#include <system_error>
#include <thread>
#include <utility>

#include "../../metalaudio_b200/csrc/copy_threads.h"

// A thread whose constructor fails the k-th time it is asked for, with either exception.
struct Failing {
    static int asked, fail_at;
    static bool no_memory;
    std::thread t;
    Failing() = default;
    template <class F>
    Failing(const F& f, int i) {
        if (++asked == fail_at || fail_at < 0) {
            if (no_memory) throw std::bad_alloc();
            throw std::system_error(std::make_error_code(std::errc::resource_unavailable_try_again));
        }
        t = std::thread(f, i);
    }
    Failing& operator=(Failing&&) = default;
    bool joinable() const { return t.joinable(); }
    void join() { t.join(); }
};
int Failing::asked = 0, Failing::fail_at = 0;
bool Failing::no_memory = false;

int main() {
    for (const bool no_memory : {false, true})
        for (const int fail_at : {-1, 0, 1, 2, 3}) {
            Failing::asked = 0;
            Failing::fail_at = fail_at;
            Failing::no_memory = no_memory;
            std::atomic<int> done[4] = {};
            ma::on_threads<4, Failing>([&](int i) { ++done[i]; });
            for (int i = 0; i < 4; ++i)
                if (done[i] != 1) {
                    std::printf("part %d done %d times (failure %d)\n", i, done[i].load(), fail_at);
                    return 1;
                }
        }
    return 0;
}
