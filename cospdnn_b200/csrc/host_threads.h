// Host work on several threads whose failures end as error codes.
#pragma once

#include <atomic>
#include <cstdio>
#include <new>
#include <thread>
#include <vector>

namespace cospdnn {

// The first failure of several threads, kept without an allocation.
struct FirstError {
    std::atomic<int> code{0};
    char message[256] = "";
    void set(int c, const char *m) noexcept {
        int none = 0;
        if (code.compare_exchange_strong(none, c)) std::snprintf(message, sizeof(message), "%s", m);
    }
};

// body() on n threads, the caller's among them; on fewer when threads or memory
// are short.  What a body throws is the error `nomem`: nothing leaves a thread.
template <typename Body>
void on_threads(int n, int nomem, FirstError &err, Body body) noexcept {
    auto guarded = [&]() noexcept {
        try {
            body();
        } catch (const std::bad_alloc &) {
            err.set(nomem, "build: out of host memory");
        } catch (...) {
            err.set(nomem, "build: host failure on a thread");
        }
    };
    std::vector<std::thread> threads;
    try {
        threads.reserve(n > 1 ? n - 1 : 0);  // no throw from the vector once a thread runs
        for (int i = 1; i < n; ++i) threads.emplace_back(guarded);
    } catch (...) {
    }
    guarded();
    for (std::thread &t : threads) t.join();
}

}  // namespace cospdnn
