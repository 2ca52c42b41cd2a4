// Work of a call split over host threads.
#pragma once
#include <cstddef>
#include <system_error>
#include <thread>
#include <utility>
#include <vector>

namespace gbt {

struct StartThread {
    template <typename F> std::thread operator()(F f) const { return std::thread(std::move(f)); }
};

// f(0), .., f(n - 1): part 0 on the calling thread, the others on a thread each, or on the calling thread from the
// first one on that cannot be started (a limit on threads). Every thread is joined before the call ends, whichever way.
// What f does on a thread may not throw.
template <typename F, typename Start = StartThread>
void in_parallel(size_t n, const F &f, Start start = Start())
{
    struct Pool {
        std::vector<std::thread> t;
        ~Pool() { for (auto &q : t) q.join(); }
    } pool;
    if (n == 0) return;
    pool.t.reserve(n - 1);
    size_t next = 1;
    try {
        for (; next < n; next++) pool.t.push_back(start([&f, next] { f(next); }));
    } catch (const std::system_error &) {
    }
    f(0);
    for (; next < n; next++) f(next);
}

}  // namespace gbt
