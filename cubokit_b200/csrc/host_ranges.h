// Work over a range of host items on several threads.
#pragma once

#include <algorithm>
#include <cstddef>
#include <thread>
#include <vector>

namespace cubo {

// body(first, last) over `count` items in ranges of at least `grain` on up to eight host threads, the caller's among them
// (a thread costs about 20 us to start; a complex value takes about 2 ns to convert on one).  body must not throw.  Where no
// memory or thread is left for another one, the caller takes the ranges that have none.
template <typename F>
void parallel_ranges(size_t count, size_t grain, const F &body) {
    const size_t most = std::max(1u, std::min(8u, std::thread::hardware_concurrency()));
    const size_t parts = std::max<size_t>(1, std::min(most, count / grain));
    std::vector<std::thread> threads;
    size_t started = 1;
    try {
        threads.reserve(parts);
        for (; started < parts; started++)
            threads.emplace_back([&body, count, parts, part = started] {
                body(count * part / parts, count * (part + 1) / parts);
            });
    } catch (...) {  // std::system_error, or std::bad_alloc for the vector or a thread's own state
    }
    body(0, count / parts);
    for (size_t part = started; part < parts; part++) body(count * part / parts, count * (part + 1) / parts);
    for (auto &t : threads) t.join();
}

}  // namespace cubo
