// Loops over ranges on the host's threads
#pragma once
#include <algorithm>
#include <cstddef>
#include <exception>
#include <new>
#include <thread>
#include <vector>

namespace nbh {

// f(begin, end) over [0, n) in runs of `run` and more, one per host thread (at
// most `most`); where no thread can be had the caller does its run itself
template <class F>
void parallel_ranges(size_t n, size_t run, size_t most, const F& f) {
    const size_t nt =
        std::max<size_t>(1, std::min({(size_t)std::thread::hardware_concurrency(), most, n / run}));
    const size_t chunk = (n + nt - 1) / nt;
    std::vector<std::thread> pool;
    try {
        pool.reserve(nt);
    } catch (const std::bad_alloc&) {
        return f((size_t)0, n);
    }
    for (size_t b = chunk; b < n; b += chunk) {
        const size_t e = std::min(n, b + chunk);
        try {
            pool.emplace_back([&f, b, e]() { f(b, e); });
        } catch (const std::exception&) {
            f(b, e);
        }
    }
    f((size_t)0, std::min(n, chunk));
    for (auto& th : pool) th.join();
}

}  // namespace nbh
