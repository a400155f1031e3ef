// Host loops over independent elements, split over a few threads.
#pragma once
#include <stdint.h>

#include <algorithm>
#include <system_error>
#include <thread>
#include <vector>

namespace vhsd {

// Calls f(begin, end) over a partition of [0, n), on at most 8 threads (the
// caller's among them) of at least `grain` elements each.  f must not throw.
// Where no thread can be started the caller does that part too.
template <typename F>
void parallel_ranges(int64_t n, int64_t grain, F f) {
    const int64_t cores = std::max<int64_t>(1, std::thread::hardware_concurrency());
    const int64_t parts = std::max<int64_t>(1, std::min<int64_t>({8, cores, n / grain}));
    std::vector<std::thread> threads;
    threads.reserve((size_t)parts);
    for (int64_t k = 1; k < parts; k++) {
        const int64_t b = n * k / parts, e = n * (k + 1) / parts;
        try {
            threads.emplace_back([&f, b, e] { f(b, e); });
        } catch (const std::system_error&) {
            f(b, e);
        }
    }
    f((int64_t)0, n / parts);
    for (std::thread& t : threads) t.join();
}

}  // namespace vhsd
