// swb_host.h -- host threads behind a C entry.  Plain C++, so that a host
// compiler checks it too.
#pragma once

#include <cstddef>
#include <thread>
#include <vector>

namespace swb {

// fn(0) .. fn(n - 1), each on a thread of its own but the last, which the caller
// runs, as it does those that no thread could be started for (a C caller must
// not see the exception).
template <class F>
void run_parts(size_t n, F &&fn) {
    std::vector<std::thread> th;
    size_t k = 0;
    try {
        for (th.reserve(n); k + 1 < n; ++k) th.emplace_back([&fn, k] { fn(k); });
    } catch (...) {
    }
    for (; k < n; ++k) fn(k);
    for (auto &t : th) t.join();
}

}  // namespace swb
