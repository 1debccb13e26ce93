// Host work spread over threads of one call.
#pragma once

#include <exception>
#include <thread>
#include <vector>

namespace mtb {

// f(0) .. f(n - 1), each once and on a thread of its own, the last one on the caller's. Where no thread can be
// started (none left, no memory) the caller runs what remains. Returns when all of them have ended and then
// rethrows the first exception by index: nothing leaves while a thread runs.
template <class F>
void run_threads(int n, F f) {
    std::vector<std::exception_ptr> failed(n);
    std::vector<std::thread> pool;
    pool.reserve(n);
    auto one = [&](int i) noexcept {
        try {
            f(i);
        } catch (...) {
            failed[i] = std::current_exception();
        }
    };
    int i = 0;
    try {
        for (; i + 1 < n; i++) pool.emplace_back(one, i);
    } catch (...) {  // f(i) has not been started
    }
    for (; i < n; i++) one(i);
    for (auto& t : pool) t.join();
    for (auto& e : failed)
        if (e) std::rethrow_exception(e);
}

}  // namespace mtb
