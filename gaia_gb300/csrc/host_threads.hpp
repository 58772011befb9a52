// Host work in parts on threads.
#pragma once
#include <exception>
#include <thread>
#include <vector>

namespace gaia {

// fn(0) ... fn(n - 1), each on a thread of its own where one can be started, on the calling
// thread where not. All have ended when it returns; the first exception of the lowest part is
// thrown again here, on the calling thread.
template <typename Fn>
void run_parts(int n, Fn&& fn) {
    std::vector<std::exception_ptr> error(static_cast<size_t>(n > 0 ? n : 0));
    auto one = [&](int k) noexcept {
        try {
            fn(k);
        } catch (...) {
            error[static_cast<size_t>(k)] = std::current_exception();
        }
    };
    std::vector<std::thread> threads;
    threads.reserve(error.size());
    int started = 1;  // part 0 is the caller's
    try {
        for (; started < n; ++started) threads.emplace_back(one, started);
    } catch (...) {  // no further thread to be had
    }
    if (n > 0) one(0);
    for (int k = started; k < n; ++k) one(k);
    for (auto& t : threads) t.join();
    for (auto& e : error)
        if (e) std::rethrow_exception(e);
}

}  // namespace gaia
