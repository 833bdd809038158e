// Work shared by a few host threads.
#pragma once
#include <algorithm>
#include <cstddef>
#include <exception>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace gvx {

// Starts a thread; a test puts one that fails in its place.
struct StartThread {
    template <class F>
    std::thread operator()(F&& f) const { return std::thread(static_cast<F&&>(f)); }
};

// Runs `work` on up to `most` threads, this one among them, and returns when all have ended.  `work`
// takes its pieces from a shared counter, so fewer threads do the same: where the system starts no
// more, the ones there are go on.  What a thread throws, the caller gets (the first of them), once no
// thread runs any more: an exception that left a thread, or a running thread's handle destroyed on
// the way out, would end the process.
template <class F, class Start = StartThread>
void run_threads(size_t most, const F& work, const Start& start = Start{}) {
    const size_t n = std::max<size_t>(1, std::min<size_t>(most, std::max(1u, std::thread::hardware_concurrency())));
    std::exception_ptr first;
    std::mutex lock;
    auto guarded = [&]() noexcept {
        try {
            work();
        } catch (...) {
            std::lock_guard<std::mutex> g(lock);
            if (!first) first = std::current_exception();
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(n - 1);
    for (size_t t = 1; t < n; t++) {
        try {
            pool.push_back(start(guarded));
        } catch (const std::system_error&) {
            break;
        }
    }
    guarded();
    for (auto& t : pool) t.join();
    if (first) std::rethrow_exception(first);
}

}  // namespace gvx
