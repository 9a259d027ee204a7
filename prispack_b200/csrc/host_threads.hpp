// Independent host work on several threads.
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <exception>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace prism {

// the host's threads, at most 16
inline unsigned host_threads() { return std::max(1u, std::min(std::thread::hardware_concurrency(), 16u)); }
// ... or PRISM_LAYOUT_THREADS, for the sweep layouts
inline unsigned layout_threads() {
    const char* e = std::getenv("PRISM_LAYOUT_THREADS");
    return e ? (unsigned)std::max(1, std::atoi(e)) : host_threads();
}

// fn(i) for i in [0, count) on up to `threads` host threads, the caller's among them (the items
// are independent: the results do not depend on the thread count).  Where the host has no more
// threads to give, those that started do the work.  An exception of an item reaches the caller
// once every thread has ended; items not yet begun are then left out.
template <typename F>
void host_parallel_for(uint32_t count, unsigned threads, F&& fn) {
    threads = std::min<unsigned>(threads, count);
    if (threads <= 1) {
        for (uint32_t i = 0; i < count; ++i) fn(i);
        return;
    }
    std::atomic<uint32_t> next{0};
    std::mutex lock;
    std::exception_ptr first;
    auto work = [&]() noexcept {
        try {
            for (uint32_t i = next++; i < count; i = next++) fn(i);
        } catch (...) {
            next = count;  // count + threads stays far below 2^32
            std::lock_guard<std::mutex> g(lock);
            if (!first) first = std::current_exception();
        }
    };
    std::vector<std::thread> pool;
    try {
        pool.reserve(threads - 1);
        for (unsigned t = 1; t < threads; ++t) pool.emplace_back(work);
    } catch (const std::system_error&) {
    } catch (const std::bad_alloc&) {
    }
    work();
    for (auto& t : pool) t.join();
    if (first) std::rethrow_exception(first);
}

}  // namespace prism
