// adi_threads.hpp -- host set-up work over several threads.  Plain C++, shared with the host tests.
#pragma once

#include <exception>
#include <mutex>
#include <system_error>
#include <thread>
#include <vector>

namespace lss_gb300 {

// f(w) for the shares w = 0 .. shares - 1, each on a thread of its own as far as threads can be had (share 0 and
// the rest on the caller's).  Returns when all are done; an exception of a share is thrown here then.
template <typename F> void run_shares(unsigned shares, F &&f)
{
    std::exception_ptr failed;
    std::mutex lock;
    auto share = [&](unsigned w) {
        try {
            f(w);
        } catch (...) {
            const std::lock_guard<std::mutex> hold(lock);
            if (!failed) failed = std::current_exception();
        }
    };
    std::vector<std::thread> pool;
    unsigned next = 1;
    try {
        pool.reserve(shares);
        for (; next < shares; ++next) pool.emplace_back(share, next);
    } catch (const std::exception &) { // no more threads (or no memory for them)
    }
    share(0);
    for (unsigned w = next; w < shares; ++w) share(w);
    for (auto &t : pool) t.join();
    if (failed) std::rethrow_exception(failed);
}

} // namespace lss_gb300
