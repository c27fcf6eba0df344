// run_shares (csrc/adi_threads.hpp) with threads and with a share that throws, or with an argument, where no
// thread can be had (address space used up): prints "ok" when every share ran once and the exception arrived.
#include "adi_threads.hpp"

#include <atomic>
#include <cstdio>
#include <fstream>
#include <new>
#include <sys/resource.h>

static bool all_once(unsigned shares)
{
    std::vector<std::atomic<int>> ran(shares);
    lss_gb300::run_shares(shares, [&](unsigned w) { ++ran[w]; });
    for (auto &r : ran)
        if (r != 1) return false;
    return true;
}

int main(int argc, char **)
{
    if (argc > 1) {
        long pages = 0;
        std::ifstream("/proc/self/statm") >> pages;
        const rlimit lim{static_cast<rlim_t>(pages) * 4096 + (1 << 20), RLIM_INFINITY}; // less than a thread's stack
        if (setrlimit(RLIMIT_AS, &lim)) return std::puts("setrlimit"), 1;
        bool none = false;
        try {
            std::thread([] {}).join();
        } catch (const std::system_error &) {
            none = true;
        }
        if (!none) return std::puts("a thread could be had"), 77;
        if (!all_once(9)) return std::puts("without threads"), 1;
    } else {
        if (!all_once(1) || !all_once(7)) return std::puts("threads"), 1;
        bool arrived = false;
        try {
            lss_gb300::run_shares(5, [](unsigned w) {
                if (w == 3) throw std::bad_alloc();
            });
        } catch (const std::bad_alloc &) {
            arrived = true;
        }
        if (!arrived) return std::puts("exception"), 1;
    }
    std::puts("ok");
    return 0;
}
