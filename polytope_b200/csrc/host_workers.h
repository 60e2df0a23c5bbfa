// host_workers.h -- a few host threads that share one call's work (pt_trace's pageable arrays, abi.cpp).
#pragma once

#include <algorithm>
#include <cstdint>
#include <thread>

#if defined(__linux__)
#include <sched.h>
#endif

namespace pt {

constexpr int kWorkers = 8;
// Below, the threads cost more than they bring.  Pipelined copies / workers on a B200's host of 16 threads, medians
// of several runs (ms): 65,536 rays 0.35 / 0.32 to 0.44, 80,000 0.40 / 0.47 to 0.51, 90,000 0.43 / 0.36 to 0.54
// (two workers), 98,304 0.46 / 0.34 to 0.43 (three), 131,072 0.58 / 0.38 (four).
constexpr uint64_t kPageableRays = 3 << 15;

// Whether this process may run on one processor only.
inline bool one_processor() {
#if defined(__linux__)
    cpu_set_t set;
    if (sched_getaffinity(0, sizeof set, &set) == 0 && CPU_COUNT(&set) == 1) return true;
#endif
    return std::thread::hardware_concurrency() == 1;
}

// Workers for n rays on a host of that many threads (0: not known): half the threads, but two at least, and two
// chunks of 16,384 rays or more for each.  With one worker nothing overlaps, nor do several on one
// processor; such calls take the pipelined copies instead.  1 M rays on a B200's host, process bound to
// one / two / four of its 16 threads: pipelined 5.5 / 5.2 / 5.3 ms, eight workers 7.1 / 3.7 / 2.2, two
// workers on two processors 3.6.
inline int pageable_workers(uint64_t n, unsigned threads, bool one) {
    if (n < kPageableRays || one) return 1;
    return (int)std::min<uint64_t>({(uint64_t)kWorkers, std::max(2u, threads / 2), n >> 15});
}

// work(0) in the calling thread and work(1) .. work(count - 1) in threads of their own, or fewer where the
// system gives no more of them; returns when all have ended.  Throws nothing if `work` does not: a thread
// that cannot be had, for want of memory too, must not end the process while others run.
template <class Work>
void run_workers(int count, Work& work) {
    std::thread pool[kWorkers - 1];
    int started = 0;
    try {
        while (started < std::min(count, kWorkers) - 1) {
            const int w = started + 1;
            pool[started] = std::thread([&work, w] { work(w); });
            started = w;
        }
    } catch (...) {
    }
    work(0);
    for (int k = 0; k < started; ++k) pool[k].join();
}

}  // namespace pt
