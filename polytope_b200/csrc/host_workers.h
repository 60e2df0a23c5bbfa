// host_workers.h -- a few host threads that share one call's work (pt_trace's pageable arrays, abi.cpp).
#pragma once

#include <algorithm>
#include <cstdint>
#include <thread>

namespace pt {

constexpr int kWorkers = 8;
constexpr uint64_t kPageableRays = 1 << 16;  // below, the threads cost more than they bring

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
