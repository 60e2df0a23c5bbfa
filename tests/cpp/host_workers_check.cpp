// host_workers_check.cpp -- host_workers.h on the host alone.  usage: host_workers_check CASE; prints "ok"
// and exits 0 when every check of the case holds.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <new>

#include "host_workers.h"

static std::atomic<long> allowed{-1};  // allocations left before operator new fails (negative: no limit)
void* operator new(std::size_t n) {
    if (allowed.load() >= 0 && allowed.fetch_sub(1) <= 0) {
        allowed.store(0);
        throw std::bad_alloc();
    }
    if (void* p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, std::size_t) noexcept { std::free(p); }

static int failures = 0;
#define CHECK(c)                                                                \
    do {                                                                        \
        if (!(c)) {                                                             \
            std::fprintf(stderr, "%s:%d: CHECK(%s)\n", __FILE__, __LINE__, #c); \
            ++failures;                                                         \
        }                                                                       \
    } while (0)

// All of the shared work is done, by however many threads could be had.
static void threads() {
    for (long limit : {-1L, 0L, 1L, 2L, 5L})
        for (int count : {1, 2, 5, 8}) {
            std::atomic<int> next{0}, calls{0}, done{0};
            auto work = [&](int) {
                ++calls;
                while (next.fetch_add(1) < 100) ++done;
            };
            allowed.store(limit);
            pt::run_workers(count, work);
            allowed.store(-1);
            CHECK(done.load() == 100);
            CHECK(calls.load() >= 1 && calls.load() <= count);
            CHECK(limit != -1 || calls.load() == count);
            CHECK(limit != 0 || calls.load() == 1);
        }
}

// One worker (the pipelined copies) for small calls and on one processor; else two at least.
static void counts() {
    using pt::pageable_workers;
    for (uint64_t n : {0ull, 1ull, (1ull << 16) - 1, 1ull << 16, (3ull << 15) - 1, 3ull << 15, 1ull << 24})
        for (unsigned t : {0u, 1u, 2u, 16u, 256u}) {
            CHECK(pageable_workers(n, t, true) == 1);
            CHECK((pageable_workers(n, t, false) > 1) == (n >= 3 << 15));
        }
    for (unsigned t : {0u, 1u, 2u, 3u, 4u, 5u}) CHECK(pageable_workers(1u << 24, t, false) == 2);
    CHECK(pageable_workers(1u << 24, 16, false) == 8 && pageable_workers(~0ull, 256, false) == 8);
    CHECK(pageable_workers(3u << 15, 64, false) == 3 && pageable_workers((4u << 15) - 1, 64, false) == 3);
    CHECK(pageable_workers(4u << 15, 64, false) == 4);
}

int main(int argc, char** argv) {
    const char* name = argc == 2 ? argv[1] : "";
    if (!std::strcmp(name, "threads")) threads();
    else if (!std::strcmp(name, "counts")) counts();
    else return 2;
    if (failures == 0) std::puts("ok");
    return failures ? 1 : 0;
}
