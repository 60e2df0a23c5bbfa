// wide_refs_check.cu -- the references of a record's slots at the ends of their range (wide.cuh), compiled
// for the host: no kernel is launched, no device is needed.  Prints "ok" and exits 0 when all hold.
#include <cstdio>

#include "pt_internal.h"
#include "wide.cuh"

using namespace pt;

static int failures = 0;
#define CHECK(c)                                                                \
    do {                                                                        \
        if (!(c)) {                                                             \
            std::fprintf(stderr, "%s:%d: CHECK(%s)\n", __FILE__, __LINE__, #c); \
            ++failures;                                                         \
        }                                                                       \
    } while (0)

static uint4 leaf(uint32_t first, uint32_t faces) {
    uint4 b{};
    b.z = first;
    b.w = faces;
    return b;
}

int main() {
    // leaves named by their node: more than six faces, or faces beyond the 28 bits of an index
    for (uint32_t ni : {0u, 1u, kWideNodesMost / 2, kWideNodesMost - 2, kWideNodesMost - 1})
        for (const uint4& b : {leaf(0, 7), leaf(0, 65535), leaf(kWideIndex + 1, 1), leaf(kWideIndex, 7)}) {
            const uint32_t r = wide_ref(ni, b, nullptr, 0);
            CHECK(r & kWideLeaf);
            CHECK(((r >> 28) & 7u) == kWideBig);
            CHECK((r & kWideIndex) == ni);
            CHECK(r != kWideDone && r != kWideExit);
        }
    // leaves named by their first face, also with the faces of other trees before theirs
    for (uint32_t faces = 1; faces < kWideBig; ++faces)
        for (uint32_t base : {0u, 5u}) {
            const uint32_t r = wide_ref(3, leaf(kWideIndex - base, faces), nullptr, base);
            CHECK((r & kWideLeaf) && ((r >> 28) & 7u) == faces && (r & kWideIndex) == kWideIndex);
            CHECK(r != kWideDone && r != kWideExit);
        }
    if (failures == 0) std::puts("ok");
    return failures ? 1 : 0;
}
