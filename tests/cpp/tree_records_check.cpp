// tree_records_check.cpp -- which trees validate_tree numbers for four-wide records, on the host (linked
// against the library; no device is used).
//
// usage: tree_records_check CASE; prints "ok" and exits 0 when every check of the case holds.
#include <cstdio>
#include <cstring>
#include <vector>

#include "pt_internal.h"

using namespace pt;

static int failures = 0;
#define CHECK(c)                                                                \
    do {                                                                        \
        if (!(c)) {                                                             \
            std::fprintf(stderr, "%s:%d: CHECK(%s)\n", __FILE__, __LINE__, #c); \
            ++failures;                                                         \
        }                                                                       \
    } while (0)

static pt_bvh_node leaf(uint32_t first, uint16_t faces) {
    pt_bvh_node n{};
    for (int k = 0; k < 3; ++k) n.bb_max[k] = 1.f;
    n.offset = first;
    n.num_faces = faces;
    return n;
}
static pt_bvh_node inner(uint32_t high) {
    pt_bvh_node n = leaf(high, 0);
    return n;
}

struct Result {
    int rc;
    uint32_t depth = ~0u, records = ~0u;
    std::vector<uint32_t> wide_of{7u};
    explicit Result(const std::vector<pt_bvh_node>& nodes, uint32_t faces) {
        rc = validate_tree(nodes.data(), (uint32_t)nodes.size(), faces, &depth, &wide_of, &records);
    }
    bool none() const { return rc == PT_OK && wide_of.empty() && records == 0; }
};

// Trees whose nodes are all reached and whose leaves hold faces of their own are numbered.
static void numbered() {
    const Result one({leaf(0, 3)}, 3);
    CHECK(one.rc == PT_OK && one.records == 1 && one.wide_of == std::vector<uint32_t>{0});
    const Result r({inner(4), inner(2), leaf(3, 2), leaf(1, 1), leaf(0, 1)}, 5);
    CHECK(r.rc == PT_OK && r.depth == 2 && r.records == 1);
    CHECK((r.wide_of == std::vector<uint32_t>{0, kNotWide, kNotWide, kNotWide, kNotWide}));
}

// A node that no parent reaches has never been looked at, its face range included: no records, and the
// tree is accepted as one without them is.
static void unreached() {
    for (const pt_bvh_node& stray : {leaf(0x10000000u, 65535), leaf(0, 1), inner(2), inner(0xFFFFFFFFu)}) {
        const Result middle({inner(3), leaf(0, 1), stray, leaf(1, 1)}, 2);
        CHECK(middle.none() && middle.depth == 1);
        const Result tail({inner(2), leaf(0, 1), leaf(1, 1), stray}, 2);
        CHECK(tail.none() && tail.depth == 1);
        const Result after_leaf({leaf(0, 2), stray}, 2);
        CHECK(after_leaf.none() && after_leaf.depth == 0);
    }
}

// Two leaves over the same faces, the whole range or a part of it, in either order: no records, and the
// tree is accepted as one without them is.  Leaves that meet without sharing a face are numbered.
static void shared_faces() {
    struct { uint32_t a, na, b, nb; bool shares; } const cases[] = {
        {0, 2, 0, 2, true}, {0, 3, 2, 2, true}, {2, 2, 0, 3, true}, {0, 4, 1, 2, true}, {1, 2, 0, 4, true},
        {0, 2, 2, 2, false}, {2, 2, 0, 2, false}, {0, 1, 3, 1, false}};
    for (const auto& c : cases) {
        const Result r({inner(2), leaf(c.a, (uint16_t)c.na), leaf(c.b, (uint16_t)c.nb)}, 4);
        CHECK(r.rc == PT_OK && r.depth == 1);
        CHECK(c.shares ? r.none() : r.records == 1 && r.wide_of.size() == 3);
    }
}

int main(int argc, char** argv) {
    const char* name = argc == 2 ? argv[1] : "";
    if (!std::strcmp(name, "numbered")) numbered();
    else if (!std::strcmp(name, "unreached")) unreached();
    else if (!std::strcmp(name, "shared_faces")) shared_faces();
    else return 2;
    if (failures == 0) std::puts("ok");
    return failures ? 1 : 0;
}
