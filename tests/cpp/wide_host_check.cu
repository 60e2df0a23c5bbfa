// wide_host_check.cu -- the walk over four-wide records (wide.cuh) against the binary walk
// (traverse.cuh), both compiled for the host: no kernel is launched, no device is needed.
//
// usage: wide_host_check NODES TRIS RAYS
// Prints "rays N cut C unfit U rises R steps S differ D": rays whose 1/d is cut, rays that take the
// binary walk from the start, or when MinT rises, steps of the wide walk, and rays whose hit is not the
// binary walk's.
#include <cmath>
#include <cstdio>
#include <vector>

#include "pt_internal.h"
#include "wide.cuh"

using namespace pt;

template <class T>
static bool read_all(const char* path, std::vector<T>& v) {
    FILE* f = std::fopen(path, "rb");
    if (!f) return false;
    std::fseek(f, 0, SEEK_END);
    const long n = std::ftell(f);
    std::fseek(f, 0, SEEK_SET);
    v.resize((size_t)n / sizeof(T));
    const bool ok = std::fread(v.data(), sizeof(T), v.size(), f) == v.size();
    std::fclose(f);
    return ok;
}

struct Ray {
    float o[3], tmax, d[3];
    uint32_t flags;
};

template <int CAP, int SH, class Dir>
static bool walk(WideWalkT<CAP, SH>& k, const std::vector<WideNode>& wide, const std::vector<uint4>& nodes,
                 const std::vector<float4>& tris, const Dir& dir, long& steps) {
    while (k.cur != kWideDone) {
        ++steps;
        if (k.cur & kWideLeaf) {
            wide_faces(k, tris.data(), [&]() { return nodes.data(); }, dir, []() { return 0u; });
            if (k.done) break;
        } else if (!wide_visit(k, wide.data())) {
            return false;
        }
        wide_pop(k);
    }
    return true;
}

int main(int argc, char** argv) {
    std::vector<uint4> nodes;
    std::vector<float4> tris;
    std::vector<Ray> rays;
    if (argc != 4 || !read_all(argv[1], nodes) || !read_all(argv[2], tris) || !read_all(argv[3], rays)) {
        std::fprintf(stderr, "usage: %s NODES TRIS RAYS\n", argv[0]);
        return 2;
    }
    const uint32_t n = (uint32_t)(nodes.size() / 2);
    std::vector<uint32_t> depth(n, 0), wide_of(n, 0);
    uint32_t records = 0;
    for (uint32_t i = 0; i < n; ++i) {
        const uint4 b = nodes[2 * (size_t)i + 1];
        const bool leaf = (b.w & 0xFFFFu) != 0;
        if (!leaf) depth[i + 1] = depth[i + b.z] = depth[i] + 1;
        if (i == 0 || (!leaf && (depth[i] & 1u) == 0)) wide_of[i] = records++;
    }
    std::vector<WideNode> wide(records);
    float size = 0.f;
    for (int c = 0; c < 6; ++c) size = std::fmax(size, std::fabs(bitsf((&nodes[0].x)[c])));
    bool nested = size >= kWideSizeMin && size <= kWideSizeMax;
    for (uint32_t i = 0; i < n; ++i) {
        const bool leaf = (nodes[2 * (size_t)i + 1].w & 0xFFFFu) != 0;
        if (leaf) nested = wide_mark_leaf(nodes.data(), i, 0, tris.data()) && nested;
        if (i == 0 || (!leaf && (depth[i] & 1u) == 0))
            nested = wide_make(nodes.data(), wide_of.data(), i, size, 0, wide[wide_of[i]]) && nested;
    }
    if (!nested) {
        std::fprintf(stderr, "a box does not lie inside its parent's\n");
        return 3;
    }
    long cut = 0, unfit = 0, rises = 0, steps = 0, differ = 0;
    for (const Ray& ry : rays) {
        const bool any = (ry.flags & 1u) != 0;
        RayState r;
        ray_setup(r, ry.o[0], ry.o[1], ry.o[2], ry.d[0], ry.d[1], ry.d[2]);
        const TraceResult t = traverse<false>(nodes.data(), tris.data(), n, r, ry.tmax, any, false);
        WideWalkT<kWideStack, 0> k;
        wide_begin(k, ry.o[0], ry.o[1], ry.o[2], ry.d[0], ry.d[1], ry.d[2], ry.tmax, any, size);
        unfit += k.binary;
        const bool fits = !k.binary;
        cut += fits && k.cut;
        auto dir = [&](float& x, float& y, float& z) { x = ry.d[0]; y = ry.d[1]; z = ry.d[2]; };
        if (!walk(k, wide, nodes, tris, dir, steps)) {
            std::fprintf(stderr, "guard failure\n");
            return 4;
        }
        BinaryHit h{k.min_t, k.u, k.v, k.w, k.prim, k.leaf};
        if (k.binary) {
            rises += fits;
            const BinaryRay br{ry.o[0], ry.o[1], ry.o[2], ry.d[0], ry.d[1], ry.d[2], ry.tmax, any};
            if (!wide_binary_walk(nodes.data(), tris.data(), n, &br, &h)) return 4;
        }
        if (t.prim != h.prim || t.leaf != h.leaf || fbits(t.t) != fbits(h.t) || fbits(t.u) != fbits(h.u) ||
            fbits(t.v) != fbits(h.v) || fbits(t.w) != fbits(h.w))
            ++differ;
    }
    std::printf("rays %zu cut %ld unfit %ld rises %ld steps %ld differ %ld\n", rays.size(), cut, unfit, rises, steps, differ);
    return 0;
}
