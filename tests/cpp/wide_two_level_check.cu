// wide_two_level_check.cu -- the walk over a two-level scene's four-wide records (wide.cuh) against
// traverse_two_level, both compiled for the host and linked against the library for the scene's layout: no
// kernel is launched, no device is needed.
//
// usage: wide_two_level_check RAYS SEED
// Six octahedra, one of radius 50 and five of radius 0.12 close together beside it, and RAYS rays for each of three
// kinds of origins: near, 2^11 to 2^14 scene sizes away along the diagonal, and up to kWideFar of them in all
// directions.  Prints "rays N hits H empty E differ D": rays that hit something, empty slots that walks met
// at the top level, and rays whose hit is not traverse_two_level's.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "pt_internal.h"
#include "shade.cuh"
#include "wide.cuh"

using namespace pt;

static float largest(const pt_bvh_node& n) {
    float m = 0.f;
    for (int k = 0; k < 3; ++k) m = std::fmax(m, std::fmax(std::fabs(n.bb_min[k]), std::fabs(n.bb_max[k])));
    return m;
}

struct Scene {
    HostScene h;
    std::vector<WideInstance> memory;  // the instances' entries, instance 0 last, then the records
    const WideNode* wide;
    float size;
    TwoLevelView view;
};

static bool make(const std::vector<pt_mesh_desc>& meshes, Scene& s) {
    pt_scene_desc d{};
    d.meshes = meshes.data();
    d.num_meshes = (uint32_t)meshes.size();
    HostScene& h = s.h;
    if (prepare_two_level_host(&d, h) != PT_OK || h.wide_of.empty()) return false;
    const size_t ni = h.instances.size();
    s.memory.resize(ni + 4 * (size_t)h.num_wide);
    WideNode* wide = (WideNode*)(s.memory.data() + ni);
    const uint4 *nodes = (const uint4*)h.nodes.data(), *top = (const uint4*)h.tlas.data();
    float4* tris = (float4*)h.tris.data();
    bool ok = true;
    s.size = largest(h.tlas[0]);
    for (uint32_t i = 0; i < h.tlas.size(); ++i) {
        if (h.top_wide_of[i] != kNotWide) ok = wide_make(top, h.top_wide_of.data(), i, s.size, 0, wide[h.top_wide_of[i]]) && ok;
        if (h.tlas[i].num_faces == 1) s.memory[ni - 1 - h.tlas[i].offset].node = i;
    }
    for (const HostScene::Geometry& g : h.geometries) {
        const uint4* gn = nodes + 2 * (size_t)g.node_base;
        const uint32_t* number = h.wide_of.data() + g.node_base;
        for (uint32_t i = 0; i < g.num_nodes; ++i) {
            if (h.nodes[g.node_base + i].num_faces) ok = wide_mark_leaf(gn, i, g.face_base, tris) && ok;
            if (number[i] != kNotWide) ok = wide_make(gn, number, i, largest(h.nodes[g.node_base]), g.face_base, wide[number[i]]) && ok;
        }
    }
    for (size_t i = 0; i < ni; ++i) {
        WideInstance& w = s.memory[ni - 1 - i];
        w.root = h.wide_of[h.instances[i].node_base];
        w.size = largest(h.nodes[h.instances[i].node_base]);
    }
    s.wide = wide;
    s.view = TwoLevelView{nodes, tris, (uint32_t)h.nodes.size(), top, (uint32_t)h.tlas.size(), h.instances.data(), false};
    return ok;
}

// The kernels' walk of one ray.  False on a guard failure.
static bool walk(const Scene& s, const BinaryRay& ray, BinaryHit& hit, uint32_t& hit_inst, long& empty) {
    const TwoLevelView& v = s.view;
    WideWalkT<kWideStack, 0> k;
    wide_begin(k, ray.ox, ray.oy, ray.oz, ray.dx, ray.dy, ray.dz, ray.tmax, ray.any, s.size);
    bool inside = false, sure = true;
    uint32_t inst = 0;
    float entry = 0.f;
    auto dir = [&](float& x, float& y, float& z) {
        F3 o = f3(0.f, 0.f, 0.f), d = f3(ray.dx, ray.dy, ray.dz);
        wide_to_object(v.inst + inst, o, d);
        x = d.x; y = d.y; z = d.z;
    };
    hit_inst = 0;
    while (k.cur != kWideDone) {
        if (!(k.cur & kWideLeaf)) {
            if (!wide_visit(k, s.wide)) return false;
            wide_pop(k);
        } else if (k.cur == kWideExit || !inside) {
            F3 o = f3(ray.ox, ray.oy, ray.oz), d = f3(ray.dx, ray.dy, ray.dz);
            empty += k.cur == kWideEmpty;
            const bool enters = wide_cross(k, inside);
            if (k.cur == kWideDone) break;
            const uint32_t ii = k.cur & kWideIndex;
            float size = s.size;
            uint32_t root = 0;
            if (enters) {
                inst = ii;
                entry = k.min_t;
                sure = false;
                wide_to_object(v.inst + ii, o, d);
                const uint4 wi = wide_instance(s.wide, ii);
                root = wi.x;
                size = bitsf(wi.y);
            }
            ray_setup(k.r, o.x, o.y, o.z, d.x, d.y, d.z);
            const bool fits = wide_cut(k.r, k.cut, size);
            if (enters) {
                inside = wide_enter(k, root, fits);
                if (!inside) {
                    if (!k.binary) return false;
                    break;
                }
            }
        } else {
            const DeviceInstance& in = v.inst[inst];
            if (wide_faces(k, v.tris, [&]() { return v.nodes + 2 * (size_t)in.node_base; }, dir, [&]() { return in.face_base; })) {
                k.prim += in.prim_base;
                hit_inst = inst;
                if (!sure && !wide_instance_passes(s.wide, v.top, inst, ray.ox, ray.oy, ray.oz, ray.dx, ray.dy, ray.dz, entry))
                    k.binary = k.done = true;
                sure = true;
            }
            if (k.done) break;
            wide_pop(k);
        }
    }
    hit = BinaryHit{k.min_t, k.u, k.v, k.w, k.prim, k.leaf};
    return !k.binary || wide_two_level_walk(&v, &ray, &hit, &hit_inst);
}

int main(int argc, char** argv) {
    if (argc != 3) return 2;
    const long count = std::atol(argv[1]);
    std::mt19937 rng((uint32_t)std::atol(argv[2]));
    std::uniform_real_distribution<float> unit(0.f, 1.f);
    std::normal_distribution<float> normal;

    static const float x[] = {1, -1, 0, 0, 0, 0}, y[] = {0, 0, 1, -1, 0, 0}, z[] = {0, 0, 0, 0, 1, -1};
    static const uint32_t f0[] = {0, 2, 1, 3, 2, 1, 3, 0}, f1[] = {2, 1, 3, 0, 0, 2, 1, 3}, f2[] = {4, 4, 4, 4, 5, 5, 5, 5};
    std::vector<pt_mesh_desc> meshes;
    for (int m = 0; m < 6; ++m) {
        pt_mesh_desc d{};
        d.x = x; d.y = y; d.z = z;
        d.num_vertices = 6;
        d.fv0 = f0; d.fv1 = f1; d.fv2 = f2;
        d.num_faces = 8;
        d.material = PT_MAT_LAMBERT;
        const float r = m == 0 ? 50.f : 0.12f;
        const float at[3] = {m == 0 ? 0.f : 30.f + 0.3f * (m % 3), m == 0 ? 0.f : 30.f + 0.25f * (m / 3), m == 0 ? 0.f : 30.f + 0.2f * (m % 2)};
        for (int k = 0; k < 3; ++k) {
            d.object_to_world[5 * k] = r;
            d.object_to_world[4 * k + 3] = at[k];
            d.world_to_object[5 * k] = 1.f / r;
            d.world_to_object[4 * k + 3] = -at[k] / r;
        }
        d.object_to_world[15] = d.world_to_object[15] = 1.f;
        meshes.push_back(d);
    }
    Scene s;
    if (!make(meshes, s)) {
        std::fprintf(stderr, "no records: %s\n", pt_last_error());
        return 3;
    }
    long rays = 0, hits = 0, empty = 0, differ = 0;
    for (int kind = 0; kind < 3; ++kind)
        for (long i = 0; i < count; ++i, ++rays) {
            F3 d = f3(normal(rng), normal(rng), normal(rng));
            float far = 200.f * unit(rng);
            if (kind == 1) {
                const float side = i % 8 < 4 ? 1.f : -1.f;
                d = f3(side + 1e-6f * normal(rng), side + 1e-6f * normal(rng), side + 1e-6f * normal(rng));
                far = 1.5e5f + 8e5f * unit(rng);
            } else if (kind == 2) {
                far = std::exp2(10.f + 17.f * unit(rng));
            }
            const float len = std::sqrt(d.x * d.x + d.y * d.y + d.z * d.z);
            const float to[3] = {30.f + 0.3f * (rng() % 3), 30.f + 0.25f * (rng() % 2), 30.f + 0.2f * (rng() % 2)};
            const BinaryRay ray{to[0] - far * d.x / len, to[1] - far * d.y / len, to[2] - far * d.z / len, d.x / len, d.y / len, d.z / len,
                                bitsf(0x7F800000u), i % 4 != 0};
            const TwoLevelHit t = traverse_two_level<false>(s.view, ray.ox, ray.oy, ray.oz, ray.dx, ray.dy, ray.dz, ray.tmax, ray.any);
            BinaryHit h;
            uint32_t inst = 0;
            if (!walk(s, ray, h, inst, empty)) {
                std::fprintf(stderr, "guard failure\n");
                return 4;
            }
            hits += t.r.prim != kPrimNone;
            if (t.r.prim != h.prim || t.r.leaf != h.leaf || fbits(t.r.t) != fbits(h.t) || fbits(t.r.u) != fbits(h.u) ||
                fbits(t.r.v) != fbits(h.v) || fbits(t.r.w) != fbits(h.w) || (h.prim != kPrimNone && inst != t.inst))
                ++differ;
        }
    std::printf("rays %ld hits %ld empty %ld differ %ld\n", rays, hits, empty, differ);
    return 0;
}
