// wide.cuh -- the four-wide records of a tree (WideNode) and the walk over them, which gives every
// ray the hit of the binary walk (traverse.cuh), bit for bit.
//
// One record stands for a binary node and its two children: its slots are the four grandchildren (a
// child that is a leaf takes one slot and leaves the next one empty).  Their boxes are kept on an 8-bit
// grid of the record, rounded outwards.  A visit tests the four at once and pushes the children it
// hits, with their near values, in the order in which the binary walk would pop them; an entry is
// dropped when it is popped if its near value lies beyond the running MinT.
//
// Why the hits are the binary walk's.  That walk tests a leaf's faces when every box on the way passes
// at the MinT of its pop.  Where each box lies inside its parent's (checked when the records are
// made), the products (b - o) * (1/d) of a box lie between its parent's, as IEEE subtraction,
// multiplication, min and max are monotone, and MinT only falls: so a leaf is tested exactly when its
// own box passes at its own pop.
//   * The leaves come in the binary walk's order: at each of the three split planes of a record the
//     high side comes first where 1/d is negative.
//   * No leaf that the binary walk tests is left out: the grid test lets through whatever the exact
//     one does (wide_begin and wide_visit give the bounds).
//   * A face of a leaf that the binary walk would not test can be tested, but not be accepted: before
//     a leaf's first accepted face counts, its box is tested exactly (wide_faces).
//   * MinT rises when an accepted t rounds an ulp above it (the face test bounds T by MinT * det);
//     such a ray starts again on the binary walk.
//
// What bounds it: the chain of dependent record loads and the instructions of a visit.  On the 1.3
// M-face microbench a ray takes 11 visits instead of 39 binary steps.  64 bytes a record (two 256-bit
// loads a lane) instead of 128 with full-precision boxes (four): gathering 128-byte records one a lane
// runs at 52 G records/s on a B200, 64-byte ones at 128 G (L2-resident), and 11 visits at 52 G/s would
// by themselves cap that microbench at 4.9 Grays/s.
#pragma once

#include "traverse.cuh"
#include "two_level.cuh"

namespace pt {

constexpr uint32_t kWideLeaf = 0x80000000u;   // slot is a leaf: faces (ref >> 28) & 7 from ref & kWideIndex
constexpr uint32_t kWideIndex = 0x0FFFFFFFu;
constexpr uint32_t kWideBig = 7u;             // leaf of more than 6 faces: the index names its binary node
constexpr uint32_t kWideEmpty = kWideLeaf;    // empty slot: a leaf without faces (visited or entered by no walk)
constexpr uint32_t kWideDone = 0xFFFFFFFFu;   // no slot's reference: WideWalkT::cur at the end of a walk
constexpr int kWideStack = 96;                // 3 entries a level of records, at most 31 levels, a fourth on the
                                              // last, and an exit marker (trees of PT_TRAVERSAL_STACK - 2 levels)

// Slot s of axis k covers [org[k] + step * (1 + q_lo 2^-15), org[k] + step * (1 + q_hi 2^-15)], where
// step (a power of two) is 2^15 grid steps: the planes' bytes go into the mantissa of a number in [1,
// 1.0078) by one byte permutation and meet the ray in one fused multiply-add.
struct alignas(64) WideNode {
    float org[3];
    uint32_t step_xy;        // upper halves of the x and y steps (x in the upper 16 bits)
    float step_z;
    uint32_t flips;          // three bits per octant of 1/d: high side first at the root / the low / the high child
    uint32_t plane[6];       // low x, high x, low y, high y, low z, high z: one byte a slot
    uint32_t ref[4];         // record, or leaf (kWideLeaf)
};
static_assert(sizeof(WideNode) == 64, "a record is half a 128-byte line");

// Rays that the grid test is proved for (and trees: kWideSizeMin, pt_internal.h); others take the binary
// walk.  `size`: the largest coordinate of the tree's boxes.
constexpr float kWideScaleMin = 8.8817842e-16f, kWideScaleMax = 1.1258999e15f;  // least 1/d times size: 2^-50, 2^50
constexpr float kWideFar = 2097152.f;         // |origin| / size: 2^21
constexpr float kWideSlope = 1.1258999e15f;   // 2^50: |1/d| of an axis over the least one, larger ones are cut there

// ---- making the records -----------------------------------------------------------------------------

// Whether the faces of a leaf (vertices v0, v1, v2 of each record) lie in its box; notes the leaf's node
// in the record's last word (wide_leaf_passes).
PT_HD bool wide_mark_leaf(const uint4* nodes, uint32_t ni, uint32_t face_base, float4* tris) {
    const uint4 a = nodes[2 * (size_t)ni], b = nodes[2 * (size_t)ni + 1];
    const float lo[3] = {bitsf(a.x), bitsf(a.y), bitsf(a.z)}, hi[3] = {bitsf(a.w), bitsf(b.x), bitsf(b.y)};
    bool ok = true;
    for (uint32_t j = 0; j < (b.w & 0xFFFFu); ++j) {
        float4* q = tris + 3 * (size_t)(face_base + b.z + j);
        const float v[9] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z, q[1].w, q[2].x};
        for (int c = 0; c < 9; ++c) ok = ok && lo[c % 3] <= v[c] && v[c] <= hi[c % 3];
        q[2].w = bitsf(ni);
    }
    return ok;
}

// A slot's reference to binary node `ni` whose second half is `b`; wide_of: the record of each binary
// node that has one; face_base: face record of the tree's first face.
PT_HD uint32_t wide_ref(uint32_t ni, const uint4& b, const uint32_t* wide_of, uint32_t face_base) {
    const uint32_t nf = b.w & 0xFFFFu;
    if (nf == 0) return wide_of[ni];
    return nf < kWideBig && b.z + face_base <= kWideIndex ? kWideLeaf | nf << 28 | (b.z + face_base)
                                                          : kWideLeaf | kWideBig << 28 | ni;
}

PT_HD void wide_box(const uint4* nodes, uint32_t i, float lo[3], float hi[3], uint4& b) {
    const uint4 a = nodes[2 * (size_t)i];
    b = nodes[2 * (size_t)i + 1];
    lo[0] = bitsf(a.x); lo[1] = bitsf(a.y); lo[2] = bitsf(a.z);
    hi[0] = bitsf(a.w); hi[1] = bitsf(b.x); hi[2] = bitsf(b.y);
}

// Record of binary node `ni`.  Returns whether every box of its slots and of the nodes between lies
// inside its parent's.
PT_HD bool wide_make(const uint4* nodes, const uint32_t* wide_of, uint32_t ni, float size, uint32_t face_base, WideNode& w) {
    float lo[4][3], hi[4][3], plo[3], phi[3];
    bool full[4] = {false, false, false, false}, ok = true;
    uint32_t axis[3] = {0, 0, 0};
    uint4 pb;
    for (int s = 0; s < 4; ++s) w.ref[s] = kWideEmpty;
    wide_box(nodes, ni, plo, phi, pb);
    auto inside = [&](const float* l, const float* h, const float* ol, const float* oh) {
        for (int k = 0; k < 3; ++k) ok = ok && ol[k] <= l[k] && l[k] <= h[k] && h[k] <= oh[k];
    };
    auto slot = [&](int s, uint32_t i, const float* ol, const float* oh) {
        uint4 b;
        wide_box(nodes, i, lo[s], hi[s], b);
        inside(lo[s], hi[s], ol, oh);
        full[s] = true;
        w.ref[s] = wide_ref(i, b, wide_of, face_base);
    };
    if ((pb.w & 0xFFFFu) != 0) {  // the root of a tree of one leaf
        slot(0, ni, plo, phi);
    } else {
        axis[0] = pb.w >> 16;
        for (int side = 0; side < 2; ++side) {
            const uint32_t ci = side ? ni + pb.z : ni + 1;
            float clo[3], chi[3];
            uint4 cb;
            wide_box(nodes, ci, clo, chi, cb);
            if ((cb.w & 0xFFFFu) != 0) {
                slot(2 * side, ci, plo, phi);
                continue;
            }
            inside(clo, chi, plo, phi);
            axis[1 + side] = cb.w >> 16;
            slot(2 * side, ci + 1, clo, chi);
            slot(2 * side + 1, ci + cb.z, clo, chi);
        }
    }
    float step[3];
    for (int k = 0; k < 3; ++k) {
        // grid step: a power of two, at least 2^-22 of the tree's size (so that the record's origin, an
        // integer number of steps, is exact), with the box within 252 steps
        const float need = fmul(fmaxf(fsub(phi[k], plo[k]), fmul(size, 6.0081482e-05f /* 252 * 2^-22 */)), 0.003968254f /* 1/252 */);
        const float g = bitsf((fbits(need) + 0x7FFFFFu) & 0x7F800000u);
        const float inv = bitsf(0x7F000000u - fbits(g));  // 1 / g
        const float first = fsub(floorf(fmul(plo[k], inv)), 1.f);
        w.org[k] = fmul(fsub(first, 32768.f), g);
        step[k] = fmul(g, 32768.f);
        uint32_t ql = 0, qh = 0;
        for (int s = 0; s < 4; ++s) {
            // a 32nd of a step outwards on top of the rounding: it covers the rounding errors of these
            // differences (at most 2^-16 of a step) and, in wide_visit, those that go with the step
            // empty: low plane beyond the high one on every axis, which stops all rays but those from afar,
            // whose slack (wide_visit) is wider than the record; they pass over the reference (kWideEmpty)
            uint32_t a = 255u, b = 0u;
            if (full[s]) {
                const float x = floorf(fsub(fsub(fmul(lo[s][k], inv), first), 0.03125f));
                const float y = ceilf(fadd(fsub(fmul(hi[s][k], inv), first), 0.03125f));
                if (!(x >= 0.f && y <= 255.f)) ok = false;
                a = (uint32_t)fmaxf(x, 0.f);
                b = (uint32_t)fminf(y, 255.f);
            }
            ql |= a << (8 * s);
            qh |= b << (8 * s);
        }
        w.plane[2 * k] = ql;
        w.plane[2 * k + 1] = qh;
    }
    w.step_xy = (fbits(step[0]) & 0xFFFF0000u) | fbits(step[1]) >> 16;
    w.step_z = step[2];
    w.flips = 0;
    for (uint32_t oct = 0; oct < 8; ++oct)
        for (uint32_t k = 0; k < 3; ++k) w.flips |= ((oct >> axis[k]) & 1u) << (3 * oct + k);
    return ok;
}

// ---- the walk ---------------------------------------------------------------------------------------

// Stack of one lane's walk: {near, reference} pairs, the first SH in shared memory (pair i of the lane at
// base[i * stride], consecutive lanes on consecutive pairs), the rest in local memory: here, or LENT by
// the kernel (WideSpill::pairs).
template <int N, bool LENT>
struct WidePairs {
    uint2 spill[N];
};
template <int N>
struct WidePairs<N, true> {
    uint2* spill;
};
template <int CAP, int SH, bool LENT>
struct WideStack : WidePairs<CAP - SH, LENT> {
    uint2* base;
    uint32_t stride;
    PT_HD void put(int i, uint32_t ref, float near_t) {
        uint2 v;
        v.x = fbits(near_t);
        v.y = ref;
        if constexpr (SH > 0) {
            if (i < SH) { base[i * stride] = v; return; }
        }
        this->spill[i - SH] = v;
    }
    PT_HD uint2 get(int i) const {
        if constexpr (SH > 0) {
            if (i < SH) return base[i * stride];
        }
        return this->spill[i - SH];
    }
};

template <int CAP = kWideStack, int SH = 0, bool LENT = false>
struct WideWalkT {
    RayState r;         // ix, iy, iz cut at kWideSlope times the least of them (cut: some was)
    float min_t;
    uint32_t prim, leaf;
    float u, v, w;
    bool any, done, cut;
    bool binary;        // the hit is the binary walk's to find (unsuitable ray, or MinT rose)
    uint32_t cur;       // what comes next: a record, a leaf (kWideLeaf), or kWideDone
    int sp;
    WideStack<CAP, SH, LENT> stack;
};

// Cuts 1/d of a ray (r set up for direction d) for a tree of the given size; false for the rays that the
// grid test is not proved for: with a NaN, an origin 2^21 tree sizes away or a direction of extreme
// length.
//
// 1/d is cut at 2^50 times the least of the three.  A plane ahead of the origin is then met sooner, so
// near only falls.  The far plane lies a 32nd of a grid step, at least 2^-27 of the tree's size, beyond
// the box: a ray whose origin is not past the box meets it no sooner than 2^23 * size * least, and
// every box of the tree ends before 2 (1 + 2^21) * size * least on the axis of the least 1/d.
PT_HD bool wide_cut(RayState& r, bool& cut, float size) {
    const float ax = fabs_(r.ix), ay = fabs_(r.iy), az = fabs_(r.iz);
    const float least = fminf(fminf(ax, ay), az), most = fmaxf(fmaxf(ax, ay), az), top = fmul(least, kWideSlope);
    const float far_o = fmaxf(fmaxf(fabs_(r.ox), fabs_(r.oy)), fabs_(r.oz));
    const float scale = fmul(least, size);
    const bool fits = scale >= kWideScaleMin && scale <= kWideScaleMax && top < bitsf(0x7F800000u) &&
                      far_o <= fmul(kWideFar, size) && ax == ax && ay == ay && az == az && r.ox == r.ox && r.oy == r.oy && r.oz == r.oz;
    cut = !(most <= top);
    if (cut) {
        r.ix = ax > top ? bitsf(fbits(top) | (fbits(r.ix) & 0x80000000u)) : r.ix;
        r.iy = ay > top ? bitsf(fbits(top) | (fbits(r.iy) & 0x80000000u)) : r.iy;
        r.iz = az > top ? bitsf(fbits(top) | (fbits(r.iz) & 0x80000000u)) : r.iz;
    }
    return fits;
}

// Starts the walk of the ray in k.r at record 0.  Rays that wide_cut refused (fits), and those with a
// negative or NaN far bound (the binary walk's test of an origin strictly inside a box cannot matter
// for the others), are done at once, `binary` set.
template <int CAP, int SH, bool LENT>
PT_HD void wide_start(WideWalkT<CAP, SH, LENT>& k, float tmax, bool any, bool fits) {
    fits = fits && tmax >= 0.f;
    k.min_t = tmax;
    k.prim = kPrimNone;
    k.leaf = kPrimNone;
    k.u = k.v = k.w = 0.f;
    k.any = any;
    k.done = k.binary = !fits;
    k.cur = fits ? 0u : kWideDone;
    k.sp = 0;
}

template <int CAP, int SH, bool LENT>
PT_HD void wide_begin(WideWalkT<CAP, SH, LENT>& k, float ox, float oy, float oz, float dx, float dy, float dz, float tmax, bool any,
                      float size) {
    ray_setup(k.r, ox, oy, oz, dx, dy, dz);
    const bool fits = wide_cut(k.r, k.cut, size);
    wide_start(k, tmax, any, fits);
}

// Rays (or paths) that a warp takes from the counter, `left` being those not handed out when it last took
// some: twice `chunk` while there are plenty, kWideFew when each warp has little left to do, so that all end
// together.  Against `chunk` throughout (64), on a B200, with frames twice as large: 16.7 M rays 5130 -> 5075
// us, 1 M occlusion rays 514 -> 484, 1 M on box faces 430 -> 420, a 641x479x4 frame 2.72 -> 2.53 ms, 24 uneven
// renders 25.0 -> 24.5 ms; few from `share` on instead of twice that 518 on the occlusion rays; shares of the
// rest (left / (2 warps)) 575, as early takers keep too much.  Few of 8 from there on: within 0.6 % of 16, but
// a 320x240x8 frame 7 % slower; of 32: 2 to 5 % slower, that frame 16 %.  Two-level queries were 1 % slower
// with it and take `chunk` throughout.
constexpr uint32_t kWideFew = 16;
PT_HD uint32_t wide_take(uint32_t left, uint32_t warps, uint32_t chunk) {
    const uint32_t share = warps * chunk;
    return left > 8 * share ? 2 * chunk : left > 4 * share ? chunk : left > 2 * share ? 32u : kWideFew;
}

// The binary walk of a whole ray, out of line: the hit in *out, false on a guard failure; stack has room for
// kStackCap entries.  Nodes come in two 128-bit loads: ptxas 12.9 does not compile the 256-bit load in a
// function that is not inlined.
struct BinaryRay { float ox, oy, oz, dx, dy, dz, tmax; bool any; };
struct BinaryHit { float t, u, v, w; uint32_t prim, leaf; };
PT_COLD bool wide_binary_walk(const uint4* nodes, const float4* tris, uint32_t num_nodes, const BinaryRay* ray, BinaryHit* out,
                              uint32_t* stack) {
    RayWalkT<1, 0> k;
    walk_begin(k, ray->ox, ray->oy, ray->oz, ray->dx, ray->dy, ray->dz, ray->tmax, ray->any, false);
    const bool inside = needs_inside_test(k.r, ray->tmax);
    bool ok = true;
    int sp = 0;
    stack[sp++] = 0;
    while (ok && !k.done && sp > 0) {
        const uint32_t ni = stack[--sp];
        if (ni >= num_nodes) { ok = false; break; }
        const uint4 a = ldg(nodes + 2 * (size_t)ni), b = ldg(nodes + 2 * (size_t)ni + 1);
        if (!box_hits(k.r, bitsf(a.x), bitsf(a.y), bitsf(a.z), bitsf(a.w), bitsf(b.x), bitsf(b.y), k.min_t, inside)) continue;
        const uint32_t nf = b.w & 0xFFFFu;
        if (nf > 0) {
            walk_leaf<false>(k, tris, b.z, nf);
            continue;
        }
        if (sp + 2 > kStackCap) { ok = false; break; }
        const bool neg = neg_on(k.r, b.w >> 16);
        stack[sp++] = neg ? ni + 1 : ni + b.z;
        stack[sp++] = neg ? ni + b.z : ni + 1;
    }
    out->t = k.min_t;
    out->u = k.u; out->v = k.v; out->w = k.w;
    out->prim = k.prim; out->leaf = k.leaf;
    return ok;
}
PT_HD bool wide_binary_walk(const uint4* nodes, const float4* tris, uint32_t num_nodes, const BinaryRay* ray, BinaryHit* out) {
    uint32_t stack[kStackCap];
    return wide_binary_walk(nodes, tris, num_nodes, ray, out, stack);
}

// A kernel's local memory for one lane's walks.  A ray that goes to the binary walk has ended its own, so that
// walk's ray, hit and stacks (TL: of both levels) lie where its stack was.  Without that, and with 100 pairs,
// the kernels' frames were 1184 to 1536 bytes; above 1024 the context's local memory grows by 46 to 98
// MiB at the first launch, also that of a call that is to allocate none (pt_render_noalloc).
template <int SH, bool TL>
union WideSpill {
    uint2 pairs[kWideStack - SH];
    struct {
        BinaryRay ray;
        BinaryHit hit;
        uint32_t stack[kStackCap + (TL ? kTopStackCap : 0)];
    } rest;
};

// The next entry that MinT does not rule out (or kWideDone), into k.cur.
template <int CAP, int SH, bool LENT>
PT_HD void wide_pop(WideWalkT<CAP, SH, LENT>& k) {
    k.cur = kWideDone;
    while (k.sp > 0) {
        const uint2 e = k.stack.get(--k.sp);
        if (!(bitsf(e.x) > k.min_t)) {
            k.cur = e.y;
            return;
        }
    }
}

PT_HD float wide_byte(uint32_t word, int s) {  // 1 + byte s of word * 2^-15
#ifdef __CUDA_ARCH__
    return bitsf(__byte_perm(word, 0x3F800000u, 0x7604u | s << 4));
#else
    return bitsf(0x3F800000u | ((word >> (8 * s)) & 0xFFu) << 8);
#endif
}

// a * b + c on two numbers at once
PT_HD void wide_fma2(float a0, float a1, float b0, float b1, float c0, float c1, float& d0, float& d1) {
#ifdef __CUDA_ARCH__
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(pack2(a0, a1)), "l"(pack2(b0, b1)), "l"(pack2(c0, c1)));
    unpack2(d, d0, d1);
#else
    d0 = ffma(a0, b0, c0);
    d1 = ffma(a1, b1, c1);
#endif
}

// Visits record k.cur: tests its four boxes and pushes the children hit.  False on a guard failure.
//
// Plane f in [1, 1.0078) of an axis meets the ray at f * A + B, A = step * i, B = (org - o) * i.  The
// errors of B, of the sum and of the exact test's own product are at most 2.5 * 2^-23 |B| + 2.5 *
// 2^-23 |A|.  The second part is 0.01 of a grid step, within the 32nd by which planes lie outwards; for
// the first, near takes B - 2^-21 |B| and far B + 2^-20 |B|, which also holds the factor 1 + 2 gamma_3
// = 1 + 3 * 2^-23 that the exact test puts on far; far's A has that factor too.  Nothing overflows:
// |A| <= 2^9 size * 2^50 least, |B| <= 2^22 size * 2^50 least, and size * least <= 2^50.
template <int CAP, int SH, bool LENT>
PT_HD bool wide_visit(WideWalkT<CAP, SH, LENT>& k, const WideNode* __restrict__ wide) {
    const uint4* p = (const uint4*)(wide + k.cur);
    uint4 w0, w1, w2, w3;
    ldg_node(p, w0, w1);
    ldg_node(p + 2, w2, w3);
    const float eps_n = -4.7683716e-07f, eps_f = 9.5367432e-07f, gm = bitsf(PT_GAMMA_MUL_BITS);
    const float Ax = fmul(bitsf(w0.w & 0xFFFF0000u), k.r.ix), Ay = fmul(bitsf(w0.w << 16), k.r.iy), Az = fmul(bitsf(w1.x), k.r.iz);
    const float Bx = fmul(fsub(bitsf(w0.x), k.r.ox), k.r.ix), By = fmul(fsub(bitsf(w0.y), k.r.oy), k.r.iy),
                Bz = fmul(fsub(bitsf(w0.z), k.r.oz), k.r.iz);
    const float Nx = ffma(fabs_(Bx), eps_n, Bx), Ny = ffma(fabs_(By), eps_n, By), Nz = ffma(fabs_(Bz), eps_n, Bz);
    const float Fx = ffma(fabs_(Bx), eps_f, Bx), Fy = ffma(fabs_(By), eps_f, By), Fz = ffma(fabs_(Bz), eps_f, Bz);
    const float Gx = fmul(Ax, gm), Gy = fmul(Ay, gm), Gz = fmul(Az, gm);
    const bool nx = k.r.neg & 1u, ny = k.r.neg & 2u, nz = k.r.neg & 4u;
    const uint32_t qnx = nx ? w1.w : w1.z, qfx = nx ? w1.z : w1.w;
    const uint32_t qny = ny ? w2.y : w2.x, qfy = ny ? w2.x : w2.y;
    const uint32_t qnz = nz ? w2.w : w2.z, qfz = nz ? w2.z : w2.w;
    bool h[4];
    float n[4];
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int s = 0; s < 4; ++s) {
        float x0, y0, z0, x1, y1, z1;
        wide_fma2(wide_byte(qnx, s), wide_byte(qny, s), Ax, Ay, Nx, Ny, x0, y0);
        wide_fma2(wide_byte(qfx, s), wide_byte(qfy, s), Gx, Gy, Fx, Fy, x1, y1);
        wide_fma2(wide_byte(qnz, s), wide_byte(qfz, s), Az, Gz, Nz, Fz, z0, z1);
#if defined(__CUDA_ARCH__) && PT_PACKED_BOX
        n[s] = fmaxf(max3f(x0, y0, z0), 0.f);
        h[s] = n[s] <= fminf(min3f(x1, y1, z1), k.min_t);
#else
        n[s] = fmaxf(fmaxf(x0, y0), fmaxf(z0, 0.f));
        h[s] = n[s] <= fminf(fminf(x1, y1), fminf(z1, k.min_t));
#endif
    }
    // stack positions: the child visited first lies on top
    const uint32_t f = w1.y >> (3u * k.r.neg);
    const int c0 = h[0], c1 = h[1], c2 = h[2], c3 = h[3];
    const int low = c0 + c1, high = c2 + c3;
    const int at_low = k.sp + ((f & 1u) ? 0 : high), at_high = k.sp + ((f & 1u) ? low : 0);
    const int p0 = at_low + ((f & 2u) ? 0 : c1), p1 = at_low + ((f & 2u) ? c0 : 0);
    const int p2 = at_high + ((f & 4u) ? 0 : c3), p3 = at_high + ((f & 4u) ? c2 : 0);
    if constexpr (SH >= 4) {
        if (k.sp + 4 <= SH) {
            uint2* b = k.stack.base;
            const uint32_t st = k.stack.stride;
            if (c0) b[p0 * st] = make_uint2(fbits(n[0]), w3.x);
            if (c1) b[p1 * st] = make_uint2(fbits(n[1]), w3.y);
            if (c2) b[p2 * st] = make_uint2(fbits(n[2]), w3.z);
            if (c3) b[p3 * st] = make_uint2(fbits(n[3]), w3.w);
            k.sp += low + high;
            return true;
        }
    }
    if (k.sp + low + high > CAP) return false;
    if (c0) k.stack.put(p0, w3.x, n[0]);
    if (c1) k.stack.put(p1, w3.y, n[1]);
    if (c2) k.stack.put(p2, w3.z, n[2]);
    if (c3) k.stack.put(p3, w3.w, n[3]);
    k.sp += low + high;
    return true;
}

// Whether the binary walk would test the leaf of face (v0, v1, v2) at far bound min_t: the face's own
// box lies in the leaf's, so where it passes the leaf's does; else the leaf's own decides.  `dir` gives
// the ray's direction where its 1/d was cut.
template <class K, class Nodes, class Dir>
PT_HD bool wide_leaf_passes(const K& k, float4 q0, float4 q1, float4 q2, const Nodes& nodes, float min_t, const Dir& dir) {
    RayState r;
    r.ox = k.r.ox; r.oy = k.r.oy; r.oz = k.r.oz;
    r.ix = k.r.ix; r.iy = k.r.iy; r.iz = k.r.iz;
    r.neg = 0;
    if (k.cut) {
        float dx, dy, dz;
        dir(dx, dy, dz);
        r.ix = frcp(dx); r.iy = frcp(dy); r.iz = frcp(dz);
    } else {
        const float lx = fminf(fminf(q0.x, q0.w), q1.z), ly = fminf(fminf(q0.y, q1.x), q1.w), lz = fminf(fminf(q0.z, q1.y), q2.x);
        const float hx = fmaxf(fmaxf(q0.x, q0.w), q1.z), hy = fmaxf(fmaxf(q0.y, q1.x), q1.w), hz = fmaxf(fmaxf(q0.z, q1.y), q2.x);
        if (box_hits_fast(r, lx, ly, lz, hx, hy, hz, min_t)) return true;
    }
    const uint32_t ni = fbits(q2.w);
    const uint4* q = nodes() + 2 * (size_t)ni;
    const uint4 a = ldg(q), b = ldg(q + 1);
    return box_hits(r, bitsf(a.x), bitsf(a.y), bitsf(a.z), bitsf(a.w), bitsf(b.x), bitsf(b.y), min_t, false);
}

// The faces of leaf k.cur in leaf order, as the binary walk tests them; sets k.done when the walk ends
// here (an any-hit ray accepted a face, or MinT rose and `binary` is set).  `nodes` gives the binary nodes,
// which only large leaves and boxes to be tested exactly need, `face_base` the face record of the tree's first
// face (large leaves).  Returns whether a face was accepted.
template <int CAP, int SH, bool LENT, class Nodes, class Dir, class Base>
PT_HD bool wide_faces(WideWalkT<CAP, SH, LENT>& k, const float4* __restrict__ tris, const Nodes& nodes, const Dir& dir, const Base& face_base) {
    uint32_t at = k.cur & kWideIndex, n = (k.cur >> 28) & 7u;
    if (n == kWideBig) {
        uint4 a, b;
        ldg_node(nodes() + 2 * (size_t)at, a, b);
        at = b.z + face_base();
        n = b.w & 0xFFFFu;
    }
    const float before = k.min_t;
    bool passes = false;
    for (uint32_t j = 0; j < n; ++j) {
        const size_t ti = 3 * (size_t)(at + j);
        const float4 q0 = ldg_face(tris + ti), q1 = ldg_face(tris + ti + 1), q2 = ldg_face(tris + ti + 2);
        float t, u, v, w;
        if (wald(k.r, q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w, q2.x, k.min_t, t, u, v, w)) {
            if (!passes) {
                if (!wide_leaf_passes(k, q0, q1, q2, nodes, before, dir)) return false;
                passes = true;
            }
            if (t > k.min_t && !k.any) { k.binary = k.done = true; return false; }
            k.min_t = t;
            k.prim = fbits(q2.y);
            k.leaf = at + j;
            k.u = u; k.v = v; k.w = w;
            if (k.any) { k.done = true; return true; }
        }
    }
    return passes;
}

// ---- two-level scenes -------------------------------------------------------------------------------
//
// The top-level tree's records come first in the array, then those of every geometry's tree; a table of
// the instances lies before record 0 (WideInstance, pt_internal.h).  A walk starts in world space; at a
// top-level leaf the ray is carried into its instance's object space, an exit marker is pushed and the
// walk goes on at the geometry's first record.  Boxes and faces are tested in traverse_two_level's order;
// the instance's own box is tested exactly, at the MinT of the entry, before the first face accepted in
// it counts (wide_instance_passes; where it fails, traverse_two_level takes the whole ray).  The world
// ray is set up again only when a top-level record follows an exit: most often another instance does, or
// the walk's end.
constexpr uint32_t kWideExit = 0xFFFFFFFEu;  // exit marker (its leaf bit set: no record)

// WideInstance of instance ii: {root, size, node, 0}.
PT_HD uint4 wide_instance(const WideNode* wide, uint32_t ii) { return ldg((const uint4*)wide - 1 - ii); }

// A world ray in the object space of an instance.
template <class V>
PT_HD void wide_to_object(const DeviceInstance* inst, V& o, V& d) {
    const float4* w2o = (const float4*)inst->w2o;
    const float4 m0 = ldg(w2o), m1 = ldg(w2o + 1), m2 = ldg(w2o + 2);
    const float m[12] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w, m2.x, m2.y, m2.z, m2.w};
    const V wo = o, wd = d;
    to_object(m, wo.x, wo.y, wo.z, 1.0f, o.x, o.y, o.z);
    to_object(m, wd.x, wd.y, wd.z, 0.0f, d.x, d.y, d.z);
}

// A lane at an exit marker or a top-level leaf: leaves its instance (inside), if it is in one, or passes over
// an empty slot.  Returns whether k.cur is then an instance to enter; else it is a top-level record, another
// empty slot (for the next crossing), or kWideDone.
template <int CAP, int SH, bool LENT>
PT_HD bool wide_cross(WideWalkT<CAP, SH, LENT>& k, bool& inside) {
    if (k.cur == kWideExit || k.cur == kWideEmpty) {
        inside = false;
        wide_pop(k);
    }
    return (k.cur & kWideLeaf) && k.cur != kWideEmpty && k.cur != kWideDone;
}

// Enters the instance whose tree starts at record root, with its object ray in k.r.  False when that ray is
// none for the records (wide_cut's fits; done and `binary` set) or the stack is full (done set).
template <int CAP, int SH, bool LENT>
PT_HD bool wide_enter(WideWalkT<CAP, SH, LENT>& k, uint32_t root, bool fits) {
    if (!fits || k.sp >= CAP) {
        k.done = true;
        k.binary = !fits;
        return false;
    }
    k.stack.put(k.sp++, kWideExit, 0.f);
    k.cur = root;
    return true;
}

// Whether the box of instance ii passes for world ray o, d at far bound min_t.
PT_HD bool wide_instance_passes(const WideNode* __restrict__ wide, const uint4* __restrict__ top, uint32_t ii, float ox, float oy, float oz,
                                float dx, float dy, float dz, float min_t) {
    const uint4* q = top + 2 * (size_t)wide_instance(wide, ii).z;
    const uint4 a = ldg(q), b = ldg(q + 1);
    RayState r;
    r.ox = ox; r.oy = oy; r.oz = oz;
    r.ix = frcp(dx); r.iy = frcp(dy); r.iz = frcp(dz);
    return box_hits(r, bitsf(a.x), bitsf(a.y), bitsf(a.z), bitsf(a.w), bitsf(b.x), bitsf(b.y), min_t, false);
}

// The whole ray by traverse_two_level, out of line: the hit in *out, its instance in *inst; false on a guard
// failure; stack has room for kTopStackCap + kStackCap entries.
PT_COLD bool wide_two_level_walk(const TwoLevelView* v, const BinaryRay* ray, BinaryHit* out, uint32_t* inst, uint32_t* stack) {
    const TwoLevelHit h = traverse_two_level_on<false, kStackCap, true>(stack, stack + kTopStackCap, *v, ray->ox, ray->oy, ray->oz, ray->dx,
                                                                        ray->dy, ray->dz, ray->tmax, ray->any);
    out->t = h.r.t;
    out->u = h.r.u; out->v = h.r.v; out->w = h.r.w;
    out->prim = h.r.prim; out->leaf = h.r.leaf;
    *inst = h.inst;
    return !h.r.overflow;
}
PT_HD bool wide_two_level_walk(const TwoLevelView* v, const BinaryRay* ray, BinaryHit* out, uint32_t* inst) {
    uint32_t stack[kTopStackCap + kStackCap];
    return wide_two_level_walk(v, ray, out, inst, stack);
}

}  // namespace pt
