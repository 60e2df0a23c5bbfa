// trace.cu -- ray-query kernels (Scene::intersect replacement) for sm_100a.
//
// Queries of scenes that have four-wide records (wide.cuh) run in trace_wide_kernel; counted queries and
// trees without records walk the binary nodes in the reference's order (traverse.cuh).  Rays and hits
// stream through HBM once (32 B in, 16 B out per ray); records, nodes and faces stay resident in the
// 126 MB L2 for scenes up to a few million faces.

#include <algorithm>
#include <type_traits>

#include "launch.h"
#include "traverse.cuh"
#include "two_level.cuh"
#include "shade.cuh"
#include "wide.cuh"

namespace pt {

template <bool COUNT>
__global__ void __launch_bounds__(128) trace_kernel(const uint4* __restrict__ nodes, const float4* __restrict__ tris,
                                                    uint32_t num_nodes, const float4* __restrict__ rays,
                                                    uint4* __restrict__ hits, uint64_t n, uint32_t* node_tests,
                                                    uint32_t* tri_tests, int* err, bool exact_tree) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 r0 = ld_stream(rays + 2 * i);
    const float4 r1 = ld_stream(rays + 2 * i + 1);
    RayState rs;
    ray_setup(rs, r0.x, r0.y, r0.z, r1.x, r1.y, r1.z);
    const bool any = (__float_as_uint(r1.w) & 1u) != 0;
    const TraceResult tr = traverse<COUNT>(nodes, tris, num_nodes, rs, r0.w, any, exact_tree);
    uint4 h;
    h.x = tr.prim;
    h.y = __float_as_uint(tr.t);
    h.z = __float_as_uint(tr.u);
    h.w = __float_as_uint(tr.v);
    if (tr.overflow) {
        h.x = 0xFFFFFFFEu;
        atomicExch(err, 1);
    }
    st_stream(hits + i, h);
    if (COUNT) {
        if (node_tests) node_tests[i] = tr.nodes;
        if (tri_tests) tri_tests[i] = tr.tris;
    }
}

// Persistent variant: a grid sized to the SMs; each warp takes chunks of kChunk rays from a global
// counter and refills a lane as soon as its ray finishes, so lanes stay busy despite rays of very
// different cost (any-hit rays stop early, closest-hit rays run long).  Each pass of the outer loop
// steps the walking lanes node by node until PT_LEAF_BATCH_TRACE of them hold a leaf or have
// ended, then tests those leaves' faces together (walk_round, traverse.cuh).  A ray's own node and face order is exactly
// the reference's; only which rays share a warp, and when a lane waits, changes.
// 8 blocks of 128 per SM (64 registers, almost no spills) measured 2.6 % faster than 9 blocks at
// 56 registers, where the warp vote's live state spilled.
// Node steps a walking lane takes between ballots (a lane that reaches a leaf stops early).
// Measured on a B200 (16.7 M microbench rays, two runs each, same box): 1 step 2142 -> 2 steps
// (before the node-step changes); with them 2 steps 2428, 3 steps 2470, 4 steps 2067 Mrays/s.
#ifndef PT_TRACE_STEPS
#define PT_TRACE_STEPS 3
#endif
template <bool COUNT, int SH>
__global__ void __launch_bounds__(128, 8) trace_persistent_kernel(const uint4* __restrict__ nodes,
                                                               const float4* __restrict__ tris, uint32_t num_nodes,
                                                               const float4* __restrict__ rays, uint4* __restrict__ hits,
                                                               uint64_t n, uint32_t* node_tests, uint32_t* tri_tests,
                                                               int* err, unsigned long long* counter, uint32_t kChunk,
                                                               bool exact_tree) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t lt_mask = (1u << lane) - 1u;
    uint64_t pool_next = 0, pool_end = 0;
    bool exhausted = false, active = false;
    uint64_t idx = 0;
    __shared__ uint32_t sstack[SH > 0 ? SH * 128 : 1];
    RayWalkT<kStackCap, SH> k;
    k.stack.base = sstack + threadIdx.x;
    k.stack.stride = 128;
    while (true) {
        // refill idle lanes from the warp's chunk
        const uint32_t need = __ballot_sync(0xFFFFFFFFu, !active);
        if (need && !exhausted && pool_next >= pool_end) {
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(counter, (unsigned long long)kChunk);
            base = __shfl_sync(0xFFFFFFFFu, base, 0);
            if (base >= n) {
                exhausted = true;
            } else {
                pool_next = base;
                pool_end = base + kChunk < n ? base + kChunk : n;
            }
        }
        if (need) {
            const uint64_t avail = pool_end - pool_next;
            const uint32_t rank = __popc(need & lt_mask);
            if (!active && rank < avail) {
                idx = pool_next + rank;
                const float4 r0 = ld_stream(rays + 2 * idx);
                const float4 r1 = ld_stream(rays + 2 * idx + 1);
                walk_begin(k, r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, r0.w, (__float_as_uint(r1.w) & 1u) != 0, exact_tree);
                active = true;
            }
            const uint64_t took = (uint64_t)__popc(need) < avail ? (uint64_t)__popc(need) : avail;
            pool_next += took;
        }
        if (!__any_sync(0xFFFFFFFFu, active)) {
            if (exhausted || pool_next >= pool_end) {
                if (exhausted) break;
            }
            continue;
        }
        uint32_t leaf_off = 0, leaf_n = 0;
        bool ok, at_leaf;
        if constexpr (PT_LEAF_BATCH_TRACE > 0) {
            // walk_round (traverse.cuh), written out here: the compiler allocates this form with
            // fewer spills, which measured 9 % faster on the 1.3 M-face microbench; each lane takes
            // up to PT_TRACE_STEPS node steps per ballot (fewer votes; a lane that reaches a leaf
            // skips the rest)
            ok = true;
            at_leaf = false;
            const uint32_t cand = __ballot_sync(0xFFFFFFFFu, active && k.sp > 0);
            const int want = __popc(cand) < PT_LEAF_BATCH_TRACE ? __popc(cand) : PT_LEAF_BATCH_TRACE;
            // the round's node steps, with the box test chosen once for the warp when every ray in
            // it takes the min/max form (box_mode 0) instead of per step: 2437 vs 2337 Mrays/s on a
            // B200 (1.3 M faces, 16.7 M rays)
            auto round = [&](auto fast) {
                constexpr bool kFast = decltype(fast)::value;
                while (true) {
                    const bool walking = active && ok && !at_leaf && k.sp > 0;
                    const uint32_t w = __ballot_sync(0xFFFFFFFFu, walking);
                    if (w == 0 || __popc(cand & ~w) >= want) break;
                    if (walking) {
                        int r = walk_step<COUNT, kFast>(k, nodes, num_nodes, leaf_off, leaf_n);
#pragma unroll
                        for (int extra = 1; extra < PT_TRACE_STEPS; ++extra)
                            if (r == 0 && k.sp > 0) r = walk_step<COUNT, kFast>(k, nodes, num_nodes, leaf_off, leaf_n);
                        at_leaf = r > 0;
                        ok = r >= 0;
                    }
                }
            };
            if (__all_sync(0xFFFFFFFFu, !active || k.box_mode == 0))
                round(std::true_type{});
            else
                round(std::false_type{});
        } else {
            ok = !active || walk_to_leaf<COUNT>(k, nodes, num_nodes, leaf_off, leaf_n);
            at_leaf = active && ok && leaf_n > 0;
        }
        if (at_leaf) walk_leaf<COUNT>(k, tris, leaf_off, leaf_n);
        if (active) {
            if (!ok || k.done || k.sp == 0) {
                uint4 h;
                h.x = ok ? k.prim : 0xFFFFFFFEu;
                h.y = __float_as_uint(k.min_t);
                h.z = __float_as_uint(k.u);
                h.w = __float_as_uint(k.v);
                if (!ok) atomicExch(err, 1);
                st_stream(hits + idx, h);
                if (COUNT) {
                    if (node_tests) node_tests[idx] = k.nodes;
                    if (tri_tests) tri_tests[idx] = k.tris;
                }
                active = false;
            }
        }
    }
}

// ---- four-wide walk ---------------------------------------------------------------------------------

__global__ void __launch_bounds__(128) wide_make_kernel(const uint4* __restrict__ nodes, const uint32_t* __restrict__ wide_of,
                                                        uint32_t num_nodes, float size, uint32_t face_base, WideNode* __restrict__ wide,
                                                        float4* __restrict__ tris, uint32_t* outside) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= num_nodes) return;
    bool ok = true;
    if (tris && (nodes[2 * (size_t)i + 1].w & 0xFFFFu) != 0) ok = wide_mark_leaf(nodes, i, face_base, tris);
    if (wide_of[i] != 0xFFFFFFFFu) {
        WideNode w;
        ok = wide_make(nodes, wide_of, i, size, face_base, w) && ok;
        const uint4* src = (const uint4*)&w;
        uint4* dst = (uint4*)(wide + wide_of[i]);
#pragma unroll
        for (int k = 0; k < 4; ++k) dst[k] = src[k];
    }
    if (!ok) atomicExch(outside, 1u);
}

cudaError_t launch_wide_make(const void* nodes, const uint32_t* wide_of, uint32_t num_nodes, float size, uint32_t face_base,
                             void* wide, void* tris, uint32_t* outside, cudaStream_t s) {
    if (!num_nodes) return cudaSuccess;
    wide_make_kernel<<<(num_nodes + 127) / 128, 128, 0, s>>>((const uint4*)nodes, wide_of, num_nodes, size, face_base,
                                                             (WideNode*)wide, (float4*)tris, outside);
    return cudaGetLastError();
}

// Ray queries over the four-wide records, persistent as above.  A lane's state is what its walk meets
// next (WideWalkT::cur): records are visited together until PT_WIDE_BATCH lanes hold a leaf (or all that
// still walk), then those test their faces together; lanes whose ray has ended wait until PT_WIDE_REFILL
// of them store their hits and take new rays together.  A batch smaller than the resident warps spreads
// over all of them, a few rays a warp, and needs neither counter nor memset.
// TL: a two-level scene (v): lanes at a top-level leaf or an exit marker enter or leave their instance
// PT_WIDE_ENTERS at a time.
template <int SH, bool TL>
__global__ void __launch_bounds__(128, TL ? PT_WIDE_TL_BLOCKS : PT_WIDE_BLOCKS) trace_wide_kernel(const WideNode* __restrict__ wide, const uint4* __restrict__ nodes,
                                                            const float4* __restrict__ tris, uint32_t num_nodes,
                                                            const uint4* __restrict__ top, uint32_t num_top,
                                                            const DeviceInstance* __restrict__ inst, const float4* __restrict__ rays, uint4* __restrict__ hits, uint32_t n,
                                                            int* err, unsigned long long* counter, uint32_t chunk, float size) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warp = blockIdx.x * 4 + (threadIdx.x >> 5);
    // this warp's rays: first its own chunk, then those that the counter hands out (base + take <= n + 2^13)
    uint32_t pool_next = warp * chunk < n ? warp * chunk : n, pool_end = n - pool_next < chunk ? n : pool_next + chunk;
    bool exhausted = false, loaded = false;  // loaded: the lane holds a ray whose hit is not yet stored
    uint32_t idx = 0;
    __shared__ uint2 sstack[SH > 0 ? SH * 128 : 1];
    __shared__ uint32_t sinst[TL ? 128 : 1];  // the instance that the lane's walk is in, and MinT at its entry
    __shared__ float sentry[TL ? 128 : 1];
    bool sure = true;                         // a face was accepted in it: its box has passed
    bool inside = !TL;                        // the walk is in an instance (or the scene is flattened)
    WideSpill<SH, TL> spill;
    WideWalkT<kWideStack, SH, true> k;
    k.stack.spill = spill.pairs;
    k.stack.base = sstack + threadIdx.x;
    k.stack.stride = 128;
    k.cur = kWideDone;
    k.binary = false;
    // the direction of the ray that k.r was set up for
    auto dir = [&](float& x, float& y, float& z) {
        const float4 r1 = rays[2 * (size_t)idx + 1];
        x = r1.x; y = r1.y; z = r1.z;
        if constexpr (TL) {
            F3 o = f3(0.f, 0.f, 0.f), d = f3(r1.x, r1.y, r1.z);
            wide_to_object(inst + sinst[threadIdx.x], o, d);
            x = d.x; y = d.y; z = d.z;
        }
    };
    while (true) {
        // lanes whose ray has ended store its hit and take the next ray, PT_WIDE_REFILL at a time
        const uint32_t ended = __ballot_sync(0xFFFFFFFFu, k.cur == kWideDone);
        if (__popc(ended) >= (exhausted ? 32 : PT_WIDE_REFILL)) {
            if (k.cur == kWideDone && loaded) {
                bool ok = !k.done || k.any || k.binary;
                uint4 h;
                if (k.binary) {
                    const float4 r0 = rays[2 * (size_t)idx], r1 = rays[2 * (size_t)idx + 1];
                    auto& rest = spill.rest;
                    rest.ray = BinaryRay{r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, r0.w, k.any};
                    if constexpr (TL) {
                        const TwoLevelView view{nodes, tris, num_nodes, top, num_top, inst, false};
                        uint32_t hit_inst;
                        ok = wide_two_level_walk(&view, &rest.ray, &rest.hit, &hit_inst, rest.stack);
                    } else {
                        ok = wide_binary_walk(nodes, tris, num_nodes, &rest.ray, &rest.hit, rest.stack);
                    }
                    const BinaryHit b = rest.hit;
                    h = make_uint4(b.prim, __float_as_uint(b.t), __float_as_uint(b.u), __float_as_uint(b.v));
                } else {
                    h = make_uint4(k.prim, __float_as_uint(k.min_t), __float_as_uint(k.u), __float_as_uint(k.v));
                }
                if (!ok) {
                    h.x = 0xFFFFFFFEu;
                    atomicExch(err, 1);
                }
                st_stream(hits + idx, h);
                loaded = false;
            }
            if (!exhausted && pool_next >= pool_end) {
                unsigned long long base = (unsigned long long)gridDim.x * 4 * chunk;
                const uint32_t take = TL ? chunk : wide_take(n - pool_end, gridDim.x * 4, chunk);
                if (base < n) {
                    if (lane == 0) base += atomicAdd(counter, (unsigned long long)take);
                    base = __shfl_sync(0xFFFFFFFFu, base, 0);
                }
                if (base >= n) {
                    exhausted = true;
                } else {
                    pool_next = (uint32_t)base;
                    pool_end = n - pool_next < take ? n : pool_next + take;
                }
            }
            const uint32_t avail = pool_end - pool_next;
            const uint32_t rank = __popc(ended & ((1u << lane) - 1u));
            if (k.cur == kWideDone && rank < avail) {
                idx = pool_next + rank;
                const float4 r0 = ld_stream(rays + 2 * (size_t)idx);
                const float4 r1 = ld_stream(rays + 2 * (size_t)idx + 1);
                wide_begin(k, r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, r0.w, (__float_as_uint(r1.w) & 1u) != 0, size);
                inside = !TL;
                loaded = true;
            }
            const uint32_t took = min((uint32_t)__popc(ended), avail);
            pool_next += took;
            if (took == 0 && exhausted && ended == 0xFFFFFFFFu) break;
            continue;
        }
        const bool crosses = TL && k.cur != kWideDone && (k.cur == kWideExit || ((k.cur & kWideLeaf) && !inside));
        auto at_face = [&]() { return (k.cur & kWideLeaf) && k.cur < kWideExit && (!TL || inside); };
        const uint32_t leaves = __ballot_sync(0xFFFFFFFFu, at_face());
        int live = __popc(~ended);
        if constexpr (TL) {
            const uint32_t crossing = __ballot_sync(0xFFFFFFFFu, crosses);
            live -= __popc(crossing);  // the lanes that walk
            if (__popc(crossing) >= PT_WIDE_ENTERS || (crossing && live == 0)) {
                if (crosses) {
                    const float4 r0 = rays[2 * (size_t)idx], r1 = rays[2 * (size_t)idx + 1];
                    F3 o = f3(r0.x, r0.y, r0.z), d = f3(r1.x, r1.y, r1.z);
                    const bool enters = wide_cross(k, inside);
                    if (k.cur != kWideDone) {  // into an instance, or back to a top-level record
                        const uint32_t ii = k.cur & kWideIndex;
                        uint4 wi = make_uint4(0u, __float_as_uint(size), 0u, 0u);
                        if (enters) {
                            sinst[threadIdx.x] = ii;
                            sentry[threadIdx.x] = k.min_t;
                            sure = false;
                            wide_to_object(inst + ii, o, d);
                            wi = wide_instance(wide, ii);
                        }
                        ray_setup(k.r, o.x, o.y, o.z, d.x, d.y, d.z);
                        const bool fits = wide_cut(k.r, k.cut, __uint_as_float(wi.y));
                        if (enters) {
                            inside = wide_enter(k, wi.x, fits);
                            if (!inside) {
                                k.any = k.any && k.binary;  // a guard failure is no any-hit result
                                k.cur = kWideDone;
                            }
                        }
                    }
                }
                continue;
            }
        }
        const bool last = !TL && exhausted;  // the warp's last rays
        if (__popc(leaves) >= min(live, last ? PT_WIDE_LAST_BATCH : PT_WIDE_BATCH)) {
#pragma unroll 1
            for (int step = 0; step < (last ? PT_WIDE_LAST_LEAVES : 1) && at_face(); ++step) {
                if constexpr (TL) {
                    const DeviceInstance* in = inst + sinst[threadIdx.x];
                    if (wide_faces(k, tris, [&]() { return nodes + 2 * (size_t)ldg(&in->node_base); }, dir,
                                   [&]() { return ldg(&in->face_base); })) {
                        k.prim += ldg(&in->prim_base);
                        if (!sure) {
                            const float4 r0 = rays[2 * (size_t)idx], r1 = rays[2 * (size_t)idx + 1];
                            if (!wide_instance_passes(wide, top, sinst[threadIdx.x], r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, sentry[threadIdx.x]))
                                k.binary = k.done = true;
                            sure = true;
                        }
                    }
                } else {
                    wide_faces(k, tris, [&]() { return nodes; }, dir, []() { return 0u; });
                }
                if (k.done) k.cur = kWideDone; else wide_pop(k);
            }
        } else {
#pragma unroll 1
            for (int step = 0; step < PT_WIDE_STEPS && !(k.cur & kWideLeaf); ++step) {
                if (wide_visit(k, wide)) wide_pop(k);
                else { k.done = true; k.any = k.binary = false; k.cur = kWideDone; }  // guard failure
            }
        }
    }
}

// Ray queries on a two-level scene: one thread per ray, traverse_two_level.
template <bool COUNT>
__global__ void __launch_bounds__(128) trace_two_level_kernel(const TwoLevelView v, const float4* __restrict__ rays,
                                                              uint4* __restrict__ hits, uint64_t n, uint32_t* node_tests,
                                                              uint32_t* tri_tests, int* err) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 r0 = ld_stream(rays + 2 * i);
    const float4 r1 = ld_stream(rays + 2 * i + 1);
    const bool any = (__float_as_uint(r1.w) & 1u) != 0;
    const TwoLevelHit th = traverse_two_level<COUNT>(v, r0.x, r0.y, r0.z, r1.x, r1.y, r1.z, r0.w, any);
    uint4 h;
    h.x = th.r.prim;
    h.y = __float_as_uint(th.r.t);
    h.z = __float_as_uint(th.r.u);
    h.w = __float_as_uint(th.r.v);
    if (th.r.overflow) {
        h.x = 0xFFFFFFFEu;
        atomicExch(err, 1);
    }
    st_stream(hits + i, h);
    if (COUNT) {
        if (node_tests) node_tests[i] = th.r.nodes;
        if (tri_tests) tri_tests[i] = th.r.tris;
    }
}

cudaError_t launch_trace(const TraceArgs& a, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    if (a.wide && a.counter && !a.node_tests && !a.tri_tests && a.n < 0xFFFF0000ull) {  // 32-bit ray numbers
        const int sh = a.shared_stack;
        auto pick = [sh](auto k0, auto k8, auto k16, auto k24, auto k32) {
            return sh >= 32 ? k32 : sh >= 24 ? k24 : sh >= 16 ? k16 : sh >= 8 ? k8 : k0;
        };
        auto kern = a.instances ? pick(trace_wide_kernel<0, true>, trace_wide_kernel<8, true>, trace_wide_kernel<16, true>,
                                       trace_wide_kernel<24, true>, trace_wide_kernel<32, true>)
                                : pick(trace_wide_kernel<0, false>, trace_wide_kernel<8, false>, trace_wide_kernel<16, false>,
                                       trace_wide_kernel<24, false>, trace_wide_kernel<32, false>);
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 128, 0);
        if (e != cudaSuccess) return e;
        const uint64_t warps = (uint64_t)sms * (per_sm < 1 ? 1 : per_sm) * 4;
        uint64_t ch = a.chunk ? a.chunk : 64u;
        ch = std::max<uint64_t>(1, std::min(ch, (a.n + warps - 1) / warps));
        const uint64_t grid = std::min<uint64_t>(warps / 4, ((a.n + ch - 1) / ch + 3) / 4);
        if (grid * 4 * ch < a.n) e = cudaMemsetAsync(a.counter, 0, sizeof(unsigned long long), s);
        if (e != cudaSuccess) return e;
        kern<<<(unsigned)grid, 128, 0, s>>>((const WideNode*)a.wide, (const uint4*)a.nodes, (const float4*)a.tris, a.num_nodes,
                                            (const uint4*)a.top_nodes, a.top_num_nodes, (const DeviceInstance*)a.instances, (const float4*)a.rays, (uint4*)a.hits, (uint32_t)a.n, a.err,
                                            (unsigned long long*)a.counter, (uint32_t)ch, a.wide_size);
        return cudaGetLastError();
    }
    if (a.instances) {
        const TwoLevelView v{(const uint4*)a.nodes, (const float4*)a.tris, a.num_nodes, (const uint4*)a.top_nodes,
                             a.top_num_nodes, (const DeviceInstance*)a.instances, a.exact_tree};
        const uint64_t grid = (a.n + 127) / 128;
        if (grid > 0x7FFFFFFFull) return cudaErrorInvalidValue;
        if (a.node_tests || a.tri_tests)
            trace_two_level_kernel<true><<<(unsigned)grid, 128, 0, s>>>(v, (const float4*)a.rays, (uint4*)a.hits, a.n,
                                                                        a.node_tests, a.tri_tests, a.err);
        else
            trace_two_level_kernel<false><<<(unsigned)grid, 128, 0, s>>>(v, (const float4*)a.rays, (uint4*)a.hits, a.n,
                                                                         nullptr, nullptr, a.err);
        return cudaGetLastError();
    }
    if (a.counter) {
        int dev = 0, sms = 0, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        const bool counted = a.node_tests || a.tri_tests;
        const int sh = a.shared_stack;
        auto pick = [sh](auto k0, auto k8, auto k16, auto k24, auto k32) {
            return sh >= 32 ? k32 : sh >= 24 ? k24 : sh >= 16 ? k16 : sh >= 8 ? k8 : k0;
        };
        auto kern_f = pick(trace_persistent_kernel<false, 0>, trace_persistent_kernel<false, 8>, trace_persistent_kernel<false, 16>,
                           trace_persistent_kernel<false, 24>, trace_persistent_kernel<false, 32>);
        auto kern_t = pick(trace_persistent_kernel<true, 0>, trace_persistent_kernel<true, 8>, trace_persistent_kernel<true, 16>,
                           trace_persistent_kernel<true, 24>, trace_persistent_kernel<true, 32>);
        cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, counted ? kern_t : kern_f, 128, 0);
        if (e != cudaSuccess) return e;
        if (per_sm < 1) per_sm = 1;
        uint64_t grid = (uint64_t)sms * per_sm;
        const uint32_t ch = a.chunk ? a.chunk : 64u;
        const uint64_t need = ((a.n + ch - 1) / ch * 32 + 127) / 128;
        if (grid > need) grid = need;
        e = cudaMemsetAsync(a.counter, 0, sizeof(unsigned long long), s);
        if (e != cudaSuccess) return e;
        if (counted)
            kern_t<<<(unsigned)grid, 128, 0, s>>>((const uint4*)a.nodes, (const float4*)a.tris, a.num_nodes,
                                                  (const float4*)a.rays, (uint4*)a.hits, a.n, a.node_tests, a.tri_tests,
                                                  a.err, (unsigned long long*)a.counter, a.chunk ? a.chunk : 64u, a.exact_tree);
        else
            kern_f<<<(unsigned)grid, 128, 0, s>>>((const uint4*)a.nodes, (const float4*)a.tris, a.num_nodes,
                                                  (const float4*)a.rays, (uint4*)a.hits, a.n, nullptr, nullptr, a.err,
                                                  (unsigned long long*)a.counter, a.chunk ? a.chunk : 64u, a.exact_tree);
        return cudaGetLastError();
    }
    const uint32_t block = 128;
    const uint64_t grid = (a.n + block - 1) / block;
    if (grid > 0x7FFFFFFFull) return cudaErrorInvalidValue;
    if (a.node_tests || a.tri_tests)
        trace_kernel<true><<<(unsigned)grid, block, 0, s>>>(
            (const uint4*)a.nodes, (const float4*)a.tris, a.num_nodes, (const float4*)a.rays, (uint4*)a.hits, a.n,
            a.node_tests, a.tri_tests, a.err, a.exact_tree);
    else
        trace_kernel<false><<<(unsigned)grid, block, 0, s>>>(
            (const uint4*)a.nodes, (const float4*)a.tris, a.num_nodes, (const float4*)a.rays, (uint4*)a.hits, a.n,
            nullptr, nullptr, a.err, a.exact_tree);
    return cudaGetLastError();
}

// ---- self-tests of the exact helpers ------------------------------------------------------------

__global__ void selftest_f64_kernel(const float4* in, float* out, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 v = in[i];
    out[i] = f64_diff_emulated(v.x, v.y, v.z, v.w);
}

__global__ void selftest_sincos_kernel(const float* u, float2* out, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float s, c;
    sincos_2pi(u[i], s, c);
    out[i] = make_float2(s, c);
}

__global__ void selftest_philox_kernel(const uint4* in, uint4* out, uint32_t n, uint32_t k0, uint32_t k1) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint4 v = in[i];
    uint32_t c[4] = {v.x, v.y, v.z, v.w};
    philox4x32(c, k0, k1);
    out[i] = make_uint4(c[0], c[1], c[2], c[3]);
}

__global__ void selftest_box_kernel(const float* in, uint32_t* out, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float* c = in + 16 * (size_t)i;
    RayState r;
    ray_setup(r, c[6], c[7], c[8], c[9], c[10], c[11]);
    // as a traversal runs it: the scene-level NaN flag set when this box holds a NaN, then the
    // ray's own box mode (the min/max test for finite rays)
    bool nan_box = false;
    for (int k = 0; k < 6; ++k) nan_box = nan_box || c[k] != c[k];
    out[i] = box_test(r, box_mode_for(r, c[12], nan_box), c[0], c[1], c[2], c[3], c[4], c[5], c[12]) ? 1u : 0u;
}

cudaError_t launch_selftest_box(const float* in16, uint32_t* hit, uint32_t n, cudaStream_t s) {
    if (!n) return cudaSuccess;
    selftest_box_kernel<<<(n + 127) / 128, 128, 0, s>>>(in16, hit, n);
    return cudaGetLastError();
}

cudaError_t launch_selftest_f64(const float* in4, float* out, uint32_t n, cudaStream_t s) {
    if (!n) return cudaSuccess;
    selftest_f64_kernel<<<(n + 127) / 128, 128, 0, s>>>((const float4*)in4, out, n);
    return cudaGetLastError();
}
cudaError_t launch_selftest_sincos(const float* u, float* out2, uint32_t n, cudaStream_t s) {
    if (!n) return cudaSuccess;
    selftest_sincos_kernel<<<(n + 127) / 128, 128, 0, s>>>(u, (float2*)out2, n);
    return cudaGetLastError();
}
cudaError_t launch_selftest_philox(const uint32_t* in4, uint32_t* out4, uint32_t n, uint64_t seed, cudaStream_t s) {
    if (!n) return cudaSuccess;
    selftest_philox_kernel<<<(n + 127) / 128, 128, 0, s>>>((const uint4*)in4, (uint4*)out4, n, (uint32_t)seed,
                                                          (uint32_t)(seed >> 32));
    return cudaGetLastError();
}

}  // namespace pt
