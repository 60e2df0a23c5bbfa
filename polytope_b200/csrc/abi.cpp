// abi.cpp -- the C ABI (include/polytope_b200.h): scene upload, ray queries, error reporting.

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <thread>
#include <vector>

#include <cuda_runtime.h>

#include "exact_math.h"
#include "host_workers.h"
#include "launch.h"
#include "pt_internal.h"

namespace pt {

namespace {
thread_local std::string g_last_error;

struct DeviceGuard {  // makes `dev` current for the scope and restores the caller's device
    int prev = -1;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) prev = -1;
        if (prev != dev) cudaSetDevice(dev);
    }
    ~DeviceGuard() {
        int cur = -1;
        if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
    }
};

int cuda_fail(cudaError_t e, const char* what) {
    return fail(PT_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
}

#define PT_CUDA(call)                                     \
    do {                                                  \
        cudaError_t e_ = (call);                          \
        if (e_ != cudaSuccess) return cuda_fail(e_, #call); \
    } while (0)

size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }

float largest_coordinate(const pt_bvh_node& root) {
    float m = 0.f;
    for (int k = 0; k < 3; ++k) m = std::max(m, std::max(std::fabs(root.bb_min[k]), std::fabs(root.bb_max[k])));
    return m;
}

// The four-wide records of the scene's trees (wide.cuh), made on the device from the uploaded nodes.  Trees of
// extreme size (wide_sizes_fit) get none and keep the binary walk, as do those with a box outside its
// parent's (only a caller's own tree can have one) and those whose records do not fit in memory.  `base`
// holds wide_bytes(h): the instance table, the records, then the numbering and a flag.
bool wide_sizes_fit(const HostScene& h) {
    auto fits = [](const pt_bvh_node& root) {
        const float size = largest_coordinate(root);
        return size >= kWideSizeMin && size <= kWideSizeMax;
    };
    if (!h.two_level) return fits(h.nodes[0]);
    bool all = fits(h.tlas[0]);
    for (const HostScene::Geometry& g : h.geometries) all = all && fits(h.nodes[g.node_base]);
    return all;
}
size_t wide_table_bytes(const HostScene& h) { return up256(sizeof(WideInstance) * h.instances.size()); }
size_t wide_bytes(const HostScene& h) {
    return wide_table_bytes(h) + 64 * (size_t)h.num_wide + 4 * (h.wide_of.size() + h.top_wide_of.size() + 1);
}

int make_wide(pt_scene* s, const HostScene& h, char* base) {
    struct Tree { const void* nodes; const uint32_t* wide_of; uint32_t num_nodes, face_base; float size; bool faces; };
    std::vector<Tree> trees;
    std::vector<WideInstance> table(h.instances.size());
    const size_t n = h.wide_of.size(), nt = h.top_wide_of.size();
    char* records = base + wide_table_bytes(h);
    uint32_t* number = (uint32_t*)(records + 64 * (size_t)h.num_wide);
    if (h.two_level) {
        trees.push_back({s->dev.tlas_nodes, number + n, (uint32_t)nt, 0, largest_coordinate(h.tlas[0]), false});
        for (const HostScene::Geometry& g : h.geometries)
            trees.push_back({(const char*)s->dev.nodes + sizeof(pt_bvh_node) * (size_t)g.node_base, number + g.node_base, g.num_nodes,
                             g.face_base, largest_coordinate(h.nodes[g.node_base]), true});
        for (size_t i = 0; i < h.tlas.size(); ++i)
            if (h.tlas[i].num_faces == 1) table[table.size() - 1 - h.tlas[i].offset].node = (uint32_t)i;
        for (size_t i = 0; i < h.instances.size(); ++i) {
            WideInstance& w = table[table.size() - 1 - i];  // instance 0 lies just before record 0
            w.root = h.wide_of[h.instances[i].node_base];
            w.size = largest_coordinate(h.nodes[h.instances[i].node_base]);
        }
    } else {
        trees.push_back({s->dev.nodes, number, (uint32_t)n, 0, largest_coordinate(h.nodes[0]), true});
    }
    uint32_t outside = 0;
    cudaError_t e = cudaMemcpy(number, h.wide_of.data(), 4 * n, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && nt) e = cudaMemcpy(number + n, h.top_wide_of.data(), 4 * nt, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && !table.empty())
        e = cudaMemcpy(records - sizeof(WideInstance) * table.size(), table.data(), sizeof(WideInstance) * table.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(number + n + nt, 0, 4);
    for (const Tree& t : trees)
        if (e == cudaSuccess)
            e = launch_wide_make(t.nodes, t.wide_of, t.num_nodes, t.size, t.face_base, records, t.faces ? s->dev.tris : nullptr,
                                 number + n + nt, nullptr);
    if (e == cudaSuccess) e = cudaMemcpy(&outside, number + n + nt, 4, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return cuda_fail(e, "four-wide records");
    if (outside) return PT_OK;
    s->dev.wide = records;
    s->wide_size = trees[0].size;
    return PT_OK;
}

void free_scene(pt_scene* s) {
    if (!s) return;
    DeviceGuard g(s->device);
    void* bufs[] = {s->memory, s->dev_in, s->dev_out, s->trace_err};
    for (void* b : bufs)
        if (b) cudaFree(b);
    if (s->pin_in) cudaFreeHost(s->pin_in);
    if (s->pin_out) cudaFreeHost(s->pin_out);
    for (void*& st : s->streams)
        if (st) cudaStreamDestroy((cudaStream_t)st);
    for (void*& ev : s->events)
        if (ev) cudaEventDestroy((cudaEvent_t)ev);
    delete s;
}

bool is_pinned(const void* p) {
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return attr.type == cudaMemoryTypeHost;
}

// Rays per chunk of the host-pointer pipeline.  Measured on the 16.7 M-ray microbench end to end:
// 1 M-ray chunks 1436 Mrays/s, 512 K 1413, 2 M 1339 (longer fill and drain), 256 K 1030, over binary nodes; over
// four-wide records 1590, and 768 K and 512 K within 1 % of that, 256 K 1430.
constexpr size_t kChunkRays = size_t(1) << 20;
constexpr int kSlots = 4;  // chunks in flight: one being copied in, one or two in kernels, one copied out
constexpr size_t kStagingIn = kSlots * kChunkRays * sizeof(pt_ray), kStagingOut = kSlots * kChunkRays * sizeof(pt_hit);

int ensure_staging(pt_scene* s) {
    if (s->staging_rays) return PT_OK;
    for (void*& st : s->streams) PT_CUDA(cudaStreamCreateWithFlags((cudaStream_t*)&st, cudaStreamNonBlocking));
    for (int i = 0; i < 3 * kSlots + 1; ++i)
        PT_CUDA(cudaEventCreateWithFlags((cudaEvent_t*)&s->events[i], cudaEventDisableTiming));
    if (cudaMalloc(&s->dev_in, kStagingIn) != cudaSuccess || cudaMalloc(&s->dev_out, kStagingOut) != cudaSuccess ||
        cudaMalloc(&s->trace_err, sizeof(int)) != cudaSuccess)
        return fail(PT_ENOMEM, "cudaMalloc staging buffers");
    if (cudaMallocHost(&s->pin_in, kStagingIn) != cudaSuccess || cudaMallocHost(&s->pin_out, kStagingOut) != cudaSuccess)
        return fail(PT_ENOMEM, "cudaMallocHost staging buffers");
    s->staging_rays = kChunkRays;
    return PT_OK;
}

}  // namespace

void set_error(const std::string& msg) { g_last_error = msg; }
int fail(int code, const std::string& msg) {
    g_last_error = msg;
    return code;
}

// Host arrays that are not pinned: each of up to kWorkers threads takes chunks through its own part of the
// staging buffers and its own stream -- rays into pinned memory, to the device, kernel, hits back, out of
// pinned memory.  Copying into and out of the staging buffers is what such a call spends its time on
// (one thread: 5.9 ms for 1 M rays on a host of 16 threads, of which the kernel takes 0.3), so it is what
// runs in parallel, and one worker's copies overlap another's transfers and kernel: 1.9 ms with eight;
// 100 k rays 0.47 -> 0.35 to 0.43, 300 k 1.18 -> 0.63.
static int trace_pageable(pt_scene* s, const TraceArgs& common, const pt_ray* rays, uint64_t n, pt_hit* hits, bool pin_rays,
                          bool pin_hits, cudaEvent_t dep, int workers) {
    constexpr uint64_t slot_rays = kSlots * kChunkRays / kWorkers;
    // at least two chunks a worker, so that its second copy-in follows the first's results closely
    const uint64_t chunk = std::min(slot_rays, (n + 2 * workers - 1) / (2 * workers)), chunks = (n + chunk - 1) / chunk;
    std::atomic<uint64_t> next{0};
    std::atomic<bool> failed{false};
    std::mutex mu;
    int rc = PT_OK;
    std::string message;
    PT_CUDA(cudaStreamSynchronize((cudaStream_t)s->streams[0]));  // the flag is clear before any kernel
    auto work = [&](int w) {
        auto run = [&]() -> int {
            PT_CUDA(cudaSetDevice(s->device));
            cudaStream_t st = (cudaStream_t)s->streams[w];
            PT_CUDA(cudaStreamWaitEvent(st, dep, 0));
            pt_ray *pin = (pt_ray*)s->pin_in + w * slot_rays, *din = (pt_ray*)s->dev_in + w * slot_rays;
            pt_hit *pout = (pt_hit*)s->pin_out + w * slot_rays, *dout = (pt_hit*)s->dev_out + w * slot_rays;
            TraceArgs a = common;
            for (uint64_t c; !failed.load() && (c = next.fetch_add(1)) < chunks;) {
                const uint64_t off = c * chunk, cnt = std::min(chunk, n - off);
                const pt_ray* src = rays + off;
                if (!pin_rays) {
                    std::memcpy(pin, src, cnt * sizeof(pt_ray));
                    src = pin;
                }
                PT_CUDA(cudaMemcpyAsync(din, src, cnt * sizeof(pt_ray), cudaMemcpyHostToDevice, st));
                a.rays = din;
                a.hits = dout;
                a.n = cnt;
                a.counter = (unsigned long long*)s->ray_counters + (s->counter_next.fetch_add(1) % PT_RAY_COUNTERS);
                const cudaError_t e = launch_trace(a, st);
                if (e != cudaSuccess) return cuda_fail(e, "trace kernel launch");
                PT_CUDA(cudaMemcpyAsync(pin_hits ? hits + off : pout, dout, cnt * sizeof(pt_hit), cudaMemcpyDeviceToHost, st));
                PT_CUDA(cudaStreamSynchronize(st));
                if (!pin_hits) std::memcpy(hits + off, pout, cnt * sizeof(pt_hit));
            }
            return PT_OK;
        };
        int r = PT_ENOMEM;
        try {
            r = run();
        } catch (const std::bad_alloc&) {  // a message found no memory
            g_last_error = "no host memory";
        }
        if (r != PT_OK) {
            std::unique_lock<std::mutex> lock(mu);
            if (!failed.exchange(true)) {
                rc = r;
                message.swap(g_last_error);
            }
            lock.unlock();
            cudaStreamSynchronize((cudaStream_t)s->streams[w]);  // nothing of this call still uses the arrays
        }
    };
    run_workers(workers, work);
    return rc == PT_OK ? PT_OK : fail(rc, message);
}

int scene_trace(pt_scene* s, const pt_ray* rays, uint64_t n, pt_hit* hits, uint32_t* node_tests, uint32_t* tri_tests,
                uint32_t mem_flags, void* stream) {
    if (!s) return fail(PT_EINVAL, "scene is NULL");
    if (n == 0) return PT_OK;
    if (!rays || !hits) return fail(PT_EINVAL, "rays or hits is NULL");
    if ((int)s->max_depth + 2 > PT_TRAVERSAL_STACK)
        return fail(PT_ESTACK, "tree depth " + std::to_string(s->max_depth) + " exceeds the traversal stack");
    DeviceGuard g(s->device);
    TraceArgs a{};
    a.nodes = s->dev.nodes;
    a.tris = s->dev.tris;
    a.num_nodes = s->num_nodes;
    a.err = (int*)s->err_flag;
    a.shared_stack = (int)s->trace_tuning.shared_stack;
    a.chunk = s->trace_tuning.queue_chunk;
    a.instances = s->dev.instances;
    a.top_nodes = s->dev.tlas_nodes;
    a.top_num_nodes = s->dev.tlas_num_nodes;
    a.exact_tree = s->nan_boxes;
    a.wide = s->dev.wide;
    a.wide_size = s->wide_size;
    auto next_counter = [s]() {
        return (void*)((unsigned long long*)s->ray_counters + (s->counter_next.fetch_add(1) % PT_RAY_COUNTERS));
    };
    if (mem_flags & PT_MEM_DEVICE) {
        a.counter = next_counter();
        a.rays = rays;
        a.hits = hits;
        a.n = n;
        a.node_tests = node_tests;
        a.tri_tests = tri_tests;
        cudaError_t e = launch_trace(a, (cudaStream_t)stream);
        if (e != cudaSuccess) return cuda_fail(e, "trace kernel launch");
        return PT_OK;
    }
    // Host pointers: 1 M-ray chunks through kSlots staging slots and three engines at once -- a
    // stream of host->device copies, two kernel streams (so one chunk's kernel tail overlaps the
    // next), and a stream of device->host copies -- ordered per slot by events.  Pageable arrays
    // go through the pinned staging of their slot.
    std::lock_guard<std::mutex> lock(s->staging_mu);
    int rc = ensure_staging(s);
    if (rc) return rc;
    cudaStream_t h2d = (cudaStream_t)s->streams[0], d2h = (cudaStream_t)s->streams[3];
    cudaStream_t kst[2] = {(cudaStream_t)s->streams[1], (cudaStream_t)s->streams[2]};
    cudaEvent_t* ev = (cudaEvent_t*)s->events;
    cudaEvent_t *ev_in = ev, *ev_k = ev + kSlots, *ev_out = ev + 2 * kSlots, dep = ev[3 * kSlots];
    PT_CUDA(cudaEventRecord(dep, (cudaStream_t)stream));
    for (int i = 0; i < 4; ++i) PT_CUDA(cudaStreamWaitEvent((cudaStream_t)s->streams[i], dep, 0));
    a.err = (int*)s->trace_err;  // this call's own flag: the asynchronous calls raise err_flag
    PT_CUDA(cudaMemsetAsync(s->trace_err, 0, sizeof(int), h2d));  // before every copy-in, so before every kernel
    const bool pin_rays = is_pinned(rays), pin_hits = is_pinned(hits);
    const bool counted = node_tests || tri_tests;
    const int workers = counted || (pin_rays && pin_hits) ? 1 : pageable_workers(n, std::thread::hardware_concurrency(), one_processor());
    if (workers > 1) {
        rc = trace_pageable(s, a, rays, n, hits, pin_rays, pin_hits, dep, workers);
        if (rc) return rc;
        int err = 0;
        PT_CUDA(cudaMemcpy(&err, s->trace_err, sizeof(int), cudaMemcpyDeviceToHost));
        if (err) return fail(PT_ESTACK, "a ray exceeded the traversal stack (malformed or too deep tree)");
        return PT_OK;
    }
    uint32_t* dcounts = nullptr;
    if (counted && cudaMalloc(&dcounts, 2 * sizeof(uint32_t) * n) != cudaSuccess)
        return fail(PT_ENOMEM, "cudaMalloc count buffers");
    struct Free { uint32_t* p; ~Free() { if (p) cudaFree(p); } } free_counts{dcounts};
    // Chunks: full slots in the middle, and a quarter then a half slot at both ends on long calls.
    // The kernels wait for the first chunk's copy-in, and the last chunk's kernel and copy-out are
    // all that runs after the final copy-in: short end chunks shorten both waits.
    std::vector<std::pair<uint64_t, uint64_t>> chunks;  // (first ray, count)
    if (n >= 4 * (uint64_t)kChunkRays) {
        const uint64_t q = kChunkRays / 4, h = kChunkRays / 2;
        chunks.push_back({0, q});
        chunks.push_back({q, h});
        uint64_t off = q + h;
        while (n - off > h + q) {
            const uint64_t cnt = std::min<uint64_t>(kChunkRays, n - off - (h + q));
            chunks.push_back({off, cnt});
            off += cnt;
        }
        chunks.push_back({off, h});
        chunks.push_back({off + h, q});
    } else {
        for (uint64_t off = 0; off < n; off += kChunkRays) chunks.push_back({off, std::min<uint64_t>(kChunkRays, n - off)});
    }
    const uint64_t nchunks = chunks.size();
    uint64_t in_slot[kSlots];
    for (int k = 0; k < kSlots; ++k) in_slot[k] = ~0ull;  // chunk whose data occupies each slot
    auto drain = [&](int slot) -> int {  // pageable hits: move the slot's results out
        if (in_slot[slot] == ~0ull) return PT_OK;
        PT_CUDA(cudaEventSynchronize(ev_out[slot]));
        if (!pin_hits) {
            const uint64_t off = chunks[in_slot[slot]].first, cnt = chunks[in_slot[slot]].second;
            std::memcpy(hits + off, (pt_hit*)s->pin_out + slot * kChunkRays, cnt * sizeof(pt_hit));
        }
        in_slot[slot] = ~0ull;
        return PT_OK;
    };
    // Chunk c's hits out, once its kernel ran and chunk c + 1's rays are in (next): a copy in that starts beside a
    // copy out under way starts 45 us late and runs slower, and copies out that begin with a copy in end
    // before the next.  16.7 M rays on 1.3 M faces 11.30 -> 10.56 ms.
    auto copy_out = [&](uint64_t c, cudaEvent_t next) -> int {
        const int slot = (int)(c % kSlots);
        const uint64_t off = chunks[c].first;
        PT_CUDA(cudaStreamWaitEvent(d2h, ev_k[slot], 0));
        if (next) PT_CUDA(cudaStreamWaitEvent(d2h, next, 0));
        void* dst = pin_hits ? (void*)(hits + off) : (void*)((pt_hit*)s->pin_out + slot * kChunkRays);
        PT_CUDA(cudaMemcpyAsync(dst, (pt_hit*)s->dev_out + slot * kChunkRays, chunks[c].second * sizeof(pt_hit), cudaMemcpyDeviceToHost, d2h));
        PT_CUDA(cudaEventRecord(ev_out[slot], d2h));
        return PT_OK;
    };
    for (uint64_t c = 0; c < nchunks; ++c) {
        const int slot = (int)(c % kSlots);
        const bool reused = in_slot[slot] != ~0ull;
        if (reused && !pin_hits) {
            rc = drain(slot);
            if (rc) return rc;
        }
        const uint64_t off = chunks[c].first, cnt = chunks[c].second;
        pt_ray* din = (pt_ray*)s->dev_in + slot * kChunkRays;
        pt_hit* dout = (pt_hit*)s->dev_out + slot * kChunkRays;
        const void* src = rays + off;
        if (!pin_rays) {
            if (reused) PT_CUDA(cudaEventSynchronize(ev_in[slot]));  // the slot's previous copy-in has read it
            std::memcpy((pt_ray*)s->pin_in + slot * kChunkRays, rays + off, cnt * sizeof(pt_ray));
            src = (pt_ray*)s->pin_in + slot * kChunkRays;
        }
        if (reused) PT_CUDA(cudaStreamWaitEvent(h2d, ev_k[slot], 0));  // din is free once its kernel ran
        PT_CUDA(cudaMemcpyAsync(din, src, cnt * sizeof(pt_ray), cudaMemcpyHostToDevice, h2d));
        PT_CUDA(cudaEventRecord(ev_in[slot], h2d));
        cudaStream_t k = kst[c & 1];
        PT_CUDA(cudaStreamWaitEvent(k, ev_in[slot], 0));
        if (reused) PT_CUDA(cudaStreamWaitEvent(k, ev_out[slot], 0));  // dout is free once copied out
        a.rays = din;
        a.hits = dout;
        a.n = cnt;
        a.counter = next_counter();
        a.node_tests = counted ? dcounts + off : nullptr;
        a.tri_tests = counted ? dcounts + n + off : nullptr;
        cudaError_t e = launch_trace(a, k);
        if (e != cudaSuccess) return cuda_fail(e, "trace kernel launch");
        PT_CUDA(cudaEventRecord(ev_k[slot], k));
        in_slot[slot] = c;
        if (c > 0 && (rc = copy_out(c - 1, ev_in[slot]))) return rc;
    }
    rc = copy_out(nchunks - 1, nullptr);
    if (rc) return rc;
    for (uint64_t c = nchunks > kSlots ? nchunks - kSlots : 0; c < nchunks; ++c) {
        rc = drain((int)(c % kSlots));
        if (rc) return rc;
    }
    PT_CUDA(cudaStreamSynchronize(d2h));
    if (counted) {
        std::vector<uint32_t> tmp(2 * n);
        PT_CUDA(cudaMemcpy(tmp.data(), dcounts, 2 * n * sizeof(uint32_t), cudaMemcpyDeviceToHost));
        if (node_tests) std::memcpy(node_tests, tmp.data(), n * sizeof(uint32_t));
        if (tri_tests) std::memcpy(tri_tests, tmp.data() + n, n * sizeof(uint32_t));
    }
    int err = 0;
    PT_CUDA(cudaMemcpy(&err, s->trace_err, sizeof(int), cudaMemcpyDeviceToHost));
    if (err) return fail(PT_ESTACK, "a ray exceeded the traversal stack (malformed or too deep tree)");
    return PT_OK;
}


// Host-side layout of a scene (everything pt_scene_create uploads).
int prepare_scene_host(const pt_scene_desc* desc, HostScene& h) {
    if (!desc->meshes || desc->num_meshes == 0) return fail(PT_EINVAL, "scene has no meshes");
    for (uint32_t m = 0; m < desc->num_meshes; ++m) {
        const pt_mesh_desc& d = desc->meshes[m];
        if (d.material != PT_MAT_LAMBERT && d.material != PT_MAT_MIRROR)
            return fail(PT_EINVAL, "mesh " + std::to_string(m) + ": unknown material");
    }
    WorldMeshes w;
    int rc = bake_world(desc->meshes, desc->num_meshes, w);
    if (rc) return rc;
    BuiltTree t;
    if (desc->nodes) {
        if (!desc->leaf_pairs) return fail(PT_EINVAL, "nodes given without leaf_pairs");
        t.nodes.assign(desc->nodes, desc->nodes + desc->num_nodes);
        t.leaf_pairs.assign(desc->leaf_pairs, desc->leaf_pairs + 2 * (size_t)w.num_prims);
        for (size_t i = 0; i < w.num_prims; ++i) {
            const uint32_t m = t.leaf_pairs[2 * i], f = t.leaf_pairs[2 * i + 1];
            if (m >= desc->num_meshes || f >= desc->meshes[m].num_faces)
                return fail(PT_EINVAL, "leaf pair " + std::to_string(i) + " out of range");
        }
    } else {
        rc = build_bvh(desc->meshes, desc->num_meshes, w, 0, t);
        if (rc) return rc;
    }
    rc = validate_tree(t.nodes.data(), (uint32_t)t.nodes.size(), w.num_prims, &h.max_depth, &h.wide_of, &h.num_wide);
    if (rc) return rc;
    h.num_prims = w.num_prims;
    h.prim_base = w.prim_base;
    h.nodes.swap(t.nodes);
    // faces in leaf order, 48 B each: {v0.xyz v1.x}{v1.yz v2.xy}{v2.z prim mesh, leaf}: the last word is 0 until the
    // records are made, then the face's leaf node (wide_mark_leaf)
    h.tris.assign(12 * (size_t)w.num_prims, 0.f);
    for (size_t i = 0; i < w.num_prims; ++i) {
        const uint32_t m = t.leaf_pairs[2 * i], f = t.leaf_pairs[2 * i + 1];
        const uint32_t p = w.prim_base[m] + f;
        float* o = &h.tris[12 * i];
        std::memcpy(o, &w.tri[9 * (size_t)p], 9 * sizeof(float));
        o[9] = bitsf(p);
        o[10] = bitsf(m);
    }
    prepare_shading_host(desc, w, h);
    return PT_OK;
}

void prepare_shading_host(const pt_scene_desc* desc, const WorldMeshes& w, HostScene& h) {
    h.meshes.resize(desc->num_meshes);
    bool any_normals = false;
    for (uint32_t m = 0; m < desc->num_meshes; ++m) {
        const pt_mesh_desc& d = desc->meshes[m];
        h.meshes[m].material = d.material;
        h.meshes[m].is_light = d.is_light ? 1 : 0;
        std::memcpy(h.meshes[m].albedo, d.albedo, sizeof(d.albedo));
        std::memcpy(h.meshes[m].emission, d.emission, sizeof(d.emission));
        h.meshes[m].has_normals = (d.nx && d.ny && d.nz) ? 1 : 0;
        if (h.meshes[m].has_normals) any_normals = true;
    }
    if (any_normals) {  // world vertex normals per prim (Transform::ApplyInPlace(Normal&), mesh.cpp:388-400)
        h.normals.assign(9 * (size_t)w.num_prims, 0.f);
        for (uint32_t m = 0; m < desc->num_meshes; ++m) {
            const pt_mesh_desc& d = desc->meshes[m];
            if (!(d.nx && d.ny && d.nz)) continue;
            for (uint32_t f = 0; f < d.num_faces; ++f) {
                const uint32_t vi[3] = {d.fv0[f], d.fv1[f], d.fv2[f]};
                float* o = &h.normals[9 * (size_t)(w.prim_base[m] + f)];
                for (int k = 0; k < 3; ++k) {
                    o[3 * k] = d.nx[vi[k]];
                    o[3 * k + 1] = d.ny[vi[k]];
                    o[3 * k + 2] = d.nz[vi[k]];
                    apply_normal(d.world_to_object, &o[3 * k]);
                }
            }
        }
    }
    // area lights (every face of an emitting mesh, mesh/face order): world triangle, then the
    // running sum of 0.5 * |(v1 - v0) x (v2 - v0)| as the CDF
    h.light_area = 0.f;
    for (uint32_t p = 0; p < w.num_prims; ++p) {
        const uint32_t m = w.prim_mesh[p];
        if (!desc->meshes[m].is_light) continue;
        const float* v = &w.tri[9 * (size_t)p];
        const float e0[3] = {v[3] - v[0], v[4] - v[1], v[5] - v[2]};
        const float e1[3] = {v[6] - v[0], v[7] - v[1], v[8] - v[2]};
        const float c[3] = {e0[1] * e1[2] - e0[2] * e1[1], e0[2] * e1[0] - e0[0] * e1[2], e0[0] * e1[1] - e0[1] * e1[0]};
        const float area = 0.5f * std::sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
        h.light_area = h.light_area + area;
        for (int k = 0; k < 9; ++k) h.light_tris.push_back(v[k]);
        h.light_tris.push_back(bitsf(p));  // 12 floats per record: v0 v1 v2, prim, mesh, pad
        h.light_tris.push_back(bitsf(m));
        h.light_tris.push_back(0.f);
        h.light_cdf.push_back(h.light_area);
    }
}

}  // namespace pt

using namespace pt;

extern "C" {

const char* pt_last_error(void) { return g_last_error.c_str(); }
const char* pt_version(void) { return "polytope_b200 0.1 (sm_100a)"; }

int pt_bvh_build(const pt_mesh_desc* meshes, uint32_t num_meshes, int threads, pt_bvh_node* nodes_out,
                 uint32_t* num_nodes_out, uint32_t* leaf_pairs_out) {
    if (!meshes || num_meshes == 0) return fail(PT_EINVAL, "no meshes");
    if (!num_nodes_out) return fail(PT_EINVAL, "num_nodes_out is NULL");
    WorldMeshes w;
    int rc = bake_world(meshes, num_meshes, w);
    if (rc) return rc;
    BuiltTree t;
    rc = build_bvh(meshes, num_meshes, w, threads, t);
    if (rc) return rc;
    if (!nodes_out) {
        *num_nodes_out = (uint32_t)t.nodes.size();
        return PT_OK;
    }
    if (*num_nodes_out < t.nodes.size()) return fail(PT_EINVAL, "nodes_out too small");
    std::memcpy(nodes_out, t.nodes.data(), t.nodes.size() * sizeof(pt_bvh_node));
    *num_nodes_out = (uint32_t)t.nodes.size();
    if (leaf_pairs_out) std::memcpy(leaf_pairs_out, t.leaf_pairs.data(), t.leaf_pairs.size() * sizeof(uint32_t));
    return PT_OK;
}

}  // extern "C"

namespace {
int device_count_ok() {
    int ndev = 0;
    cudaError_t ce = cudaGetDeviceCount(&ndev);
    if (ce != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return fail(PT_ECUDA, "no CUDA device available (there is no CPU fallback)");
    }
    return PT_OK;
}

// Uploads a prepared scene (either layout) into a new handle.
int create_from_host(const pt_scene_desc* desc, HostScene& h, pt_scene** out) {
    int rc = PT_OK;
    std::unique_ptr<pt_scene> s(new pt_scene());
    cudaGetDevice(&s->device);
    s->num_nodes = (uint32_t)h.nodes.size();
    s->num_prims = h.num_prims;
    s->num_meshes = desc->num_meshes;
    s->max_depth = h.max_depth;
    s->prim_base = h.prim_base;
    s->has_env = desc->has_env;
    std::memcpy(s->env, desc->env, sizeof(s->env));
    s->has_normals = !h.normals.empty();
    s->dev.num_lights = (uint32_t)h.light_cdf.size();
    s->dev.light_area = h.light_area;

    auto has_nan = [](const std::vector<pt_bvh_node>& nodes) {
        for (const pt_bvh_node& n : nodes)
            for (int k = 0; k < 3; ++k)
                if (n.bb_min[k] != n.bb_min[k] || n.bb_max[k] != n.bb_max[k]) return true;
        return false;
    };
    s->nan_boxes = has_nan(h.nodes) || has_nan(h.tlas);
    s->two_level = h.two_level;
    s->dev.num_instances = (uint32_t)h.instances.size();
    s->dev.tlas_num_nodes = (uint32_t)h.tlas.size();

    // One allocation for everything the handle holds (each cudaMalloc costs scene creation 0.1 to 0.4 ms, now
    // and then some milliseconds).
    struct Part { void** dst; const void* src; size_t bytes; };
    auto part = [](void** dst, const auto& v) { return Part{dst, v.data(), sizeof(v[0]) * v.size()}; };
    const Part parts[] = {part(&s->dev.nodes, h.nodes), part(&s->dev.tris, h.tris), part(&s->dev.meshes, h.meshes),
                          part(&s->dev.prim_normals, h.normals), part(&s->dev.light_tris, h.light_tris),
                          part(&s->dev.light_cdf, h.light_cdf), part(&s->dev.instances, h.instances),
                          part(&s->dev.tlas_nodes, h.tlas)};
    size_t total = 256 + up256(8 * PT_RAY_COUNTERS);  // the error flag, the ray counters
    for (const Part& p : parts) total += up256(p.bytes);
    size_t wide = h.wide_of.empty() || s->nan_boxes || !wide_sizes_fit(h) ? 0 : wide_bytes(h);
    DeviceGuard g(s->device);
    cudaError_t e = cudaMalloc(&s->memory, total + wide);
    if (e != cudaSuccess && wide) {
        cudaGetLastError();
        wide = 0;
        e = cudaMalloc(&s->memory, total);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        s->memory = nullptr;
        free_scene(s.release());
        return fail(PT_ENOMEM, std::string("cudaMalloc scene memory: ") + cudaGetErrorString(e));
    }
    s->memory_bytes = total + wide;
    char* at = (char*)s->memory;
    s->err_flag = at;
    s->ray_counters = at + 256;
    at += 256 + up256(8 * PT_RAY_COUNTERS);
    e = cudaMemset(s->err_flag, 0, sizeof(int));
    for (const Part& p : parts) {
        if (p.bytes == 0) continue;
        *p.dst = at;
        if (e == cudaSuccess) e = cudaMemcpy(at, p.src, p.bytes, cudaMemcpyHostToDevice);
        at += up256(p.bytes);
        s->device_bytes += p.bytes;
    }
    if (e != cudaSuccess) {
        free_scene(s.release());
        return cuda_fail(e, "scene upload");
    }
    if (wide && (rc = make_wide(s.get(), h, at))) { free_scene(s.release()); return rc; }
    if (wide && !s->dev.wide) {  // no records after all: their room goes back
        void* less = nullptr;
        e = cudaMalloc(&less, total);
        if (e == cudaSuccess) {
            char *from = (char*)s->memory, *to = (char*)less;
            e = cudaMemcpy(to, from, total, cudaMemcpyDeviceToDevice);
            if (e == cudaSuccess) e = cudaStreamSynchronize(nullptr);
            for (const Part& p : parts)
                if (p.bytes) *p.dst = to + ((char*)*p.dst - from);
            s->err_flag = to;
            s->ray_counters = to + 256;
            s->memory = to;
            s->memory_bytes = total;
            cudaFree(from);
            if (e != cudaSuccess) {
                free_scene(s.release());
                return cuda_fail(e, "scene upload");
            }
        } else {
            cudaGetLastError();
        }
    }
    *out = s.release();
    return PT_OK;
}
}  // namespace

extern "C" {

int pt_scene_create(const pt_scene_desc* desc, pt_scene** out) {
    if (!desc || !out) return fail(PT_EINVAL, "desc or out is NULL");
    *out = nullptr;
    int rc = device_count_ok();
    if (rc) return rc;
    HostScene h;
    rc = prepare_scene_host(desc, h);
    if (rc) return rc;
    return create_from_host(desc, h, out);
}

int pt_scene_create_two_level(const pt_scene_desc* desc, pt_scene** out) {
    if (!desc || !out) return fail(PT_EINVAL, "desc or out is NULL");
    *out = nullptr;
    int rc = device_count_ok();
    if (rc) return rc;
    HostScene h;
    rc = prepare_two_level_host(desc, h);
    if (rc) return rc;
    if (h.tlas_depth + 2 > (uint32_t)PT_TOP_STACK) return fail(PT_ESTACK, "top-level tree too deep");
    // the persistent path kernel keeps both levels and the instance-exit marker on one stack
    if (h.tlas_depth + h.max_depth + 4 > (uint32_t)PT_TRAVERSAL_STACK)
        return fail(PT_ESTACK, "top-level plus bottom-level tree depth exceeds the traversal stack");
    return create_from_host(desc, h, out);
}

int pt_two_level_plan(const pt_scene_desc* desc, pt_two_level_info* info) {
    if (!desc || !info) return fail(PT_EINVAL, "desc or info is NULL");
    HostScene h;
    int rc = prepare_two_level_host(desc, h);
    if (rc) return rc;
    info->num_instances = (uint32_t)h.instances.size();
    info->num_geometries = h.num_geometries;
    info->blas_nodes = (uint32_t)h.nodes.size();
    info->blas_faces = (uint32_t)(h.tris.size() / 12);
    info->tlas_nodes = (uint32_t)h.tlas.size();
    info->max_depth = h.max_depth;
    info->tlas_depth = h.tlas_depth;
    info->num_prims = h.num_prims;
    info->device_bytes = sizeof(pt_bvh_node) * (uint64_t)h.nodes.size() + 4ull * h.tris.size() +
                         sizeof(DeviceMesh) * (uint64_t)h.meshes.size() + 4ull * h.normals.size() +
                         4ull * h.light_tris.size() + 4ull * h.light_cdf.size() +
                         sizeof(DeviceInstance) * (uint64_t)h.instances.size() + sizeof(pt_bvh_node) * (uint64_t)h.tlas.size();
    return PT_OK;
}

int pt_scene_destroy(pt_scene* scene) {
    if (!scene) return PT_OK;
    free_scene(scene);
    return PT_OK;
}

int pt_scene_get_info(const pt_scene* s, pt_scene_info* info) {
    if (!s || !info) return fail(PT_EINVAL, "scene or info is NULL");
    info->num_nodes = s->num_nodes;
    info->num_prims = s->num_prims;
    info->num_meshes = s->num_meshes;
    info->max_depth = s->max_depth;
    info->device_bytes = s->device_bytes;
    return PT_OK;
}

int pt_scene_device_memory(pt_scene* s, uint64_t* bytes) {
    if (!s || !bytes) return fail(PT_EINVAL, "scene or bytes is NULL");
    std::lock_guard<std::mutex> lock(s->staging_mu);
    *bytes = s->memory_bytes + (s->staging_rays ? kStagingIn + kStagingOut + sizeof(int) : 0);
    return PT_OK;
}

int pt_trace(pt_scene* scene, const pt_ray* rays, uint64_t n, pt_hit* hits, uint32_t mem_flags, void* stream) {
    return scene_trace(scene, rays, n, hits, nullptr, nullptr, mem_flags, stream);
}

int pt_trace_counted(pt_scene* scene, const pt_ray* rays, uint64_t n, pt_hit* hits, uint32_t* node_tests,
                     uint32_t* tri_tests, uint32_t mem_flags, void* stream) {
    if (!node_tests && !tri_tests) return fail(PT_EINVAL, "no count outputs");
    return scene_trace(scene, rays, n, hits, node_tests, tri_tests, mem_flags, stream);
}

int pt_scene_set_trace_tuning(pt_scene* scene, const pt_trace_tuning* t) {
    if (!scene || !t) return fail(PT_EINVAL, "scene or tuning is NULL");
    if (t->shared_stack > 32 || (t->shared_stack & 7u))
        return fail(PT_EINVAL, "shared_stack must be 0, 8, 16, 24 or 32");
    if (t->queue_chunk < 32 || t->queue_chunk > 4096 || (t->queue_chunk & 31u))
        return fail(PT_EINVAL, "queue_chunk must be a multiple of 32 in [32, 4096]");
    scene->trace_tuning = *t;
    return PT_OK;
}

int pt_scene_get_trace_tuning(const pt_scene* scene, pt_trace_tuning* t) {
    if (!scene || !t) return fail(PT_EINVAL, "scene or tuning is NULL");
    *t = scene->trace_tuning;
    return PT_OK;
}

int pt_trace_autotune(pt_scene* scene, const pt_ray* rays_dev, uint64_t n, pt_hit* hits_dev, pt_trace_tuning* best,
                      float* best_ms) {
    if (!scene || !rays_dev || !hits_dev || !n) return fail(PT_EINVAL, "scene, rays or hits is NULL");
    const pt_trace_tuning saved = scene->trace_tuning;
    pt_trace_tuning cur = saved;
    float cur_ms = 1e30f;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    auto time_it = [&](const pt_trace_tuning& t, float& ms) -> int {
        scene->trace_tuning = t;
        int rc = pt_trace(scene, rays_dev, n, hits_dev, PT_MEM_DEVICE, nullptr);  // warm-up
        if (rc) return rc;
        ms = 1e30f;
        for (int r = 0; r < 5; ++r) {  // fastest of five single launches: robust to a noisy neighbour
            cudaEventRecord(e0, 0);
            if ((rc = pt_trace(scene, rays_dev, n, hits_dev, PT_MEM_DEVICE, nullptr))) return rc;
            cudaEventRecord(e1, 0);
            cudaEventSynchronize(e1);
            float one = 0.f;
            cudaEventElapsedTime(&one, e0, e1);
            ms = std::min(ms, one);
        }
        return PT_OK;
    };
    int rc = PT_OK;
    for (uint32_t sh : {0u, 8u, 16u, 24u, 32u}) {
        pt_trace_tuning t = cur;
        t.shared_stack = sh;
        float ms = 0.f;
        if ((rc = time_it(t, ms))) break;
        if (ms < cur_ms) { cur_ms = ms; cur = t; }
    }
    for (uint32_t ch : {32u, 64u, 128u, 256u}) {
        if (rc) break;
        pt_trace_tuning t = cur;
        t.queue_chunk = ch;
        float ms = 0.f;
        if ((rc = time_it(t, ms))) break;
        if (ms < cur_ms) { cur_ms = ms; cur = t; }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    scene->trace_tuning = rc ? saved : cur;
    if (rc) return rc;
    if (best) *best = cur;
    if (best_ms) *best_ms = cur_ms;
    return PT_OK;
}

// ---- exact-arithmetic hooks for the parity tests ------------------------------------------------

float pt_host_f64_diff_emulated(float a, float b, float c, float d) { return f64_diff_emulated(a, b, c, d); }

int pt_selftest_device(int which, const void* in, void* out, uint32_t n, uint64_t seed) {
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        return fail(PT_ECUDA, "no CUDA device available");
    }
    if (which < 0 || which > 3) return fail(PT_EINVAL, "unknown selftest");
    const size_t in_b = which == 1 ? 4 * (size_t)n : (which == 3 ? 64 * (size_t)n : 16 * (size_t)n);
    const size_t out_b = (which == 0 || which == 3) ? 4 * (size_t)n : (which == 1 ? 8 * (size_t)n : 16 * (size_t)n);
    void *din = nullptr, *dout = nullptr;
    if (cudaMalloc(&din, in_b) != cudaSuccess || cudaMalloc(&dout, out_b) != cudaSuccess) {
        if (din) cudaFree(din);
        return fail(PT_ENOMEM, "cudaMalloc selftest");
    }
    cudaMemcpy(din, in, in_b, cudaMemcpyHostToDevice);
    cudaError_t e;
    if (which == 0) e = launch_selftest_f64((const float*)din, (float*)dout, n, 0);
    else if (which == 1) e = launch_selftest_sincos((const float*)din, (float*)dout, n, 0);
    else if (which == 2) e = launch_selftest_philox((const uint32_t*)din, (uint32_t*)dout, n, seed, 0);
    else e = launch_selftest_box((const float*)din, (uint32_t*)dout, n, 0);
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, out_b, cudaMemcpyDeviceToHost);
    cudaFree(din);
    cudaFree(dout);
    if (e != cudaSuccess) return cuda_fail(e, "selftest");
    return PT_OK;
}

}  // extern "C"
