"""The calls that programs built on polytope_b200 spend their time in, with inputs to time them on.

A case is a dict of plain values.  `listed()` names twelve; `draw(rng)` gives another one of the
same ranges.  Three families:

* ray queries (`kind` "query"): `Scene.intersect` on buffers of the device or of the host, closest
  hits and occlusion tests, from a thousand rays to the 16.7 M of the intersection microbench, on
  trees of 1 k to 1.3 M faces, flattened or two-level;
* frames ("frame"): `render`, `render_rgba8` and the C ABI's `pt_render` into device memory;
* many renders at once: `Batch` ("batch") and `Server` ("serve").

The scenes are those of `polytope_b200.workloads`, with seeded meshes, transforms and materials.
"""
import ctypes as C
import math

import numpy as np
import torch

import polytope_b200 as pb
from polytope_b200 import workloads as W


def listed():
    return [
        # picking and collision tests: a thousand rays at a time against one object; latency
        dict(name="query_1k", kind="query", scene="sphere", level=5, rays=1000, any=0.0, source="ball"),
        # a sensor sweep (lidar) or a low-resolution visibility buffer in a scene of boxes, ragged count
        dict(name="query_boxes_100k", kind="query", scene="boxes", faces=100_000, rays=100_003, any=0.0, source="ball"),
        # light baking: occlusion rays from points of a surface to an area light, in surface order
        dict(name="occlusion_1m", kind="query", scene="sphere", level=7, rays=1_000_000, any=1.0, source="surface"),
        # the intersection microbench: incoherent rays, half closest hit, half any hit
        dict(name="query_16m", kind="query", scene="sphere", level=8, rays=16_777_216, any=0.5, source="ball"),
        # the same call on the caller's own host arrays: rays copied in, hits copied out
        dict(name="query_host_1m", kind="query", scene="sphere", level=6, rays=1_048_577, any=0.25, source="ball", host=True),
        # queries on an instanced scene that keeps one copy of its geometry
        dict(name="query_two_level_1m", kind="query", scene="instanced", level=6, instances=5, two_level=True, rays=1_000_000,
             any=0.5, source="shell"),
        # a preview frame: the small configuration, film back on the host
        dict(name="frame_small", kind="frame", scene="sphere", level=5, out="host", width=320, height=240, spp=8, depth=4,
             flags=pb.RENDER_NEE),
        # a full-HD frame of a scene larger than the L2 cache, film left on the device (progressive viewers)
        dict(name="frame_hd", kind="frame", scene="instanced", level=8, instances=3, out="device", width=1920, height=1080, spp=16,
             depth=8, flags=pb.RENDER_NEE),
        # the frame as the reference's PNG output stores it, odd size, jittered, without light sampling
        dict(name="frame_rgba8", kind="frame", scene="boxes", faces=20_000, out="rgba8", width=641, height=479, spp=4, depth=6,
             flags=pb.RENDER_JITTER),
        # an instanced scene rendered from its two-level layout
        dict(name="frame_two_level", kind="frame", scene="instanced", level=7, instances=5, two_level=True, out="device", width=1280,
             height=720, spp=8, depth=8, flags=pb.RENDER_NEE),
        # uneven scenes in one batch (thumbnails, training views): replay and read the films
        dict(name="batch_24", kind="batch", scenes=24, max_faces=200_000, max_res=256, max_spp=64, depth=6, flags=pb.RENDER_NEE),
        # a render service: a burst of mixed requests over resident scenes, films fetched in order
        dict(name="serve_24", kind="serve", scenes=4, requests=24, max_res=512, max_spp=16, depth=5, flags=pb.RENDER_NEE),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["query", "query", "query", "host", "two_level", "frame", "frame", "frame_two_level", "batch", "serve"])
    if kind in ("query", "host"):
        c = dict(kind="query", rays=_log_int(rng, 500, 4_000_000 if kind == "query" else 1_000_000),
                 any=rng.choice([0.0, 0.25, 0.5, 1.0]), source=rng.choice(["ball", "ball", "surface"]))
        if rng.random() < 0.5:
            c.update(scene="sphere", level=rng.randint(3, 8))
        else:
            c.update(scene="boxes", faces=_log_int(rng, 1000, 500_000), source="ball")
        if kind == "host":
            c["host"] = True
        return c
    if kind == "two_level":
        return dict(kind="query", scene="instanced", level=rng.randint(4, 7), instances=rng.randint(1, 8), two_level=True,
                    rays=_log_int(rng, 1000, 1_000_000), any=rng.choice([0.0, 0.5, 1.0]), source="shell")
    if kind in ("frame", "frame_two_level"):
        width = _log_int(rng, 64, 1400)
        c = dict(kind="frame", out=rng.choice(["host", "device", "rgba8"]), width=width, height=max(48, int(width * rng.uniform(0.5, 1.0))),
                 spp=rng.choice([1, 2, 4, 7, 8]), depth=rng.randint(1, 8),
                 flags=rng.choice([0, pb.RENDER_NEE, pb.RENDER_NEE, pb.RENDER_NEE | pb.RENDER_JITTER]))
        if kind == "frame_two_level":
            c.update(scene="instanced", level=rng.randint(4, 7), instances=rng.randint(1, 8), two_level=True)
        else:
            c.update(rng.choice([dict(scene="sphere", level=rng.randint(3, 8)), dict(scene="boxes", faces=_log_int(rng, 1000, 500_000)),
                                 dict(scene="instanced", level=rng.randint(5, 7), instances=rng.randint(1, 6))]))
            c["flags"] |= rng.choice([0, 0, 0, pb.RENDER_WAVEFRONT, pb.RENDER_FUSED])
        return c
    if kind == "batch":
        return dict(kind="batch", scenes=rng.randint(2, 24), max_faces=_log_int(rng, 5000, 200_000), max_res=rng.choice([64, 128, 256]),
                    max_spp=rng.choice([4, 16, 64]), depth=rng.randint(2, 6), flags=rng.choice([0, pb.RENDER_NEE]))
    return dict(kind="serve", scenes=rng.randint(1, 4), requests=rng.randint(2, 24), max_res=rng.choice([128, 256, 512]),
                max_spp=rng.choice([1, 4, 16]), depth=rng.randint(2, 5), flags=pb.RENDER_NEE)


# ---- scenes and inputs ---------------------------------------------------------------------------

def _faces(case):
    if case["scene"] == "boxes":
        return case["faces"]
    per = 20 * 4 ** case["level"]
    return per * case["instances"] if case["scene"] == "instanced" else per


def _meshes(case, seed):
    """(meshes, environment) of a query or frame case; the displaced sphere is mesh 1."""
    if case["scene"] == "instanced":
        return W.instanced_scene(case["level"], case["instances"], seed=seed, noise_seed=7)
    if case["scene"] == "boxes":
        return W.batch_scene(case["faces"], np.random.default_rng(seed))
    x, y, z, f = pb.icosphere(case["level"], 1.0, 0.05, seed)
    return [W.quad(-1.5, 10.0), pb.Mesh(x, y, z, f), W.quad(4.0, 1.0, is_light=True, emission=(2550.0,) * 3)], (51.0,) * 3


def _unit(v):
    return v / v.norm(dim=1, keepdim=True)


def _ball(n, g):
    """n uniform points of the unit ball."""
    return _unit(torch.randn(n, 3, generator=g, device="cuda")) * torch.rand(n, 1, generator=g, device="cuda") ** (1 / 3)


def _rays(case, seed, meshes):
    """(n, 8) float32 pt_ray records on the device.  "ball": from a sphere of radius 3 to uniform
    points of the unit ball; "shell": from a sphere of radius 12 to points where the instances
    are; "surface": from points of the sphere mesh, in face order, to points of the light."""
    n = case["rays"]
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    if case["source"] == "surface":
        m = meshes[1]
        v = torch.from_numpy(np.stack([m.x, m.y, m.z], 1)).cuda()
        f = torch.from_numpy(m.faces.astype(np.int64)).cuda()[torch.randint(len(m.faces), (n,), generator=g, device="cuda").sort().values]
        w = torch.rand(n, 3, generator=g, device="cuda") + 1e-3
        w = w / w.sum(1, keepdim=True)
        a, b, c = v[f[:, 0]], v[f[:, 1]], v[f[:, 2]]
        p = a * w[:, :1] + b * w[:, 1:2] + c * w[:, 2:]
        normal = _unit(torch.linalg.cross(b - a, c - a))
        normal = torch.where((normal * p).sum(1, keepdim=True) < 0, -normal, normal)
        org = p + 1e-3 * normal
        target = torch.rand(n, 3, generator=g, device="cuda") * 2 - 1
        target[:, 1] = 4.0
    elif case["source"] == "shell":
        org = 12.0 * _unit(torch.randn(n, 3, generator=g, device="cuda"))
        target = torch.rand(n, 3, generator=g, device="cuda") * 9 - 4.5
    else:
        org = 3.0 * _unit(torch.randn(n, 3, generator=g, device="cuda"))
        target = _ball(n, g)
    any_hit = torch.rand(n, generator=g, device="cuda") < case["any"]
    d = target - org
    dist = d.norm(dim=1)
    rays = torch.empty(n, 8, device="cuda")
    rays[:, 0:3] = org
    rays[:, 3] = torch.where(any_hit, 0.999 * dist if case["source"] == "surface" else dist, torch.full_like(dist, math.inf))
    rays[:, 4:7] = d / dist[:, None]
    rays[:, 7] = any_hit.to(torch.int32).view(torch.float32)
    return rays


def _frames(rng, scenes, count, resolutions, spps, case):
    """The case's mix of resolutions and sample counts (the same for every seed), on scenes and with
    render seeds of its own."""
    mix = np.random.default_rng(23)
    out = []
    for _ in range(count):
        res = int(mix.choice([r for r in resolutions if r <= case["max_res"]]))
        spp = int(mix.choice([s for s in spps if s <= case["max_spp"]]))
        camera = W.SERVE_CAMERA if case["kind"] == "serve" else W.BATCH_CAMERA
        out.append((scenes[len(out) % len(scenes)] if case["kind"] == "batch" else scenes[int(rng.integers(len(scenes)))],
                    pb.render_desc(res, res, spp, case["depth"], camera, int(rng.integers(1 << 30)), case["flags"])))
    return out


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    if case["kind"] == "batch":
        scenes = []
        for _ in range(case["scenes"]):
            scenes.append(pb.Scene(*W.batch_scene(int(np.exp(rng.uniform(np.log(1000), np.log(case["max_faces"])))), rng)))
        jobs = _frames(rng, scenes, case["scenes"], (64, 128, 256), (4, 16, 64), case)
        return dict(case=case, batch=pb.Batch(jobs), scenes=scenes)
    if case["kind"] == "serve":
        scenes = [pb.Scene(*W.instanced_scene(6, int(rng.integers(1, 6)), seed=int(rng.integers(1 << 30)))) for _ in range(case["scenes"])]
        tuning = pb.default_tuning()
        tuning.pipeline = pb.PIPELINE_PATHS
        server = pb.Server(max_inflight=64, memory_budget=1 << 30, wave_pixels=1 << 22, tuning=tuning, host_budget=1 << 28)
        return dict(case=case, server=server, jobs=_frames(rng, scenes, case["requests"], (128, 256, 512), (1, 4, 16), case), scenes=scenes)
    meshes, env = _meshes(case, seed)
    state = dict(case=case, scene=pb.Scene(meshes, env, two_level=case.get("two_level", False)))
    if case["kind"] == "query":
        rays = _rays(case, seed, meshes)
        if case.get("host"):
            state["rays"] = rays.cpu().numpy().view(pb.RAY_DTYPE).reshape(-1)
            state["hits"] = np.zeros(case["rays"], pb.HIT_DTYPE)
        else:
            state["rays"] = rays
            state["hits"] = torch.zeros(case["rays"], 4, device="cuda")
        return state
    camera = W.INSTANCED_CAMERA if case["scene"] == "instanced" else W.BATCH_CAMERA
    state["args"] = (case["width"], case["height"], case["spp"], case["depth"], camera, seed & 0xFFFF, case["flags"])
    if case["out"] == "device":
        state["desc"] = pb.render_desc(*state["args"])
        state["rgb"] = torch.zeros(case["height"], case["width"], 3, device="cuda")
        state["prim"] = torch.zeros(case["height"], case["width"], dtype=torch.int32, device="cuda")
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        state["batch"].run()
        return [(rgb, prim.view(np.int32)) for rgb, prim in (state["batch"].output(i) for i in range(case["scenes"]))]
    if case["kind"] == "serve":
        server = state["server"]
        tickets = [server.submit(scene, desc) for scene, desc in state["jobs"]]
        films = []
        for t in tickets:
            server.wait(t)
            rgb, prim = server.fetch(t)
            films.append((rgb, prim.view(np.int32)))
        return films
    scene = state["scene"]
    if case["kind"] == "query":
        if case.get("host"):
            h = scene.intersect(state["rays"], state["hits"])
            return dict(prim=h["prim"].view(np.int32), t=h["t"], u=h["u"], v=h["v"])
        h = scene.intersect(state["rays"], state["hits"], device=True, stream=torch.cuda.current_stream().cuda_stream)
        return dict(prim=h.view(torch.int32)[:, 0], t=h[:, 1], u=h[:, 2], v=h[:, 3])
    if case["out"] == "host":
        rgb, prim = pb.render(scene, *state["args"])
        return dict(rgb=rgb, prim=prim.view(np.int32))
    if case["out"] == "rgba8":
        rgba, prim = pb.render_rgba8(scene, *state["args"])
        return dict(rgba=rgba, prim=prim.view(np.int32))
    pb.check(pb.lib.pt_render(scene.handle, C.byref(state["desc"]), state["rgb"].data_ptr(), state["prim"].data_ptr(), pb.MEM_DEVICE,
                              torch.cuda.current_stream().cuda_stream or None))
    return dict(rgb=state["rgb"], prim=state["prim"])


# ---- what a pass cannot do without ---------------------------------------------------------------

def work(case):
    """Rays and hits (or films) once, and the part of the tree that the rays can reach once: about
    1.75 kB a ray, up to the whole tree (32 B a node, 1.2 nodes and a 48 B record a face).  Flops: per
    ray about 2.4 log2(faces) box tests of 18 operations and 3.2 face tests of 60."""
    if case["kind"] in ("batch", "serve"):
        count = case["scenes"] if case["kind"] == "batch" else case["requests"]
        res = [r for r in ((64, 128, 256) if case["kind"] == "batch" else (128, 256, 512)) if r <= case["max_res"]]
        spp = [s for s in ((4, 16, 64) if case["kind"] == "batch" else (1, 4, 16)) if s <= case["max_spp"]]
        pixels = count * sum(r * r for r in res) / len(res)
        samples = pixels * sum(spp) / len(spp)
        faces = math.sqrt(1000.0 * case["max_faces"]) if case["kind"] == "batch" else 3 * 81920
        trees, rays, io = case["scenes"], 3.0 * samples, 16 * pixels
    elif case["kind"] == "frame":
        pixels = case["width"] * case["height"]
        faces, trees, rays = _faces(case), 1, 2.4 * pixels * case["spp"]
        io = (8 if case["out"] == "rgba8" else 16) * pixels
    else:
        faces, trees, rays, io = _faces(case), 1, case["rays"], 48 * case["rays"]
    if case.get("two_level"):
        faces /= case["instances"]
    tree = min(trees * faces * (48 + 1.2 * 32), 1750.0 * rays)
    return {"bytes": io + tree, "flops": rays * (2.4 * math.log2(max(2.0, faces)) * 18 + 3.2 * 60)}


def exact(case, seed):
    """Closest hits in 64 bits by testing every face (Moeller and Trumbore, "Fast, minimum storage
    ray/triangle intersection", 1997): only where that is quick.  An occlusion query's hit is the
    first face that its walk accepts, and a path-traced film follows 32-bit rays bounce by bounce:
    neither has such a value."""
    if case["kind"] != "query" or case["any"] or case.get("two_level") or case["rays"] * _faces(case) > 1.2e11:
        return None
    meshes, _ = _meshes(case, seed)
    rays = _rays(case, seed, meshes).double()
    tri = torch.cat([torch.from_numpy(np.stack([m.x, m.y, m.z], 1)[m.faces.astype(np.int64)]) for m in meshes]).cuda().double()
    v0, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    n = case["rays"]
    prim = torch.empty(n, dtype=torch.int64, device="cuda")
    t_out, u_out, v_out = (torch.empty(n, dtype=torch.float64, device="cuda") for _ in range(3))
    normal = torch.linalg.cross(e1, e2)
    step = max(1, int(4e7 // len(tri)))
    for at in range(0, n, step):
        o, d, tmax = rays[at:at + step, 0:3], rays[at:at + step, 4:7], rays[at:at + step, 3]
        # with c = o x d:  det = -d.(e1 x e2),  u det = (o - v0).(d x e2),  v det = -(o - v0).(d x e1)
        c = torch.linalg.cross(o, d)
        det = -(d @ normal.T)
        u = (c @ e2.T - d @ torch.linalg.cross(e2, v0).T) / det
        v = -(c @ e1.T - d @ torch.linalg.cross(e1, v0).T) / det
        t = (o @ normal.T - (v0 * normal).sum(1)) / det
        t = torch.where((u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0), t, torch.inf)
        best, face = t.min(1)
        hit = best <= tmax
        hit &= best < torch.inf
        row = torch.arange(len(best), device="cuda")
        b1, b2 = u[row, face], v[row, face]
        prim[at:at + step] = torch.where(hit, face, -1)
        t_out[at:at + step] = torch.where(hit, best, tmax)
        # pt_hit's u and v are the weights of the face's first and second vertex
        u_out[at:at + step] = torch.where(hit, 1 - b1 - b2, 0.0)
        v_out[at:at + step] = torch.where(hit, b1, 0.0)
    if case.get("host"):
        return dict(prim=prim.cpu().numpy(), t=t_out.cpu().numpy(), u=u_out.cpu().numpy(), v=v_out.cpu().numpy())
    return dict(prim=prim, t=t_out, u=u_out, v=v_out)
