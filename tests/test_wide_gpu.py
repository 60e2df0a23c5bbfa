"""Ray queries over the four-wide records against the counted query (the binary walk) on the B200: ray
counts around the warp, chunk and grid sizes, every shared-stack depth, rays along and almost along
the axes, trees of one leaf, leaves of more than six faces, coincident faces, and a caller's own tree
whose boxes do not nest (which keeps the binary walk)."""
import numpy as np
import pytest

import polytope_b200 as pb
from polytope_b200 import workloads as W
from test_traverse_host_cpu import edge_case_rays
from test_wide_host_cpu import axis_rays, copies, grid, scene, slanted_rays

pytestmark = pytest.mark.gpu


def same_hits(s, rays):
    got = s.intersect(rays)
    ref, _, _ = s.intersect(rays, counts=True)
    assert got.tobytes() == ref.tobytes(), int((got != ref).sum())


@pytest.mark.parametrize("name", ["small", "boxes", "instanced", "one face", "grid", "strip", "coincident", "ulps", "two of each"])
def test_wide_queries_match_the_binary_walk(cuda_device, name):
    s = pb.Scene(scene(name))
    same_hits(s, np.concatenate([edge_case_rays(40_000, 5), axis_rays(40_000, 6), slanted_rays(40_000, 7)]))
    s.close()


@pytest.mark.parametrize("n", [1, 2, 31, 33, 2959, 2961, 94_719, 94_721, 190_001, 1_000_003])
def test_ray_counts_around_warps_chunks_and_grids(cuda_device, n):
    s = pb.Scene(W.small_scene(4)[0])
    same_hits(s, edge_case_rays(n, n))
    s.close()


@pytest.mark.parametrize("chunk", [32, 64, 4096])
@pytest.mark.parametrize("n", [378_881, 757_763, 1_515_521])
def test_ray_counts_around_the_sizes_that_warps_take(cuda_device, n, chunk):
    """On 148 SMs, twice, four and eight times the chunks of 64 that all warps hold at once, and one more."""
    s = pb.Scene(W.small_scene(3)[0])
    s.set_trace_tuning(16, chunk)
    same_hits(s, np.resize(edge_case_rays(50_000, n), n))
    s.close()


@pytest.mark.parametrize("shared", [0, 8, 16, 24, 32])
def test_shared_stack_depths(cuda_device, shared):
    s = pb.Scene(scene("boxes"))
    s.set_trace_tuning(shared, 32 if shared else 4096)
    same_hits(s, edge_case_rays(70_000, 3))
    s.close()


def test_a_tree_whose_boxes_do_not_nest_keeps_its_own_hits(cuda_device):
    meshes = scene("small")
    nodes, pairs = pb.bvh_build(meshes)
    leaf = np.nonzero(nodes["num_faces"] > 0)[0][::3]
    nodes["bb"][leaf, 3:6] += np.float32(0.25)
    nodes["bb"][leaf[::2], 0] += np.float32(0.01)  # and some that leave out part of their faces
    s = pb.Scene(meshes, nodes=nodes, leaf_pairs=pairs)
    same_hits(s, edge_case_rays(60_000, 8))
    s.close()


def test_large_leaf_and_grid_together(cuda_device):
    s = pb.Scene([copies(300, 0), grid(40)])
    same_hits(s, np.concatenate([axis_rays(50_000, 1), edge_case_rays(50_000, 2)]))
    s.close()


AXIS_CAMERA = dict(eye=(0.0, 0.0, 7.0), look_at=(0.0, 0.0, 0.0), up=(0.0, 1.0, 0.0), fov=50.0)


def loose(name):
    """The scene over a tree of the caller's own whose boxes do not nest."""
    meshes = scene(name)
    nodes, pairs = pb.bvh_build(meshes)
    nodes["bb"][np.nonzero(nodes["num_faces"] > 0)[0][::3], 3:6] += np.float32(0.25)
    return pb.Scene(meshes, env=(51.0,) * 3, nodes=nodes, leaf_pairs=pairs)


@pytest.mark.parametrize("size, spp", [((1, 1), 1), ((33, 33), 3), ((130, 67), 2), ((257, 255), 1)])
@pytest.mark.parametrize("name", ["small", "boxes", "grid", "coincident"])
def test_wide_frames_match_the_fused_walk(cuda_device, name, size, spp):
    """The path and wavefront kernels over four-wide records against the one-thread-per-path kernel, with
    a camera whose middle rays run along an axis."""
    s = pb.Scene(scene(name), env=(51.0,) * 3)
    args = (size[0], size[1], spp, 5, AXIS_CAMERA, 9)
    for nee in (0, pb.RENDER_NEE):
        film, prim = pb.render(s, *args, flags=nee | pb.RENDER_FUSED)
        for pipe in (0, pb.RENDER_PERSISTENT, pb.RENDER_WAVEFRONT):
            got, gprim = pb.render(s, *args, flags=nee | pipe)
            assert got.tobytes() == film.tobytes() and gprim.tobytes() == prim.tobytes(), (name, pipe)
    s.close()


@pytest.mark.parametrize("pipeline", [pb.PIPELINE_WAVEFRONT, pb.PIPELINE_PATHS])
@pytest.mark.parametrize("threads", [64, 128, 256])
def test_batches_with_and_without_records(cuda_device, pipeline, threads):
    scenes = [pb.Scene(scene("boxes"), env=(51.0,) * 3), loose("small"), pb.Scene(scene("small"), env=(51.0,) * 3)]
    t = pb.default_tuning()
    t.pipeline, t.threads_per_block = pipeline, threads
    for pick in ([0, 2], [0, 1, 2]):
        jobs = [(scenes[k], pb.render_desc(61 + 7 * k, 40, 3, 4, AXIS_CAMERA, k, pb.RENDER_NEE)) for k in pick]
        b = pb.Batch(jobs, t)
        b.run()
        for i, (s, rd) in enumerate(jobs):
            film, prim = pb.render(s, rd.width, rd.height, rd.spp, rd.max_depth, AXIS_CAMERA, int(rd.seed),
                                   pb.RENDER_NEE | pb.RENDER_FUSED)
            got, gprim = b.output(i)
            assert got.tobytes() == film.tobytes() and gprim.tobytes() == prim.tobytes(), (pick, i)
        b.close()
    for s in scenes:
        s.close()


@pytest.mark.parametrize("threads", [64, 128, 256])
@pytest.mark.parametrize("width, depth, spp, wave", [(512, 0, 1, 0), (513, 0, 1, 0), (512, 2, 3, 0), (513, 2, 3, 0), (515, 0, 3, 256 * 600),
                                                       (512, 0, 128, 1 << 25), (512, 0, 129, 1 << 25)])
def test_waves_around_the_whole_path_limit(cuda_device, threads, width, depth, spp, wave):
    """Waves of up to 131,072 paths a bounce run as whole paths, larger ones bounce by bounce; the fifth
    case has two of the one kind and one of the other in a batch.  Up to 2^24 paths those walk the records,
    above the binary nodes."""
    s = pb.Scene(scene("boxes"), env=(51.0,) * 3)
    t = pb.default_tuning()
    t.pipeline, t.threads_per_block, t.wave_pixels = pb.PIPELINE_WAVEFRONT, threads, wave
    rd = pb.render_desc(width, 256, spp, depth, AXIS_CAMERA, 4, pb.RENDER_NEE)
    film, prim = pb.render(s, width, 256, spp, depth, AXIS_CAMERA, 4, pb.RENDER_NEE | pb.RENDER_FUSED)
    b = pb.Batch([(s, rd)], t)
    b.run()
    got, gprim = b.output(0)
    assert got.tobytes() == film.tobytes() and gprim.tobytes() == prim.tobytes()
    b.close()
    got, gprim = pb.render(s, width, 256, spp, depth, AXIS_CAMERA, 4, pb.RENDER_NEE | pb.RENDER_WAVEFRONT)
    assert got.tobytes() == film.tobytes() and gprim.tobytes() == prim.tobytes()
    s.close()


def instances(name):
    if name == "one":
        return W.instanced_scene(level=2, instances=1)[0][1:2]
    if name == "forty":
        return W.instanced_scene(level=3, instances=40)[0]
    if name == "leaves":  # geometries of one leaf, one of them large, under identity and other transforms
        m = [copies(20, 0), grid(3)]
        o = W.instanced_scene(level=2, instances=3)[0][1].object_to_world
        return m + [pb.Mesh(m[0].x, m[0].y, m[0].z, m[0].faces, object_to_world=o)]
    return W.instanced_scene(level=5, instances=5)[0]


@pytest.mark.parametrize("name", ["one", "five", "forty", "leaves"])
def test_two_level_queries_match_the_counted_walk(cuda_device, name):
    s = pb.Scene(instances(name), two_level=True)
    for n in (1, 33, 2369, 100_003):
        same_hits(s, np.concatenate([edge_case_rays(n, 5), axis_rays(n, 6), slanted_rays(n, 7)]))
    s.close()


@pytest.mark.parametrize("name", ["one", "five", "forty", "leaves"])
def test_two_level_frames_match_the_fused_walk(cuda_device, name):
    s = pb.Scene(instances(name), env=(51.0,) * 3, two_level=True)
    for size, spp in (((1, 1), 1), ((33, 33), 3), ((130, 67), 2)):
        args = (size[0], size[1], spp, 5, AXIS_CAMERA, 9)
        film, prim = pb.render(s, *args, flags=pb.RENDER_NEE | pb.RENDER_FUSED)
        got, gprim = pb.render(s, *args, flags=pb.RENDER_NEE | pb.RENDER_PERSISTENT)
        assert got.tobytes() == film.tobytes() and gprim.tobytes() == prim.tobytes()
    s.close()


@pytest.mark.parametrize("n", [65_535, 65_536, 65_537, 131_073, 4_300_007])
def test_host_arrays_around_the_worker_threshold(cuda_device, n):
    """Pageable arrays in parallel from 65,536 rays on; rays or hits in pinned memory beside them."""
    import torch
    s = pb.Scene(W.small_scene(3)[0])
    rays = np.resize(edge_case_rays(50_000, 11), n)
    ref, _, _ = s.intersect(rays, counts=True)
    assert s.intersect(rays).tobytes() == ref.tobytes()
    pinned_rays = torch.empty(32 * n, dtype=torch.uint8).pin_memory().numpy().view(pb.RAY_DTYPE)
    pinned_hits = torch.empty(16 * n, dtype=torch.uint8).pin_memory().numpy().view(pb.HIT_DTYPE)
    pinned_rays[:] = rays
    assert s.intersect(pinned_rays).tobytes() == ref.tobytes()
    s.intersect(rays, pinned_hits)
    assert pinned_hits.tobytes() == ref.tobytes()
    s.close()


def test_host_arrays_from_several_threads(cuda_device):
    from concurrent.futures import ThreadPoolExecutor
    s = pb.Scene(W.small_scene(4)[0])
    sets = [edge_case_rays(100_000 + 7 * k, k) for k in range(6)]
    ref = [s.intersect(r, counts=True)[0].tobytes() for r in sets]
    with ThreadPoolExecutor(6) as ex:
        for _ in range(3):
            assert [h.tobytes() for h in ex.map(s.intersect, sets)] == ref
    s.close()
