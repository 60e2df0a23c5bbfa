"""Frames over four-wide records against the binary walk on the B200: the same meshes and the same tree twice,
once with a leaf after its last node that no parent reaches, for which no records are made.  Every
pipeline of pt_render, pt_render_noalloc, batches and waves on both sides of the line between whole
paths and bounces must give the binary walk's film and primary ids, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import polytope_b200 as pb
from test_wide_gpu import AXIS_CAMERA
from test_wide_host_cpu import scene

pytestmark = pytest.mark.gpu
ENV = (51.0,) * 3


def both(name):
    """The scene with records, and without."""
    meshes = scene(name)
    nodes, pairs = pb.bvh_build(meshes)
    stray = nodes[np.nonzero(nodes["num_faces"] > 0)[0][:1]]
    wide = pb.Scene(meshes, env=ENV)
    binary = pb.Scene(meshes, env=ENV, nodes=np.concatenate([nodes, stray]), leaf_pairs=pairs)
    assert binary.device_memory() < binary.info().device_bytes + 16384
    assert wide.device_memory() >= binary.device_memory() + 32  # a record, less the stray node
    return wide, binary


def same(a, b, what):
    assert a[0].tobytes() == b[0].tobytes() and a[1].tobytes() == b[1].tobytes(), what


@pytest.mark.parametrize("size, spp", [((33, 33), 3), ((130, 67), 2)])
@pytest.mark.parametrize("name", ["small", "boxes", "grid", "strip", "coincident", "ulps"])
def test_frames_match_the_binary_walk(cuda_device, name, size, spp):
    import torch
    wide, binary = both(name)
    args = (size[0], size[1], spp, 5, AXIS_CAMERA, 9)
    for nee in (0, pb.RENDER_NEE):
        ref = pb.render(binary, *args, flags=nee | pb.RENDER_FUSED)
        for pipe in (0, pb.RENDER_FUSED, pb.RENDER_PERSISTENT, pb.RENDER_WAVEFRONT):
            same(pb.render(wide, *args, flags=nee | pipe), ref, (name, pipe))
            same(pb.render(binary, *args, flags=nee | pipe), ref, (name, pipe, "binary"))
        n = size[0] * size[1]
        rgb, prim = torch.zeros(3 * n, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
        d = pb.render_desc(size[0], size[1], spp, 5, AXIS_CAMERA, 9, nee)
        pb.check(pb.lib.pt_render_noalloc(wide.handle, C.byref(d), rgb.data_ptr(), prim.data_ptr(), None))
        assert wide.status() == pb.PT_OK
        same((rgb.cpu().numpy(), prim.cpu().numpy()), ref, (name, "noalloc"))


@pytest.mark.parametrize("pipeline", [pb.PIPELINE_FUSED, pb.PIPELINE_WAVEFRONT, pb.PIPELINE_PATHS])
@pytest.mark.parametrize("threads", [64, 128, 256])
def test_batches_match_the_binary_walk(cuda_device, pipeline, threads):
    t = pb.default_tuning()
    t.pipeline, t.threads_per_block = pipeline, threads
    pairs = [both("boxes"), both("small")]
    rds = [pb.render_desc(61 + 7 * k, 40, 3, 4, AXIS_CAMERA, k, pb.RENDER_NEE) for k in range(2)]
    ref = [pb.render(p[1], rd.width, rd.height, rd.spp, rd.max_depth, AXIS_CAMERA, int(rd.seed), pb.RENDER_NEE | pb.RENDER_FUSED)
           for p, rd in zip(pairs, rds)]
    for which in ((0, 0), (1, 0), (1, 1)):
        b = pb.Batch([(p[w], rd) for p, w, rd in zip(pairs, which, rds)], t)
        b.run()
        for i in range(2):
            same(b.output(i), ref[i], (which, i))
        b.close()


@pytest.mark.parametrize("width, depth, spp, wave", [(512, 2, 3, 0), (513, 2, 3, 0), (515, 0, 3, 256 * 600), (512, 0, 128, 1 << 25),
                                                     (512, 0, 129, 1 << 25)])
def test_waves_match_the_binary_walk(cuda_device, width, depth, spp, wave):
    """Waves that run as whole paths, bounce by bounce over records, and both in one batch."""
    wide, binary = both("boxes")
    t = pb.default_tuning()
    t.pipeline, t.wave_pixels = pb.PIPELINE_WAVEFRONT, wave
    rd = pb.render_desc(width, 256, spp, depth, AXIS_CAMERA, 4, pb.RENDER_NEE)
    ref = pb.render(binary, width, 256, spp, depth, AXIS_CAMERA, 4, pb.RENDER_NEE | pb.RENDER_FUSED)
    b = pb.Batch([(wide, rd)], t)
    b.run()
    same(b.output(0), ref, "batch")
    b.close()
    same(pb.render(wide, width, 256, spp, depth, AXIS_CAMERA, 4, pb.RENDER_NEE | pb.RENDER_WAVEFRONT), ref, "frame")
