"""What a scene handle says of the device memory it holds (pt_scene_device_memory), on the B200."""
import numpy as np
import pytest

import polytope_b200 as pb
from polytope_b200 import workloads as W
from test_traverse_host_cpu import edge_case_rays
from test_wide_gpu import AXIS_CAMERA, instances, loose
from test_wide_host_cpu import scene

pytestmark = pytest.mark.gpu
STAGING = 4 * (1 << 20) * (32 + 16)


def even_nodes(meshes):
    """Interior nodes at even depth, and the root: each starts a four-wide record."""
    nodes, _ = pb.bvh_build(meshes)
    depth, records = np.zeros(len(nodes), int), 0
    for i, n in enumerate(nodes):
        leaf = n["num_faces"] > 0
        if not leaf:
            depth[i + 1] = depth[i + int(n["offset"])] = depth[i] + 1
        records += i == 0 or (not leaf and depth[i] % 2 == 0)
    return records


@pytest.mark.parametrize("name", ["small", "boxes", "one face"])
def test_memory_of_a_scene_with_records(cuda_device, name):
    meshes = scene(name)
    s = pb.Scene(meshes)
    arrays, records = s.info().device_bytes, 64 * even_nodes(meshes)
    held = s.device_memory()
    assert arrays + records <= held <= arrays + records + 4 * s.info().num_nodes + 16384
    s.intersect(edge_case_rays(100, 1))
    assert held + STAGING <= s.device_memory() <= held + STAGING + 256
    s.close()


def test_memory_of_a_two_level_scene(cuda_device):
    s = pb.Scene(instances("five"), two_level=True)
    info = s.info()
    assert info.device_bytes < s.device_memory() < 1.5 * info.device_bytes + 16384
    s.close()


def stretched(meshes, factor):
    """The meshes' vertices, `factor` times as large."""
    m = [np.asarray(x, np.float32) * np.float32(factor) for x in (meshes[0].x, meshes[0].y, meshes[0].z)]
    return [pb.Mesh(*m, meshes[0].faces)]


def test_a_scene_without_records_holds_no_room_for_them(cuda_device):
    """A tree whose boxes do not nest, found when the records are made, and one of extreme size."""
    s = loose("small")
    assert s.info().device_bytes <= s.device_memory() <= s.info().device_bytes + 16384
    rays = edge_case_rays(70_000, 4)
    # the handle's arrays have moved: queries, frames and the guard flag still meet them
    assert s.intersect(rays).tobytes() == s.intersect(rays, counts=True)[0].tobytes()
    film, prim = pb.render(s, 65, 33, 2, 4, AXIS_CAMERA, 3, pb.RENDER_NEE | pb.RENDER_FUSED)
    got, gprim = pb.render(s, 65, 33, 2, 4, AXIS_CAMERA, 3, pb.RENDER_NEE)
    assert got.tobytes() == film.tobytes() and gprim.tobytes() == prim.tobytes()
    assert s.status() == 0
    s.close()
    far = pb.Scene(stretched(scene("grid"), 2.0 ** 32))
    assert far.info().device_bytes <= far.device_memory() <= far.info().device_bytes + 16384
    far.close()
