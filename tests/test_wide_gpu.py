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
