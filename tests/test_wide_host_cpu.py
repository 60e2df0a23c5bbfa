"""The walk over four-wide records (polytope_b200/csrc/wide.cuh) compiled for the host against the
binary walk: the same face, t, u, v and w, bit for bit, on every ray that it takes -- closest hits and
first accepted any-hit faces, zero and negative-zero direction components, origins inside boxes and
on their planes, far bounds of 0 and infinity, deep and single-leaf trees, leaves of more than six
faces, coincident faces (where MinT rises by an ulp and the ray goes back to the binary walk)."""
import os
import subprocess

import numpy as np
import pytest

import polytope_b200 as pb
from polytope_b200 import workloads as W
from golden.make_golden import box_edge_rays, random_rays
from oracle import pyoracle as po
from test_traverse_host_cpu import NVCC, ROOT, edge_case_rays, leaf_ordered_faces

pytestmark = pytest.mark.skipif(NVCC is None, reason="needs nvcc (host compilation only)")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = tmp_path_factory.mktemp("wide") / "wide_host_check"
    subprocess.run([NVCC, "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off,-fno-fast-math",
                    "-I", os.path.join(ROOT, "polytope_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "wide_host_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    return exe


def axis_rays(n, seed):
    """Rays along the axes (with both signs of zero) from lattice points, where box planes lie."""
    rng = np.random.default_rng(seed)
    rays = np.zeros(n, pb.RAY_DTYPE)
    d = np.where(rng.random((n, 3)) < 0.5, np.float32(0.0), np.float32(-0.0))
    d[np.arange(n), rng.integers(0, 3, n)] = rng.choice([-1.0, 1.0], n)
    rays["dir"] = d
    rays["org"] = rng.choice(np.array([-2.0, -1.5, -1.0, -0.5, 0.0, 0.25, 0.5, 1.0, 4.0], np.float32), (n, 3))
    rays["tmax"] = rng.choice(np.array([np.inf, 0.0, 0.5, 1.0, 2.0], np.float32), n)
    rays["flags"] = rng.integers(0, 2, n)
    return rays


def slanted_rays(n, seed):
    """Rays almost along an axis (components down to 2^-70 of the largest), directions of lengths from
    2^-24 to 2^24, origins from inside the scene to 2^22 scene sizes away."""
    rng = np.random.default_rng(seed)
    rays = np.zeros(n, pb.RAY_DTYPE)
    d = rng.normal(size=(n, 3)) * np.exp2(rng.integers(-70, 1, (n, 3)) * (rng.random((n, 3)) < 0.4))
    d = d / np.abs(d).max(1)[:, None]
    target = rng.uniform(-1.2, 1.2, (n, 3))
    org = target - d * np.exp2(rng.uniform(-3, 22, n) * (rng.random(n) < 0.4))[:, None]
    scale = np.exp2(rng.uniform(-24, 24, n) * (rng.random(n) < 0.3))
    rays["org"], rays["dir"] = org, d * scale[:, None]
    rays["tmax"] = np.where(rng.random(n) < 0.5, np.inf, np.abs(rng.normal(size=n)) * 3 / scale)
    rays["flags"] = rng.integers(0, 2, n)
    return rays


def grid(n):
    """An n x n lattice of axis-aligned unit quads in the plane y = 0: faces on box planes, exact ties."""
    i, j = np.meshgrid(np.arange(n), np.arange(n), indexing="ij")
    v = np.stack([i.ravel(), j.ravel()], 1)
    x = ((v[:, 0:1] + [0, 1, 1, 0]) * 0.5 - 2).ravel().astype(np.float32)
    z = ((v[:, 1:2] + [0, 0, 1, 1]) * 0.5 - 2).ravel().astype(np.float32)
    f = (np.array([[0, 1, 2], [0, 2, 3]])[None] + 4 * np.arange(n * n)[:, None, None]).reshape(-1, 3)
    return pb.Mesh(x, np.zeros_like(x), z, f.astype(np.uint32))


def strip(n):
    """Triangles whose sizes double along x: a chain-like, deep tree."""
    s = 2.0 ** -np.arange(n)
    x = np.stack([s, 1.5 * s, s], 1).ravel().astype(np.float32)
    y = np.stack([0 * s, 0 * s, 0.4 * s], 1).ravel().astype(np.float32)
    return pb.Mesh(x, y, np.zeros_like(x), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3))


def copies(n, shift):
    """n copies of one triangle, each `shift` ulps further along z: one leaf of n faces when shift is 0."""
    z = np.full((n, 3), 1.0, np.float32)
    for k in range(n):
        for _ in range(shift * k):
            z[k] = np.nextafter(z[k], np.float32(2))
    x = np.tile(np.float32([-1, 1, 0.1]), n)
    y = np.tile(np.float32([-1, -0.9, 1.1]), n)
    return pb.Mesh(x, y, z.ravel(), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3))


def scene(name):
    if name == "small":
        return W.small_scene()[0]
    if name == "boxes":
        return W.batch_scene(30_000, np.random.default_rng(3))[0]
    if name == "instanced":
        return W.instanced_scene(level=4, instances=5)[0]
    if name == "one face":
        return [pb.Mesh([-1, 1, 0], [-1, -1, 1], [0, 0, 0.5], [[0, 1, 2]])]
    return {"grid": [grid(9)], "strip": [strip(60)], "coincident": [copies(20, 0), grid(4)], "ulps": [copies(40, 1)],
            "two of each": [grid(5), grid(5), W.small_scene(2)[0][1], W.small_scene(2)[0][1]]}[name]


@pytest.mark.parametrize("name", ["small", "boxes", "instanced", "one face", "grid", "strip", "coincident", "ulps", "two of each"])
def test_wide_walk_gives_the_binary_walks_hits(harness, tmp_path, name):
    meshes = scene(name)
    nodes, pairs = pb.bvh_build(meshes)
    world = po.OracleScene(meshes, None).world_triangles()
    rays = [edge_case_rays(20_000, 5), axis_rays(20_000, 6), slanted_rays(20_000, 7)]
    if name in ("boxes", "grid"):
        rays.append(box_edge_rays(meshes[1] if name == "boxes" else meshes[0], 4000, 2000, 9))
    if name in ("coincident", "ulps", "two of each"):
        r = random_rays(20_000, 8, -2, 2)
        t = world.reshape(-1, 3)[np.random.default_rng(1).integers(0, world.size // 3, len(r))]
        d = t * np.float32(0.9) - r["org"]
        r["dir"] = d / np.linalg.norm(d, axis=1)[:, None]
        rays.append(r)
    rays = np.concatenate(rays)
    paths = [str(tmp_path / f) for f in ("nodes.bin", "tris.bin", "rays.bin")]
    nodes.tofile(paths[0])
    leaf_ordered_faces(meshes, pairs, world).tofile(paths[1])
    np.ascontiguousarray(rays, pb.RAY_DTYPE).tofile(paths[2])
    p = subprocess.run([str(harness)] + paths, capture_output=True, text=True, timeout=600)
    assert p.returncode == 0, p.stderr
    said = p.stdout.split()
    assert int(said[1]) == len(rays)
    assert int(said[3]) > 0 and int(said[5]) > 0, p.stdout
    assert said[-2:] == ["differ", "0"], p.stdout
    if name == "ulps":
        assert int(said[7]) > 0, p.stdout  # MinT rose on some ray
