"""The walk over four-wide records on the deepest tree that queries accept (62 levels), compiled for the host: every
record has four children that a ray hits, and the ray follows the chain first, so that the walk's stack
holds three entries for each of 31 levels of records and one more."""
import subprocess

import numpy as np
import pytest

import polytope_b200 as pb
from test_traverse_host_cpu import NVCC
from test_wide_host_cpu import harness  # noqa: F401  (fixture)

pytestmark = pytest.mark.skipif(NVCC is None, reason="needs nvcc (host compilation only)")
NODE = np.dtype([("bb", np.float32, 6), ("offset", np.uint32), ("num_faces", np.uint16), ("axis", np.uint16)])


def chain(depth):
    """Nodes of a tree of `depth` levels below the root: at each even level two leaves under the low child, a leaf
    and the next even level under the high one; all boxes alike."""
    out = []

    def leaf():
        out.append((0, 1))

    def inner(low, high):
        at = len(out)
        out.append(None)
        low()
        out[at] = (len(out) - at, 0)
        high()

    def level(d):
        inner(lambda: inner(leaf, leaf), lambda: inner(leaf, (lambda: level(d + 2)) if d + 2 < depth else leaf))

    level(0)
    nodes = np.zeros(len(out), NODE)
    nodes["bb"] = (-1, -1, -1, 1, 1, 1)
    for i, (offset, faces) in enumerate(out):
        nodes["offset"][i], nodes["num_faces"][i] = offset, faces
    leaves = np.nonzero(nodes["num_faces"])[0]
    nodes["offset"][leaves] = np.arange(len(leaves))
    return nodes


@pytest.mark.parametrize("depth", [60, 62])
def test_the_deepest_tree(harness, tmp_path, depth):  # noqa: F811
    nodes = chain(depth)
    n = int((nodes["num_faces"] > 0).sum())
    rng = np.random.default_rng(depth)
    tris = np.zeros((n, 12), np.float32)
    tris[:, :9] = (rng.uniform(-0.9, 0.9, (n, 1, 3)) + rng.uniform(-0.1, 0.1, (n, 3, 3))).reshape(n, 9)
    tris[:, 9] = np.arange(n, dtype=np.uint32).view(np.float32)
    rays = np.zeros(20_000, pb.RAY_DTYPE)
    rays["org"] = rng.uniform(-3, 3, (len(rays), 3))
    d = rng.uniform(-0.8, 0.8, (len(rays), 3)) - rays["org"]
    rays["dir"] = d / np.linalg.norm(d, axis=1)[:, None]
    rays["tmax"], rays["flags"] = np.inf, rng.integers(0, 2, len(rays))
    paths = [str(tmp_path / f) for f in ("nodes.bin", "tris.bin", "rays.bin")]
    for a, f in zip((nodes, tris, rays), paths):
        a.tofile(f)
    p = subprocess.run([str(harness)] + paths, capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    said = p.stdout.split()
    assert int(said[1]) == len(rays) and said[-2:] == ["differ", "0"], p.stdout
