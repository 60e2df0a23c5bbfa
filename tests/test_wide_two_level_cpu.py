"""The walk over a two-level scene's four-wide records, compiled for the host (tests/cpp/wide_two_level_check.cu,
linked against the library), against traverse_two_level: the same face, instance, t, u, v and w on closest-hit
and any-hit rays, also from so far away that walks meet empty slots of top-level records."""
import os
import subprocess

import pytest

from test_traverse_host_cpu import NVCC, ROOT

pytestmark = pytest.mark.skipif(NVCC is None, reason="needs nvcc (host compilation only)")
LIB = os.path.join(ROOT, "polytope_b200", "lib")


@pytest.mark.parametrize("seed", [1, 2])
def test_two_level_walk_gives_the_binary_walks_hits(tmp_path, seed):
    exe = tmp_path / "wide_two_level_check"
    subprocess.run([NVCC, "-O2", "-std=c++17", "-Xcompiler", "-ffp-contract=off,-fno-fast-math",
                    "-I", os.path.join(ROOT, "polytope_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "wide_two_level_check.cu"), "-o", str(exe),
                    "-L", LIB, "-lpolytope_b200", "-Xlinker", "-rpath", "-Xlinker", LIB],
                   check=True, capture_output=True, text=True)
    p = subprocess.run([str(exe), "200000", str(seed)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    said = dict(zip(p.stdout.split()[::2], map(int, p.stdout.split()[1::2])))
    assert said["rays"] == 600_000 and said["hits"] > 300_000 and said["empty"] > 10_000, p.stdout
    assert said["differ"] == 0, p.stdout
