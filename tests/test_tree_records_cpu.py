"""Which trees get four-wide records (validate_tree's numbering), on the host: tests/cpp/tree_records_check.cpp
linked against the library, and tests/cpp/wide_refs_check.cu for the records' references.  No device is
used and no tree is uploaded."""
import os
import shutil
import subprocess

import pytest

from test_traverse_host_cpu import NVCC

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIB = os.path.join(ROOT, "polytope_b200", "lib")

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    exe = tmp_path_factory.mktemp("records") / "tree_records_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-I", os.path.join(ROOT, "polytope_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "tree_records_check.cpp"), "-o", str(exe),
                    "-L", LIB, "-lpolytope_b200", "-Wl,-rpath," + LIB], check=True, capture_output=True, text=True)
    return exe


@pytest.mark.parametrize("case", ["numbered", "unreached", "shared_faces"])
def test_which_trees_are_numbered(harness, case):
    p = subprocess.run([str(harness), case], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0 and p.stdout.strip() == "ok", p.stdout + p.stderr


@pytest.mark.skipif(NVCC is None, reason="needs nvcc (host compilation only)")
def test_references_at_the_ends_of_their_range(tmp_path):
    """No slot's reference, the last node of the largest tree with records included, is one of the walk's marks."""
    exe = tmp_path / "wide_refs_check"
    subprocess.run([NVCC, "-O1", "-std=c++17", "-I", os.path.join(ROOT, "polytope_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "wide_refs_check.cu"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    p = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0 and p.stdout.strip() == "ok", p.stdout + p.stderr
