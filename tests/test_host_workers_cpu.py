"""The host threads of pt_trace's pageable arrays (polytope_b200/csrc/host_workers.h): all work is done with
however many threads the system gives, also when it has no memory for one, and one processor gets none."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

pytestmark = pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")


@pytest.mark.parametrize("case", ["threads", "counts"])
def test_host_workers(tmp_path, case):
    exe = tmp_path / "host_workers_check"
    subprocess.run(["g++", "-O1", "-std=c++17", "-Wall", "-pthread", "-I", os.path.join(ROOT, "polytope_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "host_workers_check.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    p = subprocess.run([str(exe), case], capture_output=True, text=True, timeout=60)
    assert p.returncode == 0 and p.stdout.strip() == "ok", p.stdout + p.stderr
