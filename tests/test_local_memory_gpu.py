"""Device memory that the first calls of a fresh process take beside their buffers: no kernel's frame is above the
1024 bytes a thread that a context starts with, so no first launch makes its local memory grow, also not that
of pt_render_noalloc, whose callers have no memory to give."""
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

PROGRAM = """
import ctypes as C, sys
import torch
sys.path.insert(0, {root!r})
import polytope_b200 as pb
from polytope_b200 import workloads as W

def free():
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]

meshes, env = W.small_scene(level=3)
flat, two = pb.Scene(meshes, env), pb.Scene(meshes, env, two_level=True)
out = torch.zeros(64 * 48 * 3, device="cuda")
rays, hits = torch.zeros(3200, dtype=torch.uint8, device="cuda"), torch.zeros(1600, dtype=torch.uint8, device="cuda")

def noalloc(s):
    d = pb.render_desc(64, 48, 1, 4, W.SMALL_CAMERA, 1, pb.RENDER_NEE)
    pb.check(pb.lib.pt_render_noalloc(s.handle, C.byref(d), out.data_ptr(), None, None))

def query(s):
    pb.check(pb.lib.pt_trace(s.handle, rays.data_ptr(), 100, hits.data_ptr(), pb.MEM_DEVICE, None))

last = free()
for name, call in (("noalloc", lambda: noalloc(flat)), ("noalloc two-level", lambda: noalloc(two)),
                   ("query", lambda: query(flat)), ("query two-level", lambda: query(two))):
    call()
    now = free()
    print(name, (last - now) >> 20, sep=": ")
    last = now
"""


def test_first_calls_take_no_local_memory(cuda_device):
    p = subprocess.run([sys.executable, "-c", PROGRAM.format(root=ROOT)], capture_output=True, text=True, timeout=300)
    assert p.returncode == 0, p.stderr
    taken = {line.split(": ")[0]: int(line.split(": ")[1]) for line in p.stdout.splitlines()}
    # MiB: the 6 MiB array of pt_render_noalloc and the module's code arrive with the first call
    assert taken["noalloc"] <= 12, taken
    assert all(taken[k] <= 4 for k in ("noalloc two-level", "query", "query two-level")), taken
