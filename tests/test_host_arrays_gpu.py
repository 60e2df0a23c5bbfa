"""Pageable ray and hit arrays on both sides of the line from which several host threads copy them, on the B200."""
import numpy as np
import pytest

import polytope_b200 as pb
from polytope_b200 import workloads as W
from test_traverse_host_cpu import edge_case_rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [98_303, 98_304, 98_305, 131_071])
def test_host_arrays_around_the_first_workers(cuda_device, n):
    s = pb.Scene(W.small_scene(3)[0])
    rays = np.resize(edge_case_rays(50_000, 12), n)
    assert s.intersect(rays).tobytes() == s.intersect(rays, counts=True)[0].tobytes()
    s.close()


@pytest.mark.parametrize("n", [1, 1 << 20, (1 << 20) + 1, (3 << 20) + 7, 4 << 20, (4 << 20) + 5, (6 << 20) + 3])
def test_pinned_arrays_around_the_chunks(cuda_device, n):
    """One chunk, several, and short chunks at both ends, with slots taken again: hits out of chunk c wait for the
    rays of chunk c + 1, and those of the last for none."""
    import torch
    s = pb.Scene(W.small_scene(3)[0])
    rays = torch.from_numpy(np.resize(edge_case_rays(50_021, 13), n).view(np.uint8)).pin_memory()
    hits = torch.zeros(16 * n, dtype=torch.uint8).pin_memory()
    on_device = torch.zeros(16 * n, dtype=torch.uint8, device="cuda")
    pb.check(pb.lib.pt_trace(s.handle, rays.cuda().data_ptr(), n, on_device.data_ptr(), pb.MEM_DEVICE, None))
    for _ in range(2):
        hits.zero_()
        pb.check(pb.lib.pt_trace(s.handle, rays.data_ptr(), n, hits.data_ptr(), 0, None))
        assert torch.equal(hits, on_device.cpu())
    s.close()
