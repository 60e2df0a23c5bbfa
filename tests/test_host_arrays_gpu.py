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
