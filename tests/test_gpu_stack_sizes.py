"""Stack depths that a caller may choose (GPU): every depth from 2 to 64 that the
tree does not exceed gives the hits of the default, at every width, for closest and
any hit.  The traversal's own shared memory counts toward the limit above which a
launch has to ask for more, so the depths just below it are the ones to miss."""
import numpy as np
import pytest

from encore_b200 import Accelerator, scenes
from encore_b200.accel import LaunchConfig

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [2, 4, 8])
@pytest.mark.parametrize("block", [0, 32, 96])
def test_every_stack_depth(gpu, width, block):
    import torch
    tris = scenes.random_triangles(200, seed=141, scale=1000.0)
    rays = scenes.random_sphere_rays(5000, seed=142, hi=(1000.0,) * 3)
    d = torch.from_numpy(rays).cuda()
    acc = Accelerator("wbvh", width=width).build(tris)
    want = torch.full((5000, 4), 7, dtype=torch.int32, device="cuda")
    occ = torch.full((5000,), 7, dtype=torch.uint8, device="cuda")
    acc.intersect_device(d, 5000, want)
    acc.occluded_device(d, 5000, occ)
    acc.check()
    scratch = torch.empty(acc.bin_scratch_bytes(5000), dtype=torch.uint8, device="cuda")
    for depth in range(16, 65):
        cfg = LaunchConfig(stack_depth=depth, block_threads=block, chunk=32)
        for binned in (False, True):
            h = torch.full((5000, 4), 7, dtype=torch.int32, device="cuda")
            if binned:
                acc.intersect_device_binned(d, 5000, h, scratch, launch=cfg)
            else:
                acc.intersect_device(d, 5000, h, launch=cfg)
            acc.check()
            assert torch.equal(h, want), (depth, binned)
        o = torch.full((5000,), 7, dtype=torch.uint8, device="cuda")
        acc.occluded_device(d, 5000, o, launch=cfg)
        acc.check()
        assert torch.equal(o, occ), depth
