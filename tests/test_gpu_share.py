"""Batches that fit the grid at once (GPU): each warp takes a fixed share of
the rays instead of reading the queue.  The sizes sit at the edges of the
share: one ray, a warp's worth, one ray per warp and one more, a full chunk
per warp and one more, and the first size that takes the queue.  Every hit
equals the queue form's (a launch with its chunk chosen) bit for bit, and the
small batches the oracle's brute force."""
import numpy as np
import pytest

from encore_b200 import Accelerator, scenes
from encore_b200.accel import LaunchConfig
from oracle import bindings as ob

pytestmark = pytest.mark.gpu
SCALE = 1000.0


@pytest.fixture(scope="module")
def scene():
    return scenes.random_triangles(3000, seed=61, scale=SCALE)


def batch(n):
    cam = scenes.camera_rays_jittered(n - n // 2, seed=62, eye=np.array([0.5, 0.5, -1.5]) * SCALE,
                                      look=np.array([0.5, 0.5, 0.5]) * SCALE)
    sph = scenes.random_sphere_rays(n // 2, seed=63, hi=(SCALE, SCALE, SCALE))
    r = np.concatenate([cam, sph])
    return np.ascontiguousarray(r[np.random.default_rng(64).permutation(n)])


@pytest.mark.parametrize("width", [2, 8])
@pytest.mark.parametrize("per_warp", ["1", "31", "33", "warps", "warps+1", "full", "full+1", "queue"])
def test_shared_out_batches_match_the_queue(gpu, scene, width, per_warp):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    warps = sms * 16
    n = {"1": 1, "31": 31, "33": 33, "warps": warps, "warps+1": warps + 1, "full": 32 * warps,
         "full+1": 32 * warps + 1, "queue": 32 * 4 * 9 * sms + 1}[per_warp]
    rays = batch(n)
    acc = Accelerator("wbvh", width=width).build(scene)
    d = torch.from_numpy(rays).cuda()
    hits = [torch.full((n, 4), 7, dtype=torch.int32, device="cuda") for _ in range(3)]
    occ = [torch.full((n,), 7, dtype=torch.uint8, device="cuda") for _ in range(2)]
    scratch = torch.empty(acc.bin_scratch_bytes(n), dtype=torch.uint8, device="cuda")
    acc.intersect_device(d, n, hits[0])
    acc.intersect_device(d, n, hits[1], launch=LaunchConfig(chunk=32))
    acc.intersect_device_binned(d, n, hits[2], scratch)
    acc.occluded_device(d, n, occ[0])
    acc.occluded_device(d, n, occ[1], launch=LaunchConfig(chunk=32))
    acc.check()
    assert torch.equal(hits[0], hits[1]) and torch.equal(hits[0], hits[2])
    assert torch.equal(occ[0], occ[1])
    if n <= warps + 1:
        want = ob.port_brute(scene, rays, clamp=True)
        got = hits[0].cpu().numpy()
        mism = [c for c in ob.classify(scene, rays, {"tri": got[:, 0], "t": got[:, 1].view(np.float32),
                                                     "u": got[:, 2].view(np.float32),
                                                     "v": got[:, 3].view(np.float32)}, want)[1]]
        assert "unexplained" not in mism, mism
