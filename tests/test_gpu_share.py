"""Batches that fit the grid at once (GPU): eight lanes walk one ray, or each
warp takes a fixed share of the rays, instead of reading the queue.  The sizes
sit at the edges: one ray, a warp's worth, one ray per warp and one more, the
most that eight lanes per ray take and one more, a full chunk per warp and one
more, and the first size that takes the queue.  Every hit
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
@pytest.mark.parametrize("per_warp", ["1", "31", "33", "warps", "warps+1", "few", "few+1", "full",
                                      "full+1", "queue"])
def test_shared_out_batches_match_the_queue(gpu, scene, width, per_warp):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    warps = sms * 16
    n = {"1": 1, "31": 31, "33": 33, "warps": warps, "warps+1": warps + 1, "few": 192 * sms,
         "few+1": 192 * sms + 1, "full": 32 * warps,
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


@pytest.mark.parametrize("kind", ["soup", "piled", "field", "one"])
@pytest.mark.parametrize("predicate", ["reference", "noclamp"])
def test_eight_lanes_per_ray_match_the_queue(gpu, kind, predicate):
    """Leaves of up to four triangles (more than eight in one step), equal
    distances, rays from inside, with bounds and with zero direction components."""
    import torch
    if kind == "soup":
        tris = scenes.random_triangles(4000, seed=65, scale=SCALE)
    elif kind == "piled":
        tris = np.repeat(scenes.random_triangles(40, seed=66, scale=SCALE), 60, axis=0)
    elif kind == "field":
        tris = scenes.heightfield(res=96, seed=67, scale=SCALE)
    else:
        tris = scenes.random_triangles(1, seed=68, scale=SCALE)
    rays = batch(5001)
    rays[::7, 3] = np.float32(0.2 * SCALE)
    rays[::5, 7] = np.float32(0.5 * SCALE)
    rays[::11, 4] = 0.0
    rays[::13, 5] = -0.0
    d = torch.from_numpy(rays).cuda()
    for leaf in (1, 4):
        acc = Accelerator("wbvh", max_leaf_tris=leaf, predicate=predicate).build(tris)
        hits = [torch.full((len(rays), 4), 7, dtype=torch.int32, device="cuda") for _ in range(2)]
        occ = [torch.full((len(rays),), 7, dtype=torch.uint8, device="cuda") for _ in range(2)]
        for i, lc in enumerate((None, LaunchConfig(chunk=32))):
            acc.intersect_device(d, len(rays), hits[i], launch=lc)
            acc.occluded_device(d, len(rays), occ[i], launch=lc)
        acc.check()
        assert torch.equal(hits[0], hits[1]) and torch.equal(occ[0], occ[1])
        assert kind == "one" or (hits[0][:, 0] >= 0).any()


def test_stack_limit_is_reported_by_eight_lanes_per_ray(gpu, scene):
    import torch

    from encore_b200 import EncoreError
    acc = Accelerator("wbvh").build(scene)
    rays = torch.from_numpy(batch(3000)).cuda()
    hits = torch.full((3000, 4), 7, dtype=torch.int32, device="cuda")
    acc.intersect_device(rays, 3000, hits, launch=LaunchConfig(stack_depth=2))
    with pytest.raises(EncoreError) as ei:
        acc.check()
    assert ei.value.status == 4
    assert (hits[:, 0] < len(scene)).all() and (hits[:, 0] >= -1).all()
    acc.intersect_device(rays, 3000, hits)
    acc.check()
