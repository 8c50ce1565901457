"""The kd walk where its warp form can go wrong (GPU): batches at the edges of
a warp's share and of the queue, leaves of more items than a warp has lanes,
equal distances inside a leaf (the first item in the list wins), deferred
children beyond the shared part of the stack.  Bit-exact with the oracle's
kd walk."""
import numpy as np
import pytest

from encore_b200 import Accelerator, scenes
from encore_b200.accel import HIT_DTYPE
from oracle import bindings as ob

pytestmark = pytest.mark.gpu
SCALE = 1000.0


def rays_of(n, seed):
    cam = scenes.camera_rays_jittered(n - n // 2, seed=seed, eye=np.array([0.5, 0.5, -1.5]) * SCALE,
                                      look=np.array([0.5, 0.5, 0.5]) * SCALE)
    sph = scenes.random_sphere_rays(n // 2, seed=seed + 1, hi=(SCALE, SCALE, SCALE))
    r = np.concatenate([cam, sph])
    return np.ascontiguousarray(r[np.random.default_rng(seed + 2).permutation(n)])


def piled(n, copies, seed):
    """`copies` of every triangle, so leaves hold long runs of equal items."""
    t = scenes.random_triangles(n, seed=seed, scale=SCALE)
    return np.ascontiguousarray(np.repeat(t, copies, axis=0))


SCENES = {"soup": lambda: scenes.random_triangles(6000, seed=71, scale=SCALE),
          "piled": lambda: piled(60, 150, seed=72),
          "one63": lambda: piled(1, 63, seed=75), "one64": lambda: piled(1, 64, seed=75),
          "one65": lambda: piled(1, 65, seed=75),
          "field": lambda: scenes.heightfield(res=160, seed=73, scale=SCALE)}


@pytest.mark.parametrize("name,n", [("soup", 1), ("soup", 33), ("soup", 148 * 16 + 1),
                                    ("soup", 148 * 8 * 4 * 32 + 1), ("piled", 3000),
                                    ("one63", 900), ("one64", 900), ("one65", 900),
                                    ("field", 40000)])
@pytest.mark.parametrize("predicate", ["reference", "noclamp"])
def test_walk_equals_the_oracle(gpu, name, n, predicate):
    import torch
    tris = SCENES[name]()
    rays = rays_of(n, seed=74)
    acc = Accelerator("kdtree", predicate=predicate).build(tris)
    d = torch.from_numpy(rays).cuda()
    h = torch.full((n, 4), 7, dtype=torch.int32, device="cuda")
    hb = torch.full((n, 4), 7, dtype=torch.int32, device="cuda")
    scratch = torch.empty(acc.bin_scratch_bytes(n), dtype=torch.uint8, device="cuda")
    acc.intersect_device(d, n, h)
    acc.intersect_device_binned(d, n, hb, scratch)
    acc.check()
    assert torch.equal(h, hb)
    got = h.cpu().numpy().reshape(-1).view(HIT_DTYPE)
    want = ob.PortKd(tris).closest(rays, clamp=predicate == "reference")
    assert np.array_equal(got["tri"], want["tri"])
    m = want["tri"] >= 0
    for f in ("t", "u", "v"):
        assert np.array_equal(got[f][m].view(np.int32), want[f][m].view(np.int32)), f
    # the shadow form: the closest hit, if nearer than the ray's end
    end = rays.copy()
    end[:, 7] = np.float32(0.6 * SCALE)
    occ = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
    acc.occluded_device(torch.from_numpy(end).cuda(), n, occ)
    acc.check()
    assert np.array_equal(occ.cpu().numpy(), (m & (want["t"] < end[:, 7])).astype(np.uint8))
