"""Rays of the kd walk that stand at a long leaf as soon as a lane has taken them
(GPU): the whole tree is one leaf, so the lanes that test it read a ray stored in
the same step of the warp.  Bit-exact with the oracle's kd walk."""
import numpy as np
import pytest

from encore_b200 import Accelerator, scenes
from encore_b200.accel import HIT_DTYPE
from oracle import bindings as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("items", [63, 64, 200])
@pytest.mark.parametrize("n", [33, 4096, 300_007])
def test_fresh_rays_at_a_long_leaf(gpu, items, n):
    import torch
    one = scenes.random_triangles(1, seed=131, scale=1000.0)
    tris = np.ascontiguousarray(np.repeat(one, items, axis=0))
    r = np.random.default_rng(132)
    v = one.reshape(3, 3).astype(np.float64)
    w = r.dirichlet([1, 1, 1], n)
    at = w @ v + np.where(r.random((n, 1)) < 0.3, 400.0, 0.0)  # about a third misses
    o = at + r.normal(size=(n, 3)) * 300.0
    d = at - o
    rays = np.zeros((n, 8), np.float32)
    rays[:, :3], rays[:, 4:7], rays[:, 7] = o, d / np.linalg.norm(d, axis=1, keepdims=True), np.inf
    acc = Accelerator("kdtree").build(tris)
    h = torch.full((n, 4), 7, dtype=torch.int32, device="cuda")
    acc.intersect_device(torch.from_numpy(rays).cuda(), n, h)
    acc.check()
    got = h.cpu().numpy().reshape(-1).view(HIT_DTYPE)
    want = ob.PortKd(tris).closest(rays, clamp=True)
    m = want["tri"] >= 0
    assert np.array_equal(got["tri"], want["tri"]) and 0.3 * n < m.sum() < n
    for f in ("t", "u", "v"):
        assert np.array_equal(got[f][m].view(np.int32), want[f][m].view(np.int32)), f
