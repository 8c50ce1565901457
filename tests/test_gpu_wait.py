"""Launches long enough for lanes to wait at their leaves (GPU): the hits equal
those of a launch below that size, bit for bit, for plain, binned and
multi-scene launches, at the size where the form changes and beyond it."""
import numpy as np
import pytest

from encore_b200 import Accelerator, scenes
from encore_b200.batch import BatchLaunch

pytestmark = pytest.mark.gpu
SCALE = 1000.0


@pytest.mark.parametrize("predicate", ["reference", "noclamp"])
@pytest.mark.parametrize("extra", [0, 1, 200_001])
def test_long_launches_match_short_ones(gpu, predicate, extra):
    import torch
    tris = scenes.random_triangles(6000, seed=111, scale=SCALE)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = sms * 9 * 128 * 6 + extra
    base = np.concatenate([
        scenes.camera_rays_jittered(150_000, seed=112, eye=np.array([0.5, 0.5, -1.5]) * SCALE,
                                    look=np.array([0.5, 0.5, 0.5]) * SCALE),
        scenes.random_sphere_rays(150_007, seed=113, hi=(SCALE, SCALE, SCALE))])
    d = torch.from_numpy(base).cuda()
    m = len(base)
    acc = Accelerator("wbvh", predicate=predicate).build(tris)
    short = torch.full((m, 4), 7, dtype=torch.int32, device="cuda")
    acc.intersect_device(d, m, short)
    pick = torch.randint(0, m, (n,), device="cuda", generator=torch.Generator("cuda").manual_seed(5))
    rays = d[pick].contiguous()
    want = short[pick]
    hits = torch.full((n, 4), 7, dtype=torch.int32, device="cuda")
    acc.intersect_device(rays, n, hits)
    assert torch.equal(hits, want)
    hits.fill_(7)
    scratch = torch.empty(acc.bin_scratch_bytes(n), dtype=torch.uint8, device="cuda")
    acc.intersect_device_binned(rays, n, hits, scratch)
    assert torch.equal(hits, want)
    acc.check()
    # three scenes, the first two the same triangles
    other = Accelerator("wbvh", predicate=predicate).build(scenes.heightfield(res=64, seed=114, scale=SCALE))
    alone = torch.full((m, 4), 7, dtype=torch.int32, device="cuda")
    other.intersect_device(d, m, alone)
    h = [torch.full((k, 4), 7, dtype=torch.int32, device="cuda") for k in (n // 2, n - n // 2, m)]
    # (most rays lie in a scene whose launches are of this form)
    b = BatchLaunch([(acc, rays[:n // 2], h[0]), (acc, rays[n // 2:].contiguous(), h[1]), (other, d, h[2])])
    b.launch()
    b.check()
    assert torch.equal(torch.cat(h[:2]), want) and torch.equal(h[2], alone)


def test_stack_limit_is_reported_by_long_launches(gpu):
    import torch

    from encore_b200 import EncoreError
    from encore_b200.accel import LaunchConfig
    tris = scenes.random_triangles(3000, seed=115, scale=SCALE)
    acc = Accelerator("wbvh").build(tris)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = sms * 9 * 128 * 6 + 5
    rays = torch.from_numpy(scenes.random_sphere_rays(n, seed=116, hi=(SCALE, SCALE, SCALE))).cuda()
    hits = torch.full((n, 4), 7, dtype=torch.int32, device="cuda")
    acc.intersect_device(rays, n, hits, launch=LaunchConfig(stack_depth=2))
    with pytest.raises(EncoreError) as ei:
        acc.check()
    assert ei.value.status == 4
    assert (hits[:, 0] >= -1).all() and (hits[:, 0] < 3000).all()


@pytest.mark.parametrize("scene", ["soup", "field"])
@pytest.mark.parametrize("extra", [-1, 0, 70_001])
def test_long_any_hit_launches_match_short_ones(gpu, scene, extra):
    """Any hit takes the same form at the same size; the short launches'
    answers are those of a form without waiting."""
    import torch
    tris = (scenes.random_triangles(3000, seed=117, scale=SCALE) if scene == "soup"
            else scenes.heightfield(res=96, seed=118, scale=SCALE))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = sms * 9 * 128 * 6 + extra
    base = scenes.random_sphere_rays(200_003, seed=119, hi=(SCALE, SCALE, SCALE))
    base[::3, 7] = 0.2 * SCALE  # bounded segments between unbounded rays
    d = torch.from_numpy(base).cuda()
    m = len(base)
    acc = Accelerator("wbvh").build(tris)
    short = torch.full((m,), 7, dtype=torch.uint8, device="cuda")
    acc.occluded_device(d, m, short)
    assert 0.02 * m < int((short == 1).sum()) < 0.98 * m
    pick = torch.randint(0, m, (n,), device="cuda", generator=torch.Generator("cuda").manual_seed(6))
    occ = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
    acc.occluded_device(d[pick].contiguous(), n, occ)
    acc.check()
    assert torch.equal(occ, short[pick])
