"""Device memory that calls leave behind (GPU): a map holds its arrays and nothing of
what its build needed; a refit leaves nothing with its accelerator.  Beyond the
objects at most the bound of the library's pool stays allocated."""
import numpy as np
import pytest

from encore_b200 import Accelerator, scenes
from encore_b200.wavefront import photon_map_from_device

pytestmark = pytest.mark.gpu
MB = 1 << 20


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def trim():
    Accelerator("wbvh").build(scenes.random_triangles(64, seed=181, scale=1000.0)).destroy()


def test_maps_hold_their_arrays_only(gpu):
    import torch
    n, count = 1_000_000, 24
    d = [torch.rand(n, 3, device="cuda") for _ in range(3)]
    photon_map_from_device(*d, n)
    trim()
    before = free_bytes()
    maps = [photon_map_from_device(*d, n) for _ in range(count)]
    # 48 bytes a photon, 32,768 leaves with 32 bytes of box and range each; the pool
    # takes memory in pieces of 32 MB, of which one may be begun and one be left from
    # the build (a build's scratch with every map would be 144 MB)
    arrays = count * (48 * n + 33 * 32768)
    assert before - free_bytes() <= arrays + 2 * 32 * MB
    del maps


def test_refits_leave_nothing_with_the_accelerators(gpu):
    import torch
    tris = scenes.heightfield(res=300, seed=182, scale=1000.0)
    acc = Accelerator("wbvh").build(tris)
    image = acc.save()
    accs = [acc] + [Accelerator.load(image) for _ in range(31)]
    d = torch.from_numpy(scenes.random_sphere_rays(1000, seed=183, hi=(1000.0,) * 3)).cuda()
    h = torch.zeros(1000, 4, dtype=torch.int32, device="cuda")
    for a in accs:
        a.intersect_device(d, 1000, h)
    trim()
    before = free_bytes()
    for a in accs:
        a.update(tris)
    kept = before - free_bytes()
    assert kept <= 128 * MB + 4 * MB
    trim()
    assert before - free_bytes() <= 4 * MB
    assert len(accs) * 84 * len(tris) > 256 * MB  # (what keeping it with each would take)
