"""Which kernels a call launches (GPU).  Tests that compare a form with another pass
as well if the form is never chosen; these say, by the kernels' names in a profile,
that it is, at the sizes and on the scenes those tests use."""
import numpy as np
import pytest

from encore_b200 import Accelerator, PhotonMap, scenes
from encore_b200.batch import BatchLaunch

pytestmark = pytest.mark.gpu
SCALE = 1000.0


def launched(call):
    import torch
    from torch.profiler import ProfilerActivity, profile
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return [e.name for e in p.events() if "anonymous namespace" in e.name]


def trace(any_hit=False, multi=False, ordered=False, wait=False):
    """wbvh_trace<W, CLAMP, ANY, COUNT, MULTI, LANE, ORD, WAIT>"""
    a = ["8", "true", any_hit, False, multi, False, ordered, wait]
    return "wbvh_trace<" + ", ".join(str(x).lower() for x in a) + ">"


def has(names, what):
    return any(what in n for n in names)


def test_forms_of_the_traversal(gpu):
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    long = sms * 9 * 128 * 6
    acc = Accelerator("wbvh").build(scenes.random_triangles(6000, seed=111, scale=SCALE))
    rays = torch.from_numpy(scenes.random_sphere_rays(long, seed=113, hi=(SCALE,) * 3)).cuda()
    hits = torch.zeros(long, 4, dtype=torch.int32, device="cuda")
    occ = torch.zeros(long, dtype=torch.uint8, device="cuda")
    scratch = torch.empty(acc.bin_scratch_bytes(long), dtype=torch.uint8, device="cuda")
    for n, wait in ((long, True), (long - 1, False)):
        assert has(launched(lambda: acc.intersect_device(rays, n, hits)), trace(wait=wait))
        assert has(launched(lambda: acc.intersect_device_binned(rays, n, hits, scratch)),
                   trace(ordered=True, wait=wait))
        assert has(launched(lambda: acc.occluded_device(rays, n, occ)), trace(any_hit=True, wait=wait))
    batch = BatchLaunch([(acc, rays, hits)])
    assert has(launched(batch.launch), trace(multi=True, wait=True))
    few = 192 * sms
    assert has(launched(lambda: acc.intersect_device(rays, few, hits)), "wbvh_few<true, false>")
    assert has(launched(lambda: acc.occluded_device(rays, few, occ)), "wbvh_few<true, true>")
    assert has(launched(lambda: acc.intersect_device(rays, few + 1, hits)), trace())
    # a tree whose visits test more: no waiting
    dense = Accelerator("wbvh").build(scenes.random_triangles(200_000, seed=115, scale=SCALE))
    assert has(launched(lambda: dense.intersect_device(rays, long, hits)), trace())


@pytest.mark.parametrize("width", [2, 4, 8])
def test_refits_run_on_the_device(gpu, width):
    for n in (1, 300, 9000):
        tris = scenes.random_triangles(n, seed=80, scale=SCALE)
        acc = Accelerator("wbvh", width=width).build(tris)
        assert has(launched(lambda: acc.update(tris + np.float32(1.0))), f"refit_levels<{width}>")
    acc = Accelerator.load(acc.save())
    assert has(launched(lambda: acc.update(tris)), f"refit_levels<{width}>")


@pytest.mark.parametrize("n,kernels", [(1024, []), (1025, ["split_block", "split_ranges"]),
                                       (22528, ["split_block", "split_ranges"]),
                                       (22529, ["split_cluster", "split_block", "split_ranges"])])
def test_forms_of_the_map_build(gpu, n, kernels):
    r = np.random.default_rng(191)
    pm = PhotonMap(n)
    pm.add_photons(*(r.random((n, 3)).astype(np.float32) for _ in range(3)))
    names = launched(pm.balance_and_construct)
    for k in ("split_cluster", "split_block", "split_ranges"):
        assert has(names, k) == (k in kernels)
