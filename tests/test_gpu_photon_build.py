"""The device build of a photon map (GPU): the saved image's tree against the
rule it follows.  Every range splits at its median index on the axis of its
largest extent, leaves are those ranges, boxes are exact bounds, every photon
is in the map once with its own normal and power; photons taken from host and
from device memory give the same bytes.  Sizes sit at the host build's limit,
at the tiles of the counting passes and at changes of the tree's depth."""
import struct

import numpy as np
import pytest

from encore_b200 import PhotonMap
from encore_b200.wavefront import photon_map_from_device
from oracle import bindings as ob

pytestmark = pytest.mark.gpu
HEADER = "<8sIiIIii24I2Q"


def photons(kind, n):
    r = np.random.default_rng(91)
    p = r.random((n, 3)).astype(np.float32) * np.float32([3.0, 1.0, 2.0])
    if kind == "plane":
        p[:, 1] = np.where(r.random(n) < 0.5, np.float32(0.0), np.float32(-0.0))
    elif kind == "point":
        p[:] = np.float32([1.0, -2.0, 3.0])
    elif kind == "cluster":
        p = (p * np.exp(-12.0 * r.random((n, 1))) - 0.5).astype(np.float32)
    elif kind == "grid":
        p = np.round(p * 6.0).astype(np.float32) - 5.0
    nrm = np.eye(3, dtype=np.float32)[r.integers(0, 3, n)]
    return p, nrm, r.random((n, 3)).astype(np.float32)


def image(pm):
    buf = pm.save()
    h = struct.unpack_from(HEADER, buf)
    n, nlev, box_floats, leaf_words = h[3], h[6], h[31], h[32]
    o = struct.calcsize(HEADER)
    box = np.frombuffer(buf, np.float32, box_floats, o)
    leaf = np.frombuffer(buf, np.uint32, leaf_words, o + 4 * box_floats).reshape(-1, 2)
    rec = np.frombuffer(buf, np.float32, 12 * n, o + 4 * box_floats + 4 * leaf_words)
    levels = [(h[7 + i], h[15 + i], h[23 + i]) for i in range(nlev)]
    return buf, h[5], levels, box, leaf, rec.reshape(3, n, 4)


@pytest.mark.parametrize("kind,n", [("box", 1025), ("box", 2048), ("grid", 2049), ("box", 4096),
                                    ("plane", 4097), ("point", 5000), ("cluster", 32 * 1024),
                                    ("grid", 32 * 1024 + 1), ("box", 65537), ("plane", 100003),
                                    ("cluster", 300001)])
def test_tree_follows_the_rule(gpu, kind, n):
    import torch
    pos, nrm, pw = photons(kind, n)
    host = PhotonMap(n)
    host.add_photons(pos, nrm, pw)
    host.balance_and_construct()
    dev = photon_map_from_device(*(torch.from_numpy(x).cuda() for x in (pos, nrm, pw)), n)
    buf, depth, levels, box, leaf, rec = image(dev)
    assert buf == image(host)[0]
    assert (n - 1) // 32 < (1 << depth) and (depth == 0 or n > 32 << (depth - 1))
    ids = rec[0, :, 3].view(np.int32)
    assert np.array_equal(np.sort(ids), np.arange(n))
    for got, want in zip(rec, (pos, nrm, pw)):
        assert np.array_equal(got[:, :3].view(np.int32), want[ids].view(np.int32))
    # ranges, and the split of each on its widest axis
    ranges = [(0, n)]
    p = rec[0, :, :3]
    for level in range(depth):
        nxt = []
        for b, e in ranges:
            m = b + (e - b) // 2
            ext = p[b:e].max(0) - p[b:e].min(0)
            axis = 0
            for a in (1, 2):
                if ext[a] > ext[axis]:
                    axis = a
            assert p[b:m, axis].max() <= p[m:e, axis].min()
            nxt += [(b, m), (m, e)]
        ranges = nxt
    assert np.array_equal(leaf, np.array(ranges, np.uint32))
    # boxes, level by level
    lo = np.stack([p[b:e].min(0) for b, e in ranges])
    hi = np.stack([p[b:e].max(0) for b, e in ranges])
    for i, (count, off, pad) in enumerate(levels):
        if i:
            cut = np.arange(0, len(lo), 32)
            lo, hi = np.minimum.reduceat(lo, cut), np.maximum.reduceat(hi, cut)
        assert count == len(lo) and pad == (count + 31) // 32 * 32
        b = box[off:off + 6 * pad].reshape(6, pad)
        assert np.array_equal(b[:3, :count].T, lo) and np.array_equal(b[3:, :count].T, hi)
        assert (b[:3, count:] == np.inf).all() and (b[3:, count:] == -np.inf).all()
    assert levels[-1][0] <= 32


@pytest.mark.parametrize("n", [1024, 1025, 20011])
def test_nearest_and_radiance_match_the_oracle(gpu, n):
    pos, nrm, pw = photons("box", n)
    r = np.random.default_rng(92)
    q = r.random((300, 3)).astype(np.float32) * np.float32([3.0, 1.0, 2.0])
    qn = np.eye(3, dtype=np.float32)[r.integers(0, 3, 300)]
    pm = PhotonMap(n)
    pm.add_photons(pos, nrm, pw)
    for k, r_max in ((50, 0.5), (8, 10.0)):
        want, _ = ob.port_gather(pos, nrm, pw, q, qn, k, r_max)
        assert np.allclose(pm.get_radiance_estimate(k, r_max, q, qn), want, rtol=1e-4, atol=1e-12)
        idx, d2, cnt = pm.get_nearest_n_photons(k, r_max, q, qn)
        for i in range(0, 300, 7):
            d = ((q[i] - pos) ** 2).astype(np.float32)
            d = (d[:, 0] + d[:, 1]) + d[:, 2]
            ok = np.nonzero((nrm == qn[i]).all(1) & (d < np.float32(r_max) ** 2))[0]
            near = ok[np.lexsort((ok, d[ok]))][:k]
            assert cnt[i] == len(near) and np.array_equal(idx[i, :cnt[i]], near)
            assert np.array_equal(d2[i, :cnt[i]], d[near])


def test_memory_kept_for_maps_is_bounded_and_given_back(gpu):
    """Freed maps leave at most the pool's bound behind, and nothing once an
    accelerator on the device has been destroyed."""
    import torch

    from encore_b200 import Accelerator, scenes
    small = scenes.random_triangles(64, seed=93, scale=1000.0)

    def free_bytes():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    n = 3_000_000
    d = [torch.rand(n, 3, device="cuda") for _ in range(3)]
    for _ in range(2):  # the first pass also loads the kernels
        Accelerator("wbvh").build(small).destroy()
        before = free_bytes()
        maps = [photon_map_from_device(*d, n) for _ in range(2)]
        assert before - free_bytes() >= 2 * 48 * n
        del maps
        assert before - free_bytes() <= (128 << 20) + (64 << 20)
        Accelerator("wbvh").build(small).destroy()
        left = before - free_bytes()
    assert left <= 4 << 20


def test_maps_made_and_freed_by_several_threads(gpu):
    """Threads that make, use and free maps at once, each on a stream of its
    own, get the answers one thread gets alone."""
    import threading

    import torch
    r = np.random.default_rng(94)
    sizes = [1500, 20000, 70001, 150000]
    sets = [photons("box", n) for n in sizes]
    q = (r.random((4000, 3)) * [3.0, 1.0, 2.0]).astype(np.float32)
    qn = np.eye(3, dtype=np.float32)[r.integers(0, 3, 4000)]
    dq, dn = torch.from_numpy(q).cuda(), torch.from_numpy(qn).cuda()

    def gather(i, stream):
        d = [torch.from_numpy(x).cuda() for x in sets[i]]
        torch.cuda.synchronize()
        out = torch.zeros(4000, 3, device="cuda")
        torch.cuda.synchronize()
        pm = photon_map_from_device(*d, sizes[i])
        pm.get_radiance_estimate_device(20, 0.3, dq, dn, 4000, out, stream=stream.cuda_stream)
        del pm  # waits for the gather
        return out.cpu().numpy()

    want = [gather(i, torch.cuda.Stream()) for i in range(4)]
    got, errors = {}, []

    def work(i):
        try:
            s = torch.cuda.Stream()
            got[i] = [gather(i, s) for _ in range(6)]
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)

    ts = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not errors, errors
    for i in range(4):
        for g in got[i]:
            assert np.array_equal(g.view(np.int32), want[i].view(np.int32))
