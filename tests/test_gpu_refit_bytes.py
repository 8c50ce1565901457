"""The refit's node and triangle bytes (GPU) against a plain restatement of the
rule: padded triangle boxes, children's boxes joined bottom-up, each node's
grid the finest power of two whose 255 steps cover it and that is no finer
than the floats' spacing there, child planes rounded outward.  Byte for byte
through the saved image."""
import struct

import numpy as np
import pytest

from encore_b200 import Accelerator, EncoreError, scenes

pytestmark = pytest.mark.gpu
F = np.float32
HEADER = "<8sI3i4I12f4Q"
NODE = {2: 48, 4: 64, 8: 80}


def parts(image, width):
    h = struct.unpack_from(HEADER, image)
    ntris, nnodes = h[5], h[6]
    o = struct.calcsize(HEADER)
    nodes = np.frombuffer(image, np.uint8, nnodes * NODE[width], o).reshape(nnodes, -1)
    o += nodes.size
    tris = np.frombuffer(image, np.float32, ntris * 12, o).reshape(ntris, 12)
    order = np.frombuffer(image, np.uint32, ntris, o + 48 * ntris)
    return h, nodes, tris, order


def exponent(ext, mag):
    spacing = float(np.nextafter(F(mag), F(np.inf))) - float(mag)
    e = -126
    while 255.0 * 2.0 ** e < ext or 2.0 ** e < spacing:
        e += 1
    return e


def restated(image, width, verts):
    """The image's nodes and triangle records for the moved vertices."""
    h, old, _, order = parts(image, width)
    nodes = old.copy()
    v = verts.reshape(-1, 3, 3)
    lo, hi = v.min((0, 1)), v.max((0, 1))
    pad = F(1e-5) * max((hi - lo).max(), np.abs(v).max())
    pad = pad if pad > 0 else F(1e-30)
    tlo, thi = (v.min(1) - pad)[order], (v.max(1) + pad)[order]
    box = np.zeros((len(nodes), 2, 3), F)
    for i in range(len(nodes) - 1, -1, -1):
        child_base, tri_base = struct.unpack_from("<2I", old[i].tobytes(), 16)
        slots = {}
        for c in range(width):
            m = int(old[i, 24 + c])
            if 0 < m < 32:
                slots[c] = box[child_base + m - 1]
            elif m:
                s = slice(tri_base + (m & 31), tri_base + (m & 31) + (m >> 5))
                slots[c] = np.stack([tlo[s].min(0), thi[s].max(0)])
        b = np.stack(list(slots.values()))
        box[i] = np.stack([b[:, 0].min(0), b[:, 1].max(0)])
        nodes[i, 0:12] = np.frombuffer(box[i, 0].tobytes(), np.uint8)
        for a in range(3):
            p = float(box[i, 0, a])
            e = exponent(float(box[i, 1, a]) - p, np.abs(box[i, :, a]).max())
            nodes[i, 12 + a] = e + 127
            for c in range(width):
                q = (255, 0)
                if c in slots:
                    q = (np.floor((float(slots[c][0, a]) - p) / 2.0 ** e),
                         np.ceil((float(slots[c][1, a]) - p) / 2.0 ** e))
                nodes[i, 24 + width + a * width + c] = int(q[0])
                nodes[i, 24 + width + (3 + a) * width + c] = int(q[1])
    t = v[order]
    tris = np.zeros((len(order), 12), F)
    tris[:, 0:3], tris[:, 3:6], tris[:, 6:9] = t[:, 0], t[:, 1] - t[:, 0], t[:, 2] - t[:, 0]
    tris[:, 9] = order.astype(np.int32).view(F)
    return nodes, tris, lo, hi


def moves(name, tris):
    r = np.random.default_rng(81)
    if name == "drift":
        return tris + np.tile(r.normal(0, 20, (len(tris), 3)).astype(F), (1, 3))
    if name == "scrambled":
        return tris[r.permutation(len(tris))]
    if name == "flat":  # no extent along one axis, zeros of both signs
        t = tris.reshape(-1, 3, 3).copy()
        t[..., 1] = np.where(r.random(t.shape[:2]) < 0.5, F(0.0), F(-0.0))
        return t.reshape(-1, 9)
    if name == "point":
        return np.full_like(tris, F(3.5))
    return {"tiny": tris * F(1e-38), "huge": tris * F(1e33),
            "far": tris * F(1e-3) + F(5e6)}[name]


@pytest.mark.parametrize("width", [2, 4, 8])
@pytest.mark.parametrize("n,move", [(1, "drift"), (2, "scrambled"), (7, "drift"), (40, "flat"),
                                    (300, "point"), (300, "tiny"), (300, "huge"), (2000, "far"),
                                    (2000, "flat"), (9000, "scrambled"), (9000, "drift")])
def test_refit_bytes(gpu, width, n, move):
    tris = scenes.random_triangles(n, seed=80, scale=1000.0)
    acc = Accelerator("wbvh", width=width).build(tris)
    before = acc.save()
    moved = np.ascontiguousarray(moves(move, tris), dtype=F)
    acc.update(moved)
    h, nodes, got_tris, _ = parts(acc.save(), width)
    want_nodes, want_tris, lo, hi = restated(before, width, moved)
    assert np.array_equal(nodes, want_nodes)
    assert np.array_equal(got_tris.view(np.int32), want_tris.view(np.int32))
    assert np.array_equal(np.float32(h[9:12]), lo) and np.array_equal(np.float32(h[12:15]), hi)
    acc.destroy()


def test_infinite_vertices_are_refused_and_change_nothing(gpu):
    tris = scenes.random_triangles(500, seed=82, scale=1000.0)
    acc = Accelerator("wbvh").build(tris)
    before = acc.save()
    bad = tris.copy()
    bad[3, 4] = np.inf
    with pytest.raises(EncoreError) as ei:
        acc.update(bad)
    assert ei.value.status == 1
    assert acc.save() == before
    acc.update(tris + F(1.0))
    acc.update(tris)
    rays = scenes.random_sphere_rays(500, seed=83, hi=(1000.0, 1000.0, 1000.0))
    assert np.array_equal(acc.intersect(rays), Accelerator("wbvh").build(tris).intersect(rays))
