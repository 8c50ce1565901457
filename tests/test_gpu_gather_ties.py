"""Which of several photons at the k-th distance a gather keeps (GPU): the photons
come in the order of the walk over the saved tree; until k are held each is taken,
then a nearer one replaces the farthest, of equally far ones the one in the highest
slot.  The rule is carried out here, photon by photon, in FP32; the photons returned
have to be the same, on photons of few distinct distances, where most queries meet
many at the k-th."""
import numpy as np
import pytest

from encore_b200 import PhotonMap
from tests.test_gpu_photon_build import image

pytestmark = pytest.mark.gpu
F = np.float32


def cloud(kind, n):
    r = np.random.default_rng(121)
    if kind == "grid":
        p = r.integers(0, 9, (n, 3)).astype(F)
    elif kind == "wall":
        p = r.integers(0, 40, (n, 3)).astype(F)
        p[:, 1] = 0
    else:  # a few places, many photons each
        p = (r.random((7, 3)) * 9.0).astype(F)[r.integers(0, 7, n)]
    nrm = np.eye(3, dtype=F)[r.integers(0, 2, n)]
    return p, nrm, r.random((n, 3)).astype(F)


def walk(tree, q, qn, k, r2, ignore):
    """(squared distance, photon) of the photons kept, by slot."""
    levels, box, leaf, rec = tree
    pos, nrm = rec[0, :, :3], rec[1, :, :3]
    ids = rec[0, :, 3].view(np.int32)
    held, worst = [], None
    stack = [(len(levels), 0, F(0.0))]
    while stack:
        lv, item, d = stack.pop()
        if not d < r2:
            continue
        if lv > 0:
            count, off, pad = levels[lv - 1]
            c = np.arange(32 * item, min(32 * item + 32, count))
            b = box[off:off + 6 * pad].reshape(6, pad)[:, c]
            g = [np.maximum(np.maximum(b[a] - q[a], q[a] - b[3 + a]), F(0)) for a in range(3)]
            cd = (g[0] * g[0] + g[1] * g[1]) + g[2] * g[2]
            near = [(cd[i], int(c[i])) for i in range(len(c)) if cd[i] < r2]
            stack += [(lv - 1, i, x) for x, i in sorted(near, key=lambda e: (-e[0], -e[1]))]
            continue
        at = np.arange(*leaf[item])
        if stack and stack[-1][0] == 0 and stack[-1][2] < r2:
            more = np.arange(*leaf[stack[-1][1]])
            if len(at) + len(more) <= 32:
                stack.pop()
                at = np.concatenate([at, more])
        v = q - pos[at]
        d2 = (v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1]) + v[:, 2] * v[:, 2]
        ok = d2 < r2
        if not ignore:
            ok &= (nrm[at] == qn).all(1)
        for x, i in zip(d2[ok], at[ok]):
            if len(held) < k:
                held.append((x, int(ids[i])))
                if len(held) < k:
                    continue
            elif x < held[worst][0]:
                held[worst] = (x, int(ids[i]))
            else:
                continue
            worst = max(range(k), key=lambda s: (held[s][0], s))
            r2 = held[worst][0]
    return held


@pytest.mark.parametrize("k", [1, 8, 16, 33, 50, 100, 256])
@pytest.mark.parametrize("kind,n,r", [("grid", 900, 3.2), ("grid", 3000, 2.9), ("wall", 4000, 9.5),
                                      ("places", 2000, 30.0)])
def test_ties_at_the_last_place(gpu, kind, n, r, k):
    pos, nrm, pw = cloud(kind, n)
    rng = np.random.default_rng(122)
    q = np.round(rng.random((24, 3)) * (39 if kind == "wall" else 9)).astype(F)
    q[::3] += F(0.5)
    if kind == "wall":
        q[:, 1] = 0
    qn = np.eye(3, dtype=F)[rng.integers(0, 2, 24)]
    dropped = full = 0  # queries with more photons at the last distance; with k photons
    for caustic, ignore in ((False, False), (True, True)):
        pm = PhotonMap(n, caustic=caustic)
        pm.add_photons(pos, nrm, pw)
        pm.balance_and_construct()
        tree = image(pm)[2:6]
        idx, d2, cnt = pm.get_nearest_n_photons(k, r, q, qn, ignore_normal=ignore)
        rgb = pm.get_radiance_estimate(k, r, q, qn, ignore_normal=ignore)
        for i in range(len(q)):
            kept = sorted(walk(tree, q[i], qn[i], k, F(r) * F(r), ignore))
            assert cnt[i] == len(kept)
            assert idx[i, :cnt[i]].tolist() == [p for _, p in kept]
            assert d2[i, :cnt[i]].tolist() == [float(x) for x, _ in kept]
            if not kept:
                continue
            x = np.array([x for x, _ in kept], np.float64)
            at = [p for _, p in kept]
            with np.errstate(divide="ignore", invalid="ignore"):
                w = (x[-1] - x) / x if caustic else np.ones(len(at))
            s = (pw[at].astype(np.float64) * w[:, None]).sum(0)
            if caustic and x[-1] > 0:
                s *= k / (np.float64(F(3.14159)) * x[-1] * x[-1])
            if np.isfinite(s).all():  # (a caustic photon at the query's own place has no weight)
                # as many products and sums, and the estimate's few, of 2^-24 each
                assert np.allclose(rgb[i], s, rtol=(len(at) + 8) * 2.0 ** -24, atol=1e-30)
            v = q[i] - pos
            dist = (v[:, 0] * v[:, 0] + v[:, 1] * v[:, 1]) + v[:, 2] * v[:, 2]
            same = (dist == kept[-1][0]) & (ignore | (nrm == qn[i]).all(1))
            full += len(at) == k
            dropped += len(at) == k and same.sum() > (x == x[-1]).sum()
    assert dropped >= min(8, full // 2)
