"""The gather's candidate buffer (GPU): k at the edges of the buffer's sizes,
searches that find far more photons than k (the k nearest are kept again and
again), photons at equal distances, and launches of one query, of one query per
warp and of one more.  The distances are the k smallest of the accepted photons,
formed in FP32 in the photon test's order, and the radiance is the FP64 sum's over
the photons returned."""
import numpy as np
import pytest

from encore_b200 import PhotonMap

pytestmark = pytest.mark.gpu
F = np.float32


def cloud(kind, n, seed=101):
    r = np.random.default_rng(seed)
    if kind == "grid":  # few distinct distances
        p = r.integers(0, 12, (n, 3)).astype(F)
    elif kind == "point":
        p = np.full((n, 3), F(2.0))
    else:
        p = r.random((n, 3)).astype(F) * F(12.0)
    nrm = np.eye(3, dtype=F)[r.integers(0, 2, n)]
    return p, nrm, r.random((n, 3)).astype(F)


def distances(pos, q):
    d = q - pos
    x, y, z = (d[:, a] * d[:, a] for a in range(3))
    return (x + y) + z


def check(pm, pos, nrm, pw, q, qn, k, r, ignore, caustic):
    idx, d2, cnt = pm.get_nearest_n_photons(k, r, q, qn, ignore_normal=ignore)
    rgb = pm.get_radiance_estimate(k, r, q, qn, ignore_normal=ignore)
    for i in range(len(q)):
        d = distances(pos, q[i])
        ok = d < F(r) * F(r)
        if not ignore:
            ok &= (nrm == qn[i]).all(1)
        ok = np.nonzero(ok)[0]
        want = np.sort(d[ok])[:k]
        c = cnt[i]
        assert c == len(want)
        assert np.array_equal(d2[i, :c], want) and (d2[i, c:] == 0).all() and (idx[i, c:] == -1).all()
        got = idx[i, :c]
        assert len(set(got.tolist())) == c and np.isin(got, ok).all()
        assert np.array_equal(d[got], d2[i, :c])
        same = np.diff(d2[i, :c]) == 0
        assert (np.diff(got)[same] > 0).all()  # by distance, then by index
        # the photons of the last distance may be others than the gather's
        if c and (d[ok] == want[-1]).sum() == (want == want[-1]).sum():
            w = np.ones(c)
            if caustic:
                dd = d2[i, :c].astype(np.float64)
                w = (dd[-1] - dd) / dd
            s = (pw[got].astype(np.float64) * w[:, None]).sum(0)
            if caustic:
                s *= k / (np.float64(F(3.14159)) * dd[-1] * dd[-1])
            # c products and sums, and the estimate's few, of 2^-24 each
            assert np.allclose(rgb[i], s, rtol=(c + 8) * 2.0 ** -24, atol=1e-30)


@pytest.mark.parametrize("k", [1, 15, 16, 17, 32, 33, 64, 65, 128, 129, 255, 256])
@pytest.mark.parametrize("kind,n,r", [("box", 6000, 1.1), ("box", 6000, 30.0), ("grid", 6000, 3.5),
                                      ("point", 1500, 9.0)])
def test_the_k_nearest_are_kept(gpu, k, kind, n, r):
    pos, nrm, pw = cloud(kind, n)
    rng = np.random.default_rng(102)
    q = (rng.random((24, 3)) * 12.0).astype(F)
    if kind == "grid":
        q[::2] = np.round(q[::2])
        q += F(0.25)
    qn = np.eye(3, dtype=F)[rng.integers(0, 2, 24)]
    for caustic, ignore in ((False, False), (True, True)):
        pm = PhotonMap(n, caustic=caustic)
        pm.add_photons(pos, nrm, pw)
        check(pm, pos, nrm, pw, q, qn, k, r, ignore, caustic)


@pytest.mark.parametrize("warps", ["one", "all", "all+1", "chunks"])
def test_launch_sizes(gpu, warps):
    import torch
    pos, nrm, pw = cloud("box", 3000)
    pm = PhotonMap(3000)
    pm.add_photons(pos, nrm, pw)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    for blocks in (4, 5, 6):  # resident blocks of 8 warps per SM
        full = sms * blocks * 8
        n = {"one": 1, "all": full, "all+1": full + 1, "chunks": 16 * full + 3}[warps]
        rng = np.random.default_rng(103)
        q = (rng.random((n, 3)) * 12.0).astype(F)
        qn = np.eye(3, dtype=F)[rng.integers(0, 2, n)]
        rgb = pm.get_radiance_estimate(20, 2.0, q, qn)
        step = max(1, n // 40)
        part = pm.get_radiance_estimate(20, 2.0, q[::step], qn[::step])
        assert np.array_equal(rgb[::step].view(np.int32), part.view(np.int32))
        assert (rgb[-1] == pm.get_radiance_estimate(20, 2.0, q[-1:], qn[-1:])[0]).all()
