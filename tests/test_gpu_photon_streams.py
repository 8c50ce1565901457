"""Photon maps used on several streams (GPU): a map is complete when the call that
made it returns, by every route -- the host build of a small map, the device build,
a loaded file -- so a stream that nothing orders behind its creation reads it
whole.  The maps are made in memory that other maps have just left."""
import numpy as np
import pytest

from encore_b200 import PhotonMap
from encore_b200.wavefront import photon_map_from_device
from tests.test_gpu_photon_build import photons

pytestmark = pytest.mark.gpu


def queries(n=2000):
    r = np.random.default_rng(161)
    q = (r.random((n, 3)) * [3.0, 1.0, 2.0]).astype(np.float32)
    return q, np.eye(3, dtype=np.float32)[r.integers(0, 3, n)]


@pytest.mark.parametrize("n", [1, 32, 1000, 1024, 1025, 30000])
@pytest.mark.parametrize("route", ["host", "device", "load"])
def test_a_new_map_is_whole_on_any_stream(gpu, n, route):
    import torch
    q, qn = queries()
    dq, dn = torch.from_numpy(q).cuda(), torch.from_numpy(qn).cuda()
    sets = [photons(kind, n) for kind in ("box", "cluster")]

    def make(p):
        if route == "device":
            return photon_map_from_device(*(torch.from_numpy(x).cuda() for x in p), n)
        pm = PhotonMap(n)
        pm.add_photons(*p)
        pm.balance_and_construct()
        return PhotonMap.load(pm.save()) if route == "load" else pm

    want = [make(p).get_radiance_estimate(20, 0.4, q, qn) for p in sets]
    streams = [torch.cuda.Stream() for _ in range(3)]
    out = [torch.zeros(len(q), 3, device="cuda") for _ in range(12)]
    torch.cuda.synchronize()
    for i in range(12):
        pm = make(sets[i % 2])
        pm.get_radiance_estimate_device(20, 0.4, dq, dn, len(q), out[i],
                                        stream=streams[i % 3].cuda_stream)
        del pm
    torch.cuda.synchronize()
    for i in range(12):
        assert np.array_equal(out[i].cpu().numpy().view(np.int32), want[i % 2].view(np.int32))
