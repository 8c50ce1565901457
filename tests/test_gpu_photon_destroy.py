"""Destroying a photon map (GPU): it waits for a gather that still reads the map, and
it neither fails nor spoils a graph that another thread captures meanwhile, in the
capture modes that allow other threads to allocate and free."""
import ctypes as C
import threading

import numpy as np
import pytest

from encore_b200.wavefront import photon_map_from_device
from tests.test_gpu_photon_build import photons

pytestmark = pytest.mark.gpu


def device_photons(kind, n):
    import torch
    return [torch.from_numpy(x).cuda() for x in photons(kind, n)]


def queries():
    import torch
    r = np.random.default_rng(171)
    q = (r.random((3000, 3)) * [3.0, 1.0, 2.0]).astype(np.float32)
    n = np.eye(3, dtype=np.float32)[r.integers(0, 3, 3000)]
    return torch.from_numpy(q).cuda(), torch.from_numpy(n).cuda()


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_other_threads_may_capture(gpu, mode):
    import torch
    n = 20000
    p, (q, qn) = device_photons("box", n), queries()
    want = torch.zeros(3000, 3, device="cuda")
    pm = photon_map_from_device(*p, n)
    pm.get_radiance_estimate_device(20, 0.3, q, qn, 3000, want)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    x = torch.zeros(64, device="cuda")
    got, errors = torch.zeros(3000, 3, device="cuda"), []

    def work():
        try:
            for _ in range(3):
                m = photon_map_from_device(*p, n)
                m.get_radiance_estimate_device(20, 0.3, q, qn, 3000, got, stream=side.cuda_stream)
                m._destroy()
        except Exception as e:  # noqa: BLE001 - reported below
            errors.append(e)

    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, capture_error_mode=mode):
        x.add_(1.0)
        t = threading.Thread(target=work)
        t.start()
        t.join()
        if mode == "relaxed":  # (the other forbids it to the capturing thread)
            pm._destroy()
        x.add_(1.0)
    assert not errors, errors
    g.replay()
    torch.cuda.synchronize()
    assert (x == 2.0).all() and torch.equal(got, want)


def test_it_waits_for_a_gather_under_way(gpu):
    import torch
    n = 40000
    p, other, (q, qn) = device_photons("box", n), device_photons("cluster", n), queries()
    want = torch.zeros(3000, 3, device="cuda")
    pm = photon_map_from_device(*p, n)
    pm.get_radiance_estimate_device(20, 0.3, q, qn, 3000, want)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for _ in range(3):
        out = torch.zeros(3000, 3, device="cuda")
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            torch.cuda._sleep(20_000_000)  # the gather starts some 10 ms later
        pm.get_radiance_estimate_device(20, 0.3, q, qn, 3000, out, stream=side.cuda_stream)
        pm._destroy()
        assert side.query()
        pm2 = photon_map_from_device(*other, n)  # takes the memory
        torch.cuda.synchronize()
        assert torch.equal(out, want)
        pm2._destroy()
        pm = photon_map_from_device(*p, n)
    assert isinstance(pm.handle, C.c_void_p)
