"""The order of the photons in a map (GPU): of photons at equal distances a gather
keeps those it meets first, so a map built on the device holds its photons in
the order of the host build, photon for photon, equal coordinates included.  The
host build (photon.cpp) is compiled by itself here and gives the expected arrays.
Sizes lie at the edges of the device build's forms: the host build's limit, 32
and 1,024 photons per range, the most that one block holds, the first size that
takes a cluster, and sizes with ranges of each kind."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from encore_b200 import PhotonMap
from encore_b200.build import CSRC, INCLUDE
from encore_b200.wavefront import photon_map_from_device
from tests.test_gpu_photon_build import image, photons

WRAPPER = r'''
#include <algorithm>
#include <cstring>
#include <vector>
#include "photon.h"
extern "C" long tree(const float* pos, const float* nrm, const float* pow, long n, unsigned* leaf,
                     float* box, float* rec) {
  enc::PhotonHost h;
  enc::build_photon_tree(pos, nrm, pow, n, &h);
  std::memcpy(leaf, h.leaf.data(), 4 * h.leaf.size());
  std::memcpy(box, h.box.data(), 4 * h.box.size());
  std::memcpy(rec, h.pos4.data(), 16 * n);
  std::memcpy(rec + 4 * n, h.nrm4.data(), 16 * n);
  std::memcpy(rec + 8 * n, h.pow4.data(), 16 * n);
  return (long)h.box.size();
}
// Keys on which nth_element's partitions stay lopsided (McIlroy, "A killer
// adversary for quicksort", 1999): an element gets its value when it has to.
extern "C" void killer(long n, float* key) {
  std::vector<int> val(n, (int)n), at(n);
  for (int i = 0; i < n; ++i) at[i] = i;
  int solid = 0, candidate = 0;
  std::nth_element(at.begin(), at.begin() + n / 2, at.end(), [&](int x, int y) {
    if (val[x] == n && val[y] == n) val[x == candidate ? x : y] = solid++;
    if (val[x] == n) candidate = x;
    else if (val[y] == n) candidate = y;
    return val[x] < val[y];
  });
  for (int i = 0; i < n; ++i) key[i] = (float)val[i];
}
'''
P = C.c_void_p


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    d = tmp_path_factory.mktemp("photon_host")
    (d / "w.cpp").write_text(WRAPPER)
    so = d / "libphoton_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-pthread", "-ffp-contract=off",
                    "-I", str(CSRC), "-I", str(INCLUDE), "-I", "/usr/local/cuda/include",
                    str(d / "w.cpp"), str(CSRC / "photon.cpp"), "-o", str(so)], check=True)
    lib = C.CDLL(str(so))
    lib.tree.argtypes = [P, P, P, C.c_long, P, P, P]
    lib.tree.restype = C.c_long
    lib.killer.argtypes = [C.c_long, P]
    return lib


def order_photons(host, kind, n):
    r = np.random.default_rng(95)
    if kind in ("line", "pipe", "killer", "odd"):
        pos, nrm, pw = photons("box", n)
        i = np.arange(n)
        if kind == "killer":
            x = np.empty(n, np.float32)
            host.killer(n, x.ctypes.data)
            pos = np.ascontiguousarray(np.stack([x, 0 * x, 0 * x], 1))
        elif kind == "odd":
            pos[r.random((n, 3)) < 0.01] = np.inf
            pos[r.random((n, 3)) < 0.01] = -np.inf
            pos[r.random((n, 3)) < 0.01] = np.nan
        else:
            pos[:, 0] = i if kind == "line" else np.minimum(i, n - 1 - i)
        return pos, nrm, pw
    return photons(kind, n)


def check(host, pm, pos, nrm, pw):
    n = len(pos)
    _, depth, levels, box, leaf, rec = image(pm)
    want_leaf, want_box, want_rec = np.empty_like(leaf), np.empty_like(box), np.empty_like(rec)
    assert host.tree(pos.ctypes.data, nrm.ctypes.data, pw.ctypes.data, n, want_leaf.ctypes.data,
                     want_box.ctypes.data, want_rec.ctypes.data) == len(box)
    assert np.array_equal(rec[0, :, 3].view(np.int32), want_rec[0, :, 3].view(np.int32))
    assert np.array_equal(rec.view(np.int32), want_rec.view(np.int32))
    assert np.array_equal(leaf, want_leaf)
    assert np.array_equal(box.view(np.int32), want_box.view(np.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("kind,n", [
    ("box", 33), ("box", 1024), ("box", 1025), ("grid", 2049), ("point", 5000), ("plane", 22528),
    ("box", 22529), ("cluster", 45057), ("line", 40000), ("pipe", 73731), ("odd", 100003),
    ("grid", 150001), ("box", 500000), ("plane", 500000), ("point", 200000), ("cluster", 1300001)])
def test_device_maps_hold_the_host_builds_order(gpu, host, kind, n):
    import torch
    pos, nrm, pw = order_photons(host, kind, n)
    pm = photon_map_from_device(*(torch.from_numpy(x).cuda() for x in (pos, nrm, pw)), n)
    check(host, pm, pos, nrm, pw)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1500, 3000, 20000, 60000])
def test_photons_that_only_the_host_build_selects(gpu, host, n):
    import torch
    pos, nrm, pw = order_photons(host, "killer", n)
    pm = photon_map_from_device(*(torch.from_numpy(x).cuda() for x in (pos, nrm, pw)), n)
    check(host, pm, pos, nrm, pw)
    pm = PhotonMap(n)
    pm.add_photons(pos, nrm, pw)
    pm.balance_and_construct()
    check(host, pm, pos, nrm, pw)
