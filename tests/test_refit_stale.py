"""A refit on the host takes nothing from the boxes it finds: after refits on the device,
which leave the host's copy of the boxes as they were, it gives the bytes that it
gives after refits on the host.  The host build and refit (wbvh_build.cpp) are
compiled by themselves here."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from encore_b200 import scenes
from encore_b200.build import CSRC, INCLUDE

WRAPPER = r'''
#include <cstring>
#include "engine.h"
using namespace enc;
// Refits a tree over `base` to `last`, with or without a refit to `between` before
// it; the node bytes, and the bounds behind them.
extern "C" long refitted(const float* base, const float* between, const float* last, unsigned n, int width,
                         unsigned char* out) {
  WBVHHost h;
  build_wbvh(base, n, width, 3, &h);
  if (between) refit_wbvh(&h, between, n);
  refit_wbvh(&h, last, n);
  std::memcpy(out, h.nodes.data(), h.nodes.size());
  std::memcpy(out + h.nodes.size(), h.lo, 12);
  std::memcpy(out + h.nodes.size() + 12, h.hi, 12);
  return (long)h.nodes.size() + 24;
}
'''


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("refit_host")
    (d / "w.cpp").write_text(WRAPPER)
    so = d / "librefit_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-fPIC", "-shared", "-pthread", "-ffp-contract=off",
                    "-I", str(CSRC), "-I", str(INCLUDE), "-I", "/usr/local/cuda/include",
                    str(d / "w.cpp"), str(CSRC / "wbvh_build.cpp"), "-o", str(so)], check=True)
    x = C.CDLL(str(so))
    x.refitted.argtypes = [C.c_void_p] * 3 + [C.c_uint, C.c_int, C.c_void_p]
    x.refitted.restype = C.c_long
    return x


@pytest.mark.parametrize("width", [2, 4, 8])
@pytest.mark.parametrize("n", [1, 7, 400, 3000])
def test_boxes_found_do_not_matter(lib, width, n):
    r = np.random.default_rng(201)
    base = scenes.random_triangles(n, seed=202, scale=1000.0)
    between = (base * np.float32(7.5) + np.float32(300.0)).astype(np.float32)
    last = (base + r.normal(0, 30, base.shape)).astype(np.float32)
    out = [np.zeros(400 * n + 1000, np.uint8) for _ in range(2)]
    size = [lib.refitted(base.ctypes.data, b, last.ctypes.data, n, width, o.ctypes.data)
            for b, o in ((None, out[0]), (between.ctypes.data, out[1]))]
    assert size[0] == size[1] and np.array_equal(out[0], out[1])
