"""The scene's bounds after a refit on the device (GPU): of zeros of both signs at a
bound the first vertex's stands, as in the refit on the host, so the saved images
are the same bytes.  The host's refit is compiled by itself (test_refit_stale)."""
import numpy as np
import pytest

from encore_b200 import Accelerator, scenes
from tests.test_gpu_refit_bytes import parts
from tests.test_refit_stale import lib  # noqa: F401 - a fixture

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [2, 4, 8])
@pytest.mark.parametrize("side", [1.0, -1.0])
@pytest.mark.parametrize("first", [0.0, -0.0])
def test_signs_of_zero_bounds(gpu, lib, width, side, first):  # noqa: F811
    n = 700
    base = scenes.random_triangles(n, seed=211, scale=1000.0)
    r = np.random.default_rng(212)
    v = np.abs(base).reshape(-1, 3) * np.float32(side)
    for zero in (0.0, -0.0):
        v[r.random(v.shape) < 0.1] = zero
    for a in range(3):  # the first zero of each axis
        v[np.flatnonzero(v[:, a] == 0)[0], a] = first
    moved = np.ascontiguousarray(v.reshape(-1, 9), np.float32)
    out = np.zeros(400 * n, np.uint8)
    size = lib.refitted(base.ctypes.data, None, moved.ctypes.data, n, width, out.ctypes.data)
    acc = Accelerator("wbvh", width=width).build(base)
    acc.update(moved)
    h, nodes, _, _ = parts(acc.save(), width)
    assert np.array_equal(nodes.reshape(-1), out[:size - 24])
    bounds = np.array(h[9:15], np.float32)
    assert bounds.tobytes() == out[size - 24:size].tobytes()
    assert (bounds == 0).sum() == 3
