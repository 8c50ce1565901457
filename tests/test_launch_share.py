"""Batches spread over the warps without a queue: the launch covers every ray, with at
most 32 rays per warp, on no more blocks than the caller allows.  The rule
(engine.h: ray_share) is compiled by itself here and checked on the CPU over block
sizes, blocks per SM and batch sizes; the hits of such launches on the GPU."""
import subprocess

import pytest

from encore_b200.build import CSRC, INCLUDE

MAIN = r'''
#include <cstdio>
#include "engine.h"
int main() {
  for (int sms : {1, 20, 148})
    for (int block : {32, 64, 96, 128})
      for (int per_sm = 1; per_sm <= 16; ++per_sm) {
        enc::Launch L;
        L.block = block;
        const size_t wpb = block / 32, most = (size_t)sms * per_sm * wpb * 32;
        for (size_t k : {(size_t)0, (size_t)1, (size_t)31, (size_t)33, most / 33, most / 32, most / 32 + 1,
                         most / 2, most - 1, most, most + 1, (size_t)sms * 16, (size_t)sms * 16 + 1,
                         (size_t)sms * 128}) {
          int grid = sms * per_sm;
          const unsigned share = enc::ray_share(L, k, sms, &grid);
          const bool queue = k > most;
          if ((share == 0) != queue || grid < 1 || grid > sms * per_sm || share > 32 ||
              (!queue && (size_t)grid * wpb * share < k)) {
            std::printf("sms %d block %d per_sm %d n %zu: share %u grid %d\\n", sms, block, per_sm, k, share, grid);
            return 1;
          }
        }
        L.fixed_chunk = true;
        int grid = sms * per_sm;
        if (enc::ray_share(L, 5, sms, &grid) != 0 || grid != sms * per_sm) return 2;
      }
  return 0;
}
'''


def test_spread_batches_stay_within_the_callers_blocks(tmp_path):
    (tmp_path / "m.cpp").write_text(MAIN)
    exe = tmp_path / "m"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", str(CSRC), "-I", str(INCLUDE), "-I",
                    "/usr/local/cuda/include", str(tmp_path / "m.cpp"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("block,per_sm", [(0, 1), (32, 0), (32, 1), (96, 2)])
@pytest.mark.parametrize("width", [2, 8])
def test_chosen_shapes_give_the_same_hits(gpu, block, per_sm, width):
    import torch

    from encore_b200 import Accelerator, scenes
    from encore_b200.accel import LaunchConfig
    acc = Accelerator("wbvh", width=width).build(scenes.random_triangles(500, seed=151, scale=1000.0))
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    cfg = LaunchConfig(block_threads=block, blocks_per_sm=per_sm)
    most = sms * (per_sm or 9) * ((block or 128) // 32) * 32
    for n in (1, 128 * sms, most, most + 1):
        d = torch.from_numpy(scenes.random_sphere_rays(n, seed=152, hi=(1000.0,) * 3)).cuda()
        h = [torch.full((n, 4), 7, dtype=torch.int32, device="cuda") for _ in range(2)]
        o = [torch.full((n,), 7, dtype=torch.uint8, device="cuda") for _ in range(2)]
        acc.intersect_device(d, n, h[0], launch=cfg)
        acc.intersect_device(d, n, h[1], launch=LaunchConfig(chunk=32))
        acc.occluded_device(d, n, o[0], launch=cfg)
        acc.occluded_device(d, n, o[1], launch=LaunchConfig(chunk=32))
        acc.check()
        assert torch.equal(h[0], h[1]) and torch.equal(o[0], o[1])
