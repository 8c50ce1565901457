// Ray binning ahead of the closest-hit launch.
//
// An incoherent batch (primaries and diffuse bounces in random order) puts
// rays that share no nodes side by side in a warp.  Binning groups rays by a
// key of their origin cell and direction, so the rays a warp takes from the
// queue walk similar paths through the tree: fewer distinct nodes per warp
// step, more lanes active per instruction, more L1 hits.
//
// Two kernels that stream over the batch, and a scan between them:
//   bin_keys     key per ray (origin cell x direction cell, interleaved bit by
//                bit into one integer) + a histogram of the keys;
//   bin_sums, bin_scan   exclusive prefix sum of the histogram, in place;
//   bin_scatter  each ray's slot in its bucket, order[slot] = ray index.
// The traversal then takes queue index q as ray order[q] and writes its hit
// at that ray's own index, so callers see no reordering.  The order inside a
// bucket depends on atomic timing; the hits do not (each ray's result is a
// function of the ray alone).
//
// Algorithmic bytes: 32 (ray read) + 4 (key write) in the first pass, 4 (key
// read) + 4 (order write) in the last; the histogram is 4 bytes per bucket.
// What bounds the passes is atomics on the buckets that hold most rays (an
// image's eye rays share their origin's cell), so a block first counts the
// keys of kBinTile rays in a table in shared memory: a key's slot is its hash,
// the last key written there owns it, and the others -- rarely a key that many
// rays have -- add to their bucket directly.  2,000,001 rays (a quarter of them
// eye rays), 65,536 buckets: 57 + 108 + 54 us for keys, scan and scatter with
// one add per distinct key of a warp and a scan by one block, about 60 us in all
// now.  1,024 / 2,048 rays per block: 9 / 30 us more; a table that resolves its
// collisions by compare-and-swap: 20 us more; __match_any ahead of the table: 8.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "engine.h"

namespace enc {
namespace {

constexpr unsigned kFullMask = 0xffffffffu;

__device__ __forceinline__ uint32_t quantise(float x, float lo, float scale, int bits) {
  if (bits <= 0) return 0u;
  const float mx = (float)((1u << bits) - 1u);
  float q = (x - lo) * scale;
  q = fminf(fmaxf(q, 0.0f), mx);  // fmaxf drops a NaN: it lands in cell 0
  return (uint32_t)q;
}

// The key of one ray.  Dimensions: origin (or the probe point o + len * d)
// x, y, z over the scene box, then the direction's octahedral coordinates
// u, v in [-1, 1] (the unit direction projected onto the octahedron
// |x| + |y| + |z| = 1, the lower half folded out).  Bits are interleaved from
// the most significant level down, so each prefix of the key is a coarser
// cell of the same five-dimensional grid.
__device__ __forceinline__ uint32_t ray_key(const float4 r0, const float4 r1, const BinSpec& k) {
  float ox = r0.x, oy = r0.y, oz = r0.z;
  const float dx = r1.x, dy = r1.y, dz = r1.z;
  if (k.probe_len > 0.0f) {
    ox = fmaf(k.probe_len, dx, ox);
    oy = fmaf(k.probe_len, dy, oy);
    oz = fmaf(k.probe_len, dz, oz);
  }
  const float ad = fabsf(dx) + fabsf(dy) + fabsf(dz);
  float u = 0.0f, v = 0.0f;
  if (ad > 0.0f) {
    u = dx / ad;
    v = dz / ad;
    if (dy < 0.0f) {
      const float fu = (1.0f - fabsf(v)) * (u < 0.0f ? -1.0f : 1.0f);
      const float fv = (1.0f - fabsf(u)) * (v < 0.0f ? -1.0f : 1.0f);
      u = fu;
      v = fv;
    }
  }
  uint32_t q[5];
  q[0] = quantise(ox, k.lo[0], k.scale[0], k.bits[0]);
  q[1] = quantise(oy, k.lo[1], k.scale[1], k.bits[1]);
  q[2] = quantise(oz, k.lo[2], k.scale[2], k.bits[2]);
  q[3] = quantise(u, -1.0f, 0.5f * (float)(1u << k.bits[3]), k.bits[3]);
  q[4] = quantise(v, -1.0f, 0.5f * (float)(1u << k.bits[4]), k.bits[4]);
  uint32_t key = 0;
#pragma unroll
  for (int d = 0; d < 5; ++d)
    for (int b = 0; b < k.bits[d]; ++b) key |= ((q[d] >> b) & 1u) << k.place[d][b];
  return key;
}

constexpr int kBinRows = 2;
constexpr uint32_t kBinTile = 256 * kBinRows;  // rays a block takes
constexpr uint32_t kBinSlots = 2 * kBinTile;   // slots of the block's table
constexpr int kSlotsPerThread = kBinSlots / 256;
constexpr uint32_t kNoKey = 0xffffffffu;       // keys have at most kBinMaxKeyBits bits

__device__ __forceinline__ uint32_t slot_of(uint32_t key) {
  return (key * 2654435761u) / (0xffffffffu / kBinSlots + 1u);
}

__global__ void __launch_bounds__(256) bin_keys(const float4* __restrict__ rays, uint32_t n,
                                                const __grid_constant__ BinSpec spec,
                                                uint32_t* __restrict__ keys,
                                                uint32_t* __restrict__ hist) {
  __shared__ uint32_t s_key[kBinSlots], s_cnt[kBinSlots];
#pragma unroll
  for (int j = 0; j < kSlotsPerThread; ++j) s_cnt[threadIdx.x + 256 * j] = 0;
  uint32_t key[kBinRows];
#pragma unroll
  for (int r = 0; r < kBinRows; ++r) {
    const uint32_t i = blockIdx.x * kBinTile + r * 256 + threadIdx.x;
    key[r] = kNoKey;
    if (i < n) {
      key[r] = ray_key(__ldg(rays + 2 * (size_t)i), __ldg(rays + 2 * (size_t)i + 1), spec);
      keys[i] = key[r];
      s_key[slot_of(key[r])] = key[r];
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kBinRows; ++r) {
    if (key[r] == kNoKey) continue;
    const uint32_t h = slot_of(key[r]);
    if (s_key[h] == key[r]) atomicAdd(&s_cnt[h], 1u);
    else atomicAdd(hist + key[r], 1u);
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kSlotsPerThread; ++j) {
    const uint32_t c = s_cnt[threadIdx.x + 256 * j];
    if (c) atomicAdd(hist + s_key[threadIdx.x + 256 * j], c);
  }
}

// The scan of the histogram: at most kScanBlocks blocks of `per` buckets each
// (their sums fit in the 256 bytes that the order array always has, which is
// written only later).
constexpr uint32_t kScanBlocks = 64;

// Sum of one value per thread of a block of 256 threads, in every thread; the
// caller's exclusive prefix in *before.
__device__ __forceinline__ uint32_t block_sum(uint32_t v, uint32_t* s_warp, uint32_t* before) {
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(kFullMask, incl, d);
    if ((int)lane >= d) incl += t;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  uint32_t sum = 0, pre = incl - v;
#pragma unroll
  for (unsigned w = 0; w < 8; ++w) {
    if (w < warp) pre += s_warp[w];
    sum += s_warp[w];
  }
  __syncthreads();
  *before = pre;
  return sum;
}

__global__ void __launch_bounds__(256) bin_sums(const uint32_t* __restrict__ hist, uint32_t nb,
                                                uint32_t per, uint32_t* sums) {
  __shared__ uint32_t s_warp[8];
  const uint32_t b = blockIdx.x * per, e = min(b + per, nb);
  uint32_t c = 0, before;
  for (uint32_t i = b + threadIdx.x; i < e; i += 256) c += hist[i];
  c = block_sum(c, s_warp, &before);
  if (threadIdx.x == 0) sums[blockIdx.x] = c;
}

__global__ void __launch_bounds__(256) bin_scan(uint32_t* hist, uint32_t nb, uint32_t per,
                                                const uint32_t* __restrict__ sums) {
  __shared__ uint32_t s_warp[8];
  const uint32_t b = blockIdx.x * per, e = min(b + per, nb);
  uint32_t before;
  uint32_t carry = block_sum(threadIdx.x < blockIdx.x ? sums[threadIdx.x] : 0u, s_warp, &before);
  for (uint32_t at = b; at < e; at += 1024) {
    const uint32_t i = at + 4 * threadIdx.x;
    uint32_t v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = i + k < e ? hist[i + k] : 0u;
    const uint32_t sum = block_sum(v[0] + v[1] + v[2] + v[3], s_warp, &before);
    uint32_t run = carry + before;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (i + k < e) hist[i + k] = run;
      run += v[k];
    }
    carry += sum;
  }
}

__global__ void __launch_bounds__(256) bin_scatter(const uint32_t* __restrict__ keys, uint32_t n,
                                                   uint32_t* __restrict__ offs,
                                                   uint32_t* __restrict__ order) {
  __shared__ uint32_t s_key[kBinSlots], s_cnt[kBinSlots];
#pragma unroll
  for (int j = 0; j < kSlotsPerThread; ++j) s_cnt[threadIdx.x + 256 * j] = 0;
  uint32_t key[kBinRows], rank[kBinRows];
#pragma unroll
  for (int r = 0; r < kBinRows; ++r) {
    const uint32_t i = blockIdx.x * kBinTile + r * 256 + threadIdx.x;
    key[r] = i < n ? __ldg(keys + i) : kNoKey;
    if (i < n) s_key[slot_of(key[r])] = key[r];
  }
  __syncthreads();
  unsigned owned = 0;  // rows whose key has the table's slot
#pragma unroll
  for (int r = 0; r < kBinRows; ++r) {
    const uint32_t h = slot_of(key[r]);
    const bool own = key[r] != kNoKey && s_key[h] == key[r];
    if (own) owned |= 1u << r;
    rank[r] = 0;
    if (own) rank[r] = atomicAdd(&s_cnt[h], 1u);
    else if (key[r] != kNoKey) rank[r] = atomicAdd(offs + key[r], 1u);
  }
  __syncthreads();
  uint32_t base[kSlotsPerThread];
#pragma unroll
  for (int j = 0; j < kSlotsPerThread; ++j) {  // all in flight at once
    const uint32_t c = s_cnt[threadIdx.x + 256 * j];
    base[j] = c ? atomicAdd(offs + s_key[threadIdx.x + 256 * j], c) : 0u;
  }
#pragma unroll
  for (int j = 0; j < kSlotsPerThread; ++j) s_cnt[threadIdx.x + 256 * j] = base[j];
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kBinRows; ++r) {
    const uint32_t i = blockIdx.x * kBinTile + r * 256 + threadIdx.x;
    if (i < n) order[rank[r] + ((owned >> r) & 1u ? s_cnt[slot_of(key[r])] : 0u)] = i;
  }
}

}  // namespace

size_t bin_scratch_bytes(size_t nrays, int key_bits) {
  const size_t a = 256;
  auto up = [&](size_t x) { return (x + a - 1) / a * a; };
  return up(nrays * 4) + up(nrays * 4) + up(((size_t)1 << key_bits) * 4);
}

BinSpec make_bin_spec(const float lo[3], const float hi[3], int key_bits, int dir_bits,
                      float probe_frac) {
  BinSpec k{};
  for (int d = 0; d < 5; ++d) k.bits[d] = 0;
  if (key_bits < 1) key_bits = 1;
  if (key_bits > kBinMaxKeyBits) key_bits = kBinMaxKeyBits;
  if (dir_bits < 0) dir_bits = 0;
  if (dir_bits > key_bits) dir_bits = key_bits;
  float ext[3];
  double diag2 = 0.0;
  for (int i = 0; i < 3; ++i) {
    ext[i] = hi[i] > lo[i] ? hi[i] - lo[i] : 0.0f;
    diag2 += (double)ext[i] * ext[i];
  }
  const float diag = (float)std::sqrt(diag2);
  k.probe_len = probe_frac > 0.0f ? probe_frac * diag : 0.0f;
  // the probe point can leave the scene box by probe_len on every side
  for (int i = 0; i < 3; ++i) {
    k.lo[i] = lo[i] - k.probe_len;
    ext[i] += 2.0f * k.probe_len;
  }
  // direction bits split between u and v, u first
  k.bits[3] = (dir_bits + 1) / 2;
  k.bits[4] = dir_bits / 2;
  // origin bits go one at a time to the axis whose cells are widest, so the
  // cells stay close to cubes (a flat scene spends few bits on its thin axis)
  int left = key_bits - dir_bits;
  float cell[3] = {ext[0], ext[1], ext[2]};
  while (left > 0) {
    int best = 0;
    for (int i = 1; i < 3; ++i)
      if (cell[i] > cell[best]) best = i;
    if (cell[best] <= 0.0f || k.bits[best] >= kBinMaxDimBits) break;
    ++k.bits[best];
    cell[best] *= 0.5f;
    --left;
  }
  for (int i = 0; i < 3; ++i)
    k.scale[i] = ext[i] > 0.0f ? (float)(1u << k.bits[i]) / ext[i] : 0.0f;
  for (int d = 3; d < 5; ++d)
    if (k.bits[d] > kBinMaxDimBits) k.bits[d] = kBinMaxDimBits;
  int total = 0, next = 0;
  for (int d = 0; d < 5; ++d) total += k.bits[d];
  for (int level = kBinMaxDimBits - 1; level >= 0; --level)
    for (int d = 0; d < 5; ++d)
      if (level < k.bits[d]) k.place[d][level] = (uint8_t)(total - 1 - next++);
  return k;
}

int launch_bin(const float* d_rays, size_t n, const BinSpec& spec, void* d_scratch,
               uint32_t** d_order, int device, void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int total = 0;
  for (int d = 0; d < 5; ++d) total += spec.bits[d];
  if (total < 1) total = 1;
  const size_t a = 256;
  auto up = [&](size_t x) { return (x + a - 1) / a * a; };
  char* base = static_cast<char*>(d_scratch);
  uint32_t* keys = reinterpret_cast<uint32_t*>(base);
  uint32_t* order = reinterpret_cast<uint32_t*>(base + up(n * 4));
  uint32_t* hist = reinterpret_cast<uint32_t*>(base + 2 * up(n * 4));
  const uint32_t nb = 1u << total;
  cudaError_t e = cudaMemsetAsync(hist, 0, (size_t)nb * 4, s);
  if (e != cudaSuccess) return (int)e;
  const unsigned tiles = (unsigned)((n + kBinTile - 1) / kBinTile);
  const uint32_t per = std::max(4096u, nb / kScanBlocks);
  const unsigned parts = (nb + per - 1) / per;
  bin_keys<<<tiles, 256, 0, s>>>(reinterpret_cast<const float4*>(d_rays), (uint32_t)n, spec, keys,
                                 hist);
  bin_sums<<<parts, 256, 0, s>>>(hist, nb, per, order);
  bin_scan<<<parts, 256, 0, s>>>(hist, nb, per, order);
  bin_scatter<<<tiles, 256, 0, s>>>(keys, (uint32_t)n, hist, order);
  *d_order = order;
  return (int)cudaGetLastError();
}

}  // namespace enc
