// Device build of the photon tree (layout in photon.h): the host build's tree
// shape -- every range split at its median index on the axis of its largest
// extent, leaves of at most 32 photons, 32-ary boxes above them -- formed level
// by level from three sorted lists.
//
//   1. The photons are sorted along x, y and z: stable 8-bit counting passes
//      over order-preserving keys, the three axes side by side.
//   2. For each level of the tree: in the list of its split axis, a range's
//      photons at and beyond the median position go right; every list is then
//      split stably, so it stays sorted inside each new range.  A range's extent
//      is the distance of its list's ends, and its place after the split needs
//      only the count of right-going photons before it in the list: the ranges
//      of a level have two sizes, so the count at a range's start has a closed
//      form.
//      Ranges of at most 1,024 photons are split to the leaves in shared memory.
//   3. The records are written leaf by leaf from the x list, and the boxes
//      formed from them.
//
// The tree differs from the host build's (nth_element) only in the order of
// photons inside a leaf and on equal coordinates, neither of which a k-nearest
// set depends on.
//
// What bounds it: some 50 short launches (18 for the sort, three per level) of a
// few microseconds, each streaming 4 to 24 bytes per photon and axis through L2.
// 500,000 photons: 44.9 ms on the host, 0.63 ms here with a launch triple for every
// level, 0.51 with the last five in shared memory.
#include <cuda_runtime.h>

#include <algorithm>

#include "engine.h"
#include "photon.h"

namespace enc {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kThreads = 256, kRows = 8, kWarps = kThreads / 32;
constexpr uint32_t kTile = kThreads * kRows;

__device__ __forceinline__ unsigned lt_mask() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}
__device__ __forceinline__ uint32_t coord_key(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
// Item i of an axis's list (key, photon) and its digit in counting pass `pass`.
// Passes 0 and 1 sort by the upper half of the next axis's key, passes 2 to 5 by
// the axis's own key, so photons of equal coordinate -- a wall's -- are ordered
// along the wall and a split among them parts it instead of halving its density
// (a k = 50 gather in a room tested 183 photons a query with the ties in photon
// order, 159 with this).
constexpr int kPasses = 6;
struct Item {
  uint2 v;
  uint32_t digit;
};
__device__ __forceinline__ Item sort_item(const float* pos, const uint2* in, uint32_t n, int axis,
                                          int pass, uint32_t i) {
  Item it;
  it.v = in ? in[(size_t)axis * n + i] : make_uint2(coord_key(__ldg(pos + 3 * (size_t)i + axis)), i);
  const uint32_t key =
      pass < 2 ? coord_key(__ldg(pos + 3 * (size_t)it.v.y + (axis == 2 ? 0 : axis + 1))) : it.v.x;
  it.digit = (key >> (pass < 2 ? 16 + 8 * pass : 8 * (pass - 2))) & 255u;
  return it;
}

// grid (tiles, 3): digit counts of each tile, hist[(axis * 256 + digit) * tiles + tile].
__global__ void __launch_bounds__(kThreads) sort_count(const float* __restrict__ pos,
                                                       const uint2* __restrict__ in, uint32_t n,
                                                       int pass, uint32_t* hist) {
  __shared__ uint32_t s_cnt[256];
  const int axis = blockIdx.y;
  s_cnt[threadIdx.x] = 0;
  __syncthreads();
  for (int r = 0; r < kRows; ++r) {
    const uint32_t i = blockIdx.x * kTile + r * kThreads + threadIdx.x;
    if (i < n) atomicAdd(&s_cnt[sort_item(pos, in, n, axis, pass, i).digit], 1u);
  }
  __syncthreads();
  hist[(size_t)(axis * 256 + threadIdx.x) * gridDim.x + blockIdx.x] = s_cnt[threadIdx.x];
}

// Exclusive scan of one value per thread of a block of kThreads; total: the sum.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* s_warp, uint32_t* total) {
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const uint32_t t = __shfl_up_sync(kFull, incl, d);
    if ((int)lane >= d) incl += t;
  }
  if (lane == 31) s_warp[warp] = incl;
  __syncthreads();
  uint32_t before = 0, sum = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    if (w < (int)warp) before += s_warp[w];
    sum += s_warp[w];
  }
  __syncthreads();
  *total = sum;
  return before + incl - v;
}

// grid (256, 3): exclusive scan of one digit's tile counts; sums[axis * 256 + digit].
__global__ void __launch_bounds__(kThreads) sort_scan(uint32_t* hist, uint32_t tiles,
                                                      uint32_t* sums) {
  __shared__ uint32_t s_warp[kWarps];
  uint32_t* row = hist + (size_t)(blockIdx.y * 256 + blockIdx.x) * tiles;
  uint32_t carry = 0;
  for (uint32_t b = 0; b < tiles; b += kThreads) {
    const uint32_t i = b + threadIdx.x;
    uint32_t total;
    const uint32_t x = block_scan(i < tiles ? row[i] : 0u, s_warp, &total);
    if (i < tiles) row[i] = carry + x;
    carry += total;
  }
  if (threadIdx.x == 0) sums[blockIdx.y * 256 + blockIdx.x] = carry;
}

// grid (tiles, 3): each tile's items to their places, in order.  A warp takes
// kRows * 32 consecutive items; the lanes of a row with the same digit are
// ranked by __match_any, rows and warps by running counts.
__global__ void __launch_bounds__(kThreads) sort_move(const float* __restrict__ pos,
                                                      const uint2* __restrict__ in, uint32_t n,
                                                      int pass, const uint32_t* __restrict__ hist,
                                                      const uint32_t* __restrict__ sums, uint2* out,
                                                      uint32_t* list) {
  __shared__ uint32_t s_cnt[kWarps][256], s_base[256], s_warp[kWarps];
  const int axis = blockIdx.y;
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = lt_mask();
  for (int w = 0; w < kWarps; ++w) s_cnt[w][threadIdx.x] = 0;
  uint32_t total;
  s_base[threadIdx.x] = block_scan(sums[axis * 256 + threadIdx.x], s_warp, &total) +
                        hist[(size_t)(axis * 256 + threadIdx.x) * gridDim.x + blockIdx.x];
  __syncthreads();
  Item item[kRows];
  uint32_t rank[kRows];
  const uint32_t first = blockIdx.x * kTile + warp * (kRows * 32) + lane;
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    const uint32_t i = first + r * 32;
    item[r] = i < n ? sort_item(pos, in, n, axis, pass, i) : Item{make_uint2(0u, 0u), 256u};
    const uint32_t digit = item[r].digit;
    const unsigned peers = __match_any_sync(kFull, digit);
    const int leader = __ffs(peers) - 1;
    uint32_t old = 0;
    if (i < n && (int)lane == leader) {
      old = s_cnt[warp][digit];
      s_cnt[warp][digit] = old + __popc(peers);
    }
    rank[r] = __shfl_sync(kFull, old, leader) + __popc(peers & lt);
    __syncwarp();
  }
  __syncthreads();
  {  // thread d: the places of digit d, warp by warp
    uint32_t at = s_base[threadIdx.x];
    for (int w = 0; w < kWarps; ++w) {
      const uint32_t c = s_cnt[w][threadIdx.x];
      s_cnt[w][threadIdx.x] = at;
      at += c;
    }
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    if (first + r * 32 >= n) continue;
    const size_t to = (size_t)axis * n + s_cnt[warp][item[r].digit] + rank[r];
    if (list) list[to] = item[r].v.y;
    else out[to] = item[r].v;
  }
}

// The range of the tree's level `level` that list position p lies in.
struct Range {
  uint32_t b, m, e, s;  // [b, e) split at m; s: its index in the level
};
__device__ __forceinline__ Range range_of(uint32_t n, int level, uint32_t p) {
  Range r{0u, 0u, n, 0u};
  for (int l = 0; l < level; ++l) {
    const uint32_t m = r.b + (r.e - r.b) / 2;
    const bool right = p >= m;
    r.s = 2 * r.s + (right ? 1u : 0u);
    if (right) r.b = m;
    else r.e = m;
  }
  r.m = r.b + (r.e - r.b) / 2;
  return r;
}

// The right-going photons of the ranges before g, in a level whose range sizes
// are q and q + 1: a range of size z sends (z + 1) / 2 right, so they sent
// (g.b + how many of them are odd) / 2; g.b - g.s * q of them have size q + 1.
__device__ __forceinline__ uint32_t ones_before(const Range& g, uint32_t q) {
  const uint32_t big = g.b - g.s * q;
  return (g.b + ((q & 1u) ? g.s - big : big)) / 2;
}

// The side of every photon at this level: 1 beyond the median of its range in
// the list of the range's widest axis.
__global__ void __launch_bounds__(kThreads) split_side(const float* __restrict__ pos,
                                                       const uint32_t* __restrict__ lists,
                                                       uint32_t n, int level, uint8_t* side) {
  for (uint32_t p = blockIdx.x * kThreads + threadIdx.x; p < n; p += gridDim.x * kThreads) {
    const Range r = range_of(n, level, p);
    float ext[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const uint32_t* list = lists + (size_t)a * n;
      ext[a] = __ldg(pos + 3 * (size_t)__ldg(list + r.e - 1) + a) -
               __ldg(pos + 3 * (size_t)__ldg(list + r.b) + a);
    }
    int axis = 0;
    if (ext[1] > ext[0]) axis = 1;
    if (ext[2] > (axis == 1 ? ext[1] : ext[0])) axis = 2;
    side[__ldg(lists + (size_t)axis * n + p)] = p >= r.m ? 1 : 0;
  }
}

// grid (tiles, 3): photons of each tile that go right.
__global__ void __launch_bounds__(kThreads) split_count(const uint32_t* __restrict__ lists,
                                                        const uint8_t* __restrict__ side,
                                                        uint32_t n, uint32_t* cnt) {
  __shared__ uint32_t s_sum;
  if (threadIdx.x == 0) s_sum = 0;
  __syncthreads();
  uint32_t c = 0;
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    const uint32_t p = blockIdx.x * kTile + r * kThreads + threadIdx.x;
    if (p < n) c += side[__ldg(lists + (size_t)blockIdx.y * n + p)];
  }
  c = __reduce_add_sync(kFull, c);
  if ((threadIdx.x & 31u) == 0 && c) atomicAdd(&s_sum, c);
  __syncthreads();
  if (threadIdx.x == 0) cnt[blockIdx.y * gridDim.x + blockIdx.x] = s_sum;
}

// grid (tiles, 3): the stable split of each list.
__global__ void __launch_bounds__(kThreads) split_move(const uint32_t* __restrict__ lists,
                                                       const uint8_t* __restrict__ side,
                                                       uint32_t n, int level,
                                                       const uint32_t* __restrict__ cnt,
                                                       uint32_t* out) {
  __shared__ uint32_t s_part[kWarps], s_row[kRows * kWarps];
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, lt = lt_mask();
  const uint32_t* list = lists + (size_t)blockIdx.y * n;
  // right-going photons of the tiles before this one
  uint32_t before = 0;
  for (uint32_t t = threadIdx.x; t < blockIdx.x; t += kThreads)
    before += __ldg(cnt + blockIdx.y * gridDim.x + t);
  before = __reduce_add_sync(kFull, before);
  if (lane == 0) s_part[warp] = before;
  uint32_t id[kRows], in_row[kRows];
  unsigned right = 0;
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    const uint32_t p = blockIdx.x * kTile + r * kThreads + threadIdx.x;
    id[r] = p < n ? __ldg(list + p) : 0u;
    const bool one = p < n && side[id[r]] != 0;
    const unsigned m = __ballot_sync(kFull, one);
    right |= (one ? 1u : 0u) << r;
    in_row[r] = __popc(m & lt);
    if (lane == 0) s_row[r * kWarps + warp] = __popc(m);
  }
  __syncthreads();
  if (warp == 0) {  // exclusive scan of the 64 row pieces, two per lane
    const uint32_t a = s_row[2 * lane], b = s_row[2 * lane + 1];
    uint32_t incl = a + b;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t t = __shfl_up_sync(kFull, incl, d);
      if ((int)lane >= d) incl += t;
    }
    s_row[2 * lane] = incl - a - b;
    s_row[2 * lane + 1] = incl - b;
  }
  before = 0;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) before += s_part[w];
  __syncthreads();
  const uint32_t q = n >> level;  // the level's range sizes are q and q + 1
#pragma unroll
  for (int r = 0; r < kRows; ++r) {
    const uint32_t p = blockIdx.x * kTile + r * kThreads + threadIdx.x;
    if (p >= n) continue;
    const Range g = range_of(n, level, p);
    const uint32_t ones = before + s_row[r * kWarps + warp] + in_row[r] - ones_before(g, q);
    out[(size_t)blockIdx.y * n + ((right >> r) & 1u ? g.m + ones : p - ones)] = id[r];
  }
}

// The levels below `top` in shared memory: one block per range of at most kRange
// photons, its three lists as places in its x list.  `inv` (one word per photon)
// takes the photons' places in that list.  order: the photons of the last level.
constexpr uint32_t kRange = 1024;
constexpr int kPer = kRange / kThreads;  // consecutive list places per thread
__global__ void __launch_bounds__(kThreads) split_ranges(const float* __restrict__ pos,
                                                         const uint32_t* lists, uint32_t* inv,
                                                         uint32_t n, int top, int depth,
                                                         uint32_t* order) {
  __shared__ float s_pos[3][kRange];
  __shared__ uint32_t s_id[kRange], s_warp[kWarps];
  __shared__ uint16_t s_list[2][3][kRange];
  __shared__ uint8_t s_side[kRange];
  uint32_t b = 0, e = n;
  for (int l = top - 1; l >= 0; --l) {
    const uint32_t m = b + (e - b) / 2;
    if ((blockIdx.x >> l) & 1u) b = m;
    else e = m;
  }
  const uint32_t c = e - b;
  for (uint32_t i = threadIdx.x; i < c; i += kThreads) {
    const uint32_t id = lists[b + i];
    s_id[i] = id;
    inv[id] = i;
    s_list[0][0][i] = (uint16_t)i;
#pragma unroll
    for (int a = 0; a < 3; ++a) s_pos[a][i] = __ldg(pos + 3 * (size_t)id + a);
  }
  __syncthreads();
  for (int a = 1; a < 3; ++a)
    for (uint32_t i = threadIdx.x; i < c; i += kThreads)
      s_list[0][a][i] = (uint16_t)inv[lists[(size_t)a * n + b + i]];
  __syncthreads();
  int cur = 0;
  for (int level = top; level < depth; ++level, cur ^= 1) {
    Range g[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const uint32_t p = kPer * threadIdx.x + j;
      if (p >= c) continue;
      g[j] = range_of(c, level - top, p);
      float ext[3];
#pragma unroll
      for (int a = 0; a < 3; ++a)
        ext[a] = s_pos[a][s_list[cur][a][g[j].e - 1]] - s_pos[a][s_list[cur][a][g[j].b]];
      int axis = 0;
      if (ext[1] > ext[0]) axis = 1;
      if (ext[2] > (axis == 1 ? ext[1] : ext[0])) axis = 2;
      s_side[s_list[cur][axis][p]] = p >= g[j].m ? 1 : 0;
    }
    __syncthreads();
    const uint32_t q = c >> (level - top);
    const int nlists = level == depth - 1 ? 1 : 3;
    for (int a = 0; a < nlists; ++a) {
      uint32_t id[kPer], one[kPer], sum = 0, total;
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        const uint32_t p = kPer * threadIdx.x + j;
        id[j] = p < c ? s_list[cur][a][p] : 0u;
        one[j] = p < c ? s_side[id[j]] : 0u;
        sum += one[j];
      }
      uint32_t before = block_scan(sum, s_warp, &total);
#pragma unroll
      for (int j = 0; j < kPer; ++j) {
        const uint32_t p = kPer * threadIdx.x + j;
        if (p < c) {
          const uint32_t ones = before - ones_before(g[j], q);
          s_list[cur ^ 1][a][one[j] ? g[j].m + ones : p - ones] = (uint16_t)id[j];
        }
        before += one[j];
      }
    }
    __syncthreads();
  }
  for (uint32_t i = threadIdx.x; i < c; i += kThreads) order[b + i] = s_id[s_list[cur][0][i]];
}

// The bounds of a warp's 32 boxes to item j of a level's arrays.
__device__ __forceinline__ void put_bounds(float (&lo)[3], float (&hi)[3], float* box, uint32_t pad,
                                           uint32_t j, unsigned lane) {
#pragma unroll
  for (int d = 16; d > 0; d >>= 1)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = fminf(lo[a], __shfl_xor_sync(kFull, lo[a], d));
      hi[a] = fmaxf(hi[a], __shfl_xor_sync(kFull, hi[a], d));
    }
  if (lane < 6) {
    float v = lo[0];
    if (lane == 1) v = lo[1];
    if (lane == 2) v = lo[2];
    if (lane == 3) v = hi[0];
    if (lane == 4) v = hi[1];
    if (lane == 5) v = hi[2];
    box[(size_t)lane * pad + j] = v;
  }
}

// One warp per leaf (pad of them; those past count get inverted boxes): its
// range, its photons' records and their bounds.  The photons lie in a stride
// through their x order: a leaf in x order offers a gather's heap ever nearer
// photons, each of which replaces the maximum (2.7 % on a k = 50 gather).
__global__ void __launch_bounds__(kThreads) write_leaves(
    const float* __restrict__ pos, const float* __restrict__ nrm, const float* __restrict__ pw,
    const uint32_t* __restrict__ order, uint32_t n, int depth, uint32_t count, uint32_t pad,
    uint2* leaf, float* box, float4* pos4, float4* nrm4, float4* pow4) {
  const uint32_t j = blockIdx.x * kWarps + (threadIdx.x >> 5);
  const unsigned lane = threadIdx.x & 31u;
  if (j >= pad) return;
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  if (j < count) {
    uint32_t b = 0, e = n;
    for (int l = depth - 1; l >= 0; --l) {
      const uint32_t m = b + (e - b) / 2;
      if ((j >> l) & 1u) b = m;
      else e = m;
    }
    if (lane == 0) leaf[j] = make_uint2(b, e);
    const uint32_t c = e - b;  // at most 32
    if (lane < c) {
      const uint32_t stride = c % 11u ? 11u : 13u;  // coprime to c
      const uint32_t i = b + (lane * stride) % c;
      const uint32_t s = order ? __ldg(order + i) : i;
      const size_t k = 3 * (size_t)s;
      const float4 p = make_float4(__ldg(pos + k), __ldg(pos + k + 1), __ldg(pos + k + 2),
                                   __int_as_float((int)s));
      pos4[b + lane] = p;
      nrm4[b + lane] = make_float4(__ldg(nrm + k), __ldg(nrm + k + 1), __ldg(nrm + k + 2), 0.f);
      pow4[b + lane] = make_float4(__ldg(pw + k), __ldg(pw + k + 1), __ldg(pw + k + 2), 0.f);
      lo[0] = fminf(lo[0], p.x), lo[1] = fminf(lo[1], p.y), lo[2] = fminf(lo[2], p.z);
      hi[0] = fmaxf(hi[0], p.x), hi[1] = fmaxf(hi[1], p.y), hi[2] = fmaxf(hi[2], p.z);
    }
  }
  put_bounds(lo, hi, box, pad, j, lane);
}

// One warp per item of a box level above the leaves: the bounds of 32 items of
// the level below.
__global__ void __launch_bounds__(kThreads) write_boxes(float* box, uint32_t count, uint32_t pad,
                                                        const float* below, uint32_t below_count,
                                                        uint32_t below_pad) {
  const uint32_t j = blockIdx.x * kWarps + (threadIdx.x >> 5);
  const unsigned lane = threadIdx.x & 31u;
  if (j >= pad) return;
  float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  if (j < count && 32u * j + lane < below_count) {
    const float* c = below + 32u * j + lane;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      lo[a] = c[(size_t)a * below_pad];
      hi[a] = c[(size_t)(3 + a) * below_pad];
    }
  }
  put_bounds(lo, hi, box, pad, j, lane);
}

}  // namespace

size_t photon_build_scratch(size_t n) {
  const size_t tiles = (n + kTile - 1) / kTile;
  return 4 * n + 256 + n + 256 + (3 * 256 * tiles + 3 * 256) * 4;
}

int build_photon_device(const float* pos, const float* nrm, const float* pw, const DevPhotonMap& d,
                        void* scratch) {
  const uint32_t n = d.n;
  const size_t tiles = (n + kTile - 1) / kTile;
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  // The record arrays, written last, hold the items while they are sorted (24
  // bytes per photon each, in turn) and then, in their second half, the lists
  // (12 each, in turn); the last level's x list, the order of the records, and
  // the counts lie in the scratch.
  uint2* items[2] = {reinterpret_cast<uint2*>(d.d_pos4),
                     reinterpret_cast<uint2*>(d.d_pos4) + 3 * (size_t)n};
  uint32_t* lists[2] = {reinterpret_cast<uint32_t*>(items[1]),
                        reinterpret_cast<uint32_t*>(items[1]) + 3 * (size_t)n};
  char* base = static_cast<char*>(scratch);
  uint32_t* order = reinterpret_cast<uint32_t*>(base);
  uint8_t* side = reinterpret_cast<uint8_t*>(base + up(4 * (size_t)n));
  uint32_t* hist = reinterpret_cast<uint32_t*>(base + up(4 * (size_t)n) + up(n));
  uint32_t* sums = hist + 3 * 256 * tiles;
  const dim3 tg((unsigned)tiles, 3);
  const unsigned flat =
      (unsigned)std::min<size_t>(((size_t)n + kThreads - 1) / kThreads, (size_t)device_sm_count(d.device) * 8);
  if (d.depth > 0) {
    static_assert(kPasses % 2 == 0, "the last pass reads items[0] and writes over items[1]");
    for (int pass = 0; pass < kPasses; ++pass) {
      const uint2* in = pass == 0 ? nullptr : items[(pass & 1) ^ 1];
      sort_count<<<tg, kThreads>>>(pos, in, n, pass, hist);
      sort_scan<<<dim3(256, 3), kThreads>>>(hist, (uint32_t)tiles, sums);
      sort_move<<<tg, kThreads>>>(pos, in, n, pass, hist, sums, items[pass & 1],
                                  pass == kPasses - 1 ? lists[0] : nullptr);
    }
    int cur = 0, top = 0;
    while (((n + (1ull << top) - 1) >> top) > kRange) {
      split_side<<<flat, kThreads>>>(pos, lists[cur], n, top, side);
      split_count<<<tg, kThreads>>>(lists[cur], side, n, hist);
      split_move<<<tg, kThreads>>>(lists[cur], side, n, top, hist, lists[cur ^ 1]);
      cur ^= 1;
      ++top;
    }
    split_ranges<<<1u << top, kThreads>>>(pos, lists[cur], lists[cur ^ 1], n, top, d.depth, order);
  }
  write_leaves<<<(d.lvl_pad[0] + kWarps - 1) / kWarps, kThreads>>>(
      pos, nrm, pw, d.depth > 0 ? order : nullptr, n, d.depth, d.lvl_count[0], d.lvl_pad[0],
      reinterpret_cast<uint2*>(d.d_leaf), d.d_box + d.lvl_off[0],
      reinterpret_cast<float4*>(d.d_pos4), reinterpret_cast<float4*>(d.d_nrm4),
      reinterpret_cast<float4*>(d.d_pow4));
  for (int l = 1; l < d.nlevels; ++l)
    write_boxes<<<(d.lvl_pad[l] + kWarps - 1) / kWarps, kThreads>>>(
        d.d_box + d.lvl_off[l], d.lvl_count[l], d.lvl_pad[l], d.d_box + d.lvl_off[l - 1],
        d.lvl_count[l - 1], d.lvl_pad[l - 1]);
  const cudaError_t e = cudaGetLastError();
  return e != cudaSuccess ? (int)e : (int)cudaStreamSynchronize(0);
}

}  // namespace enc
