// Device build of the photon tree (layout in photon.h): the host build's tree,
// photon for photon.  Every range is split at its median index on the axis of its
// largest extent by what std::nth_element does there, so the order of equal
// coordinates and of the photons inside a leaf is the host's as well: of photons
// at equal distances a gather keeps those it meets first, and which it meets
// first must not depend on where the map was made.
//
// The algorithm is introselect (Musser 1997): while more than three elements are
// left, a pivot -- the median of the second, the middle and the last element --
// goes to the front, the others are partitioned about it as Hoare does, and the
// search goes on in the part that holds the median; after 2 log2(n) partitions a
// heap selects instead.  Only the partitions are done in parallel.  Hoare's
// pointers stop, from the left, at the elements that are not smaller than the
// pivot and, from the right, at those that are not larger; they exchange the m-th
// of the one with the m-th of the other while it lies to its left.  So an element's
// partner follows from the count of the first kind before it and of the second
// behind it.  The last three elements are put in order, equal ones left as they
// are; the heap is the library's own code.
//
//   * Ranges of more than kShared photons: one cluster of blocks per range narrows
//     the selection in device memory, and its first block ends it in shared memory
//     (split_cluster).
//   * Down to kLeafRange photons: one block per range, in shared memory
//     (split_block).
//   * The levels below that: one launch, one block per such range, its warps in
//     teams of one per range of a level (split_ranges).
//   * The records are written leaf by leaf, and the boxes formed from them.
//
// What bounds it: the length of the chain.  A level takes some eight to fifteen
// partitions, one after another, of about 2,000 cycles in a block (four barriers,
// and little between them) and 17,000 to 40,000 in a cluster.  500,000 photons: 45 ms
// on the host, 0.94 ms here (in a profile 0.62 ms in the five levels of
// split_cluster, 0.17 in the four of split_block, 0.07 in split_ranges).  Clusters of
// 16 blocks, and fewer warps as a block's range shrinks, were no faster; rounds of
// launches over the whole device in place of the clusters took 1.42 ms.  A build that sorts the photons
// along each axis once and splits the lists took 0.51 ms, but orders equal
// coordinates and a leaf's photons otherwise, and gathers with photons at equal
// distances then differed.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>

#include "engine.h"
#include "photon.h"

namespace cg = cooperative_groups;

namespace enc {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr uint32_t kTile = 2048;  // photons of a range that one block of range_extent takes
constexpr int kBlock = 1024;      // threads of the kernels with one block or cluster per range
constexpr unsigned kCluster = 8;  // blocks per cluster
// Elements that a block holds: 8 bytes each, and 2 for the partition's lists.
constexpr uint32_t kShared = 22528;
constexpr size_t kElemBytes = sizeof(float) + sizeof(uint32_t) + sizeof(uint16_t);
constexpr uint32_t kLeafRange = 1024;
// Elements left from which one warp goes on alone: a partition by a team costs it
// four barriers.
constexpr uint32_t kWarpRange = 128;
// A heap over more elements than this is left to the host build.
constexpr uint32_t kMostHeap = 2048;

// An element of a selection: the photon's coordinate on the split axis, and the
// photon.  Its assignment is its own, so the library shifts elements one by one;
// a memmove between overlapping places of shared memory came out wrong.
struct alignas(8) Elem {
  float key;
  uint32_t id;
  constexpr Elem& operator=(const Elem& o) {
    key = o.key;
    id = o.id;
    return *this;
  }
};
struct KeyLess {
  constexpr bool operator()(const Elem& a, const Elem& b) const { return a.key < b.key; }
};

__device__ __forceinline__ unsigned lt_mask() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}
__device__ __forceinline__ uint32_t coord_key(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float of_key(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}
// The coordinate a photon is split by (photon.cpp: split_coord).
__device__ __forceinline__ float split_coord(const float* pos, uint32_t id, int axis) {
  const float c = __ldg(pos + 3 * (size_t)id + axis);
  return isnan(c) ? INFINITY : c;
}

// The extents of a range of photons as six keys that are all maxima: the complement
// of the smallest coordinate's key and the largest one's, per axis; not-a-numbers
// left out.  An empty axis is (+inf, -inf).
struct Extent {
  uint32_t nlo[3], hi[3];
};
__device__ __forceinline__ Extent no_extent() {
  Extent x;
  for (int a = 0; a < 3; ++a) {
    x.nlo[a] = ~coord_key(INFINITY);
    x.hi[a] = coord_key(-INFINITY);
  }
  return x;
}
__device__ __forceinline__ void grow(Extent& x, int a, float c) {
  const bool no = isnan(c);
  x.nlo[a] = max(x.nlo[a], no ? 0u : ~coord_key(c));
  x.hi[a] = max(x.hi[a], no ? 0u : coord_key(c));
}
__device__ __forceinline__ void grow(Extent& x, const float* pos, uint32_t id) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    grow(x, a, __ldg(pos + 3 * (size_t)id + a));
  }
}
__device__ __forceinline__ void warp_extent(Extent& x) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    x.nlo[a] = __reduce_max_sync(kFull, x.nlo[a]);
    x.hi[a] = __reduce_max_sync(kFull, x.hi[a]);
  }
}
__device__ __forceinline__ int widest(const Extent& x) {
  float e[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) e[a] = __fsub_rn(of_key(x.hi[a]), of_key(~x.nlo[a]));
  int axis = 0;
  if (e[1] > e[0]) axis = 1;
  if (e[2] > (axis == 1 ? e[1] : e[0])) axis = 2;
  return axis;
}

// Range s of the tree's level `level`: [b, e), split at m.
struct Range {
  uint32_t b, m, e;
};
__device__ __forceinline__ Range range_of(uint32_t n, int level, uint32_t s) {
  Range r{0u, 0u, n};
  for (int l = level - 1; l >= 0; --l) {
    const uint32_t m = r.b + (r.e - r.b) / 2;
    if ((s >> l) & 1u) r.b = m;
    else r.e = m;
  }
  r.m = r.b + (r.e - r.b) / 2;
  return r;
}

__device__ __forceinline__ int select_depth(uint32_t n) { return 2 * (31 - __clz((int)n)); }

// Which of the places x, y, z holds the median of their keys x, y, z.
__device__ __forceinline__ uint32_t median_place(uint32_t x, float kx, uint32_t y, float ky, uint32_t z,
                                                 float kz) {
  if (kx < ky) return ky < kz ? y : (kx < kz ? z : x);
  return kx < kz ? x : (ky < kz ? z : y);
}

// ---------------------------------------------------------------------------
// Partitions.  A team of warps -- one, some of a block, a block, a cluster -- has
//   warps(), warp()   how many it has, and which of them the caller is;
//   sync()            a barrier that also orders the team's memory accesses;
//   offsets(ge, le)   of the counts of all its warps: the sum of `ge` over the
//                     warps before the caller's, of `le` over those behind it;
//   results(swaps, cut)  the sum and the minimum over its warps.
// The last two are barriers too.

struct WarpTeam {
  __device__ unsigned warps() const { return 1; }
  __device__ unsigned warp() const { return 0; }
  __device__ void sync() const { __syncwarp(); }
  __device__ void offsets(uint32_t& ge, uint32_t& le) const { ge = le = 0; }
  __device__ void results(uint32_t&, uint32_t&) const { __syncwarp(); }
};

// What the warps of a block tell each other.
struct TeamShared {
  uint32_t ge[kBlock / 32], le[kBlock / 32], swaps[kBlock / 32], cut[kBlock / 32];
  uint32_t all_ge, all_le, all_swaps, all_cut;  // of a block of a cluster
};

// `n` warps of a block, from warp `first` on; id: their barrier (0: the block's).
struct BlockTeam {
  unsigned n, first, id;
  TeamShared& s;
  __device__ unsigned warps() const { return n; }
  __device__ unsigned warp() const { return (threadIdx.x >> 5) - first; }
  __device__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n * 32) : "memory"); }
  __device__ void put_counts(uint32_t ge, uint32_t le) const {
    if ((threadIdx.x & 31u) == 0) {
      s.ge[warp()] = ge;
      s.le[warp()] = le;
    }
    sync();
  }
  __device__ void offsets(uint32_t& ge, uint32_t& le) const {
    put_counts(ge, le);
    const unsigned lane = threadIdx.x & 31u;
    ge = __reduce_add_sync(kFull, lane < warp() ? s.ge[lane] : 0u);
    le = __reduce_add_sync(kFull, lane > warp() && lane < n ? s.le[lane] : 0u);
  }
  __device__ void results(uint32_t& swaps, uint32_t& cut) const {
    const unsigned lane = threadIdx.x & 31u;
    if (lane == 0) {
      s.swaps[warp()] = swaps;
      s.cut[warp()] = cut;
    }
    sync();
    swaps = __reduce_add_sync(kFull, lane < n ? s.swaps[lane] : 0u);
    cut = __reduce_min_sync(kFull, lane < n ? s.cut[lane] : ~0u);
  }
};

// The blocks of a cluster.
struct ClusterTeam {
  BlockTeam block;
  unsigned rank;
  __device__ unsigned warps() const { return block.n * kCluster; }
  __device__ unsigned warp() const { return rank * block.n + block.warp(); }
  __device__ void sync() const { cg::this_cluster().sync(); }
  __device__ const TeamShared& of(unsigned r) const { return *cg::this_cluster().map_shared_rank(&block.s, r); }
  __device__ void offsets(uint32_t& ge, uint32_t& le) const {
    block.put_counts(ge, le);
    const unsigned lane = threadIdx.x & 31u, w = block.warp();
    const uint32_t g = lane < block.n ? block.s.ge[lane] : 0u, e = lane < block.n ? block.s.le[lane] : 0u;
    if (w == 0) {
      const uint32_t all_ge = __reduce_add_sync(kFull, g), all_le = __reduce_add_sync(kFull, e);
      if (lane == 0) {
        block.s.all_ge = all_ge;
        block.s.all_le = all_le;
      }
    }
    sync();
    ge = __reduce_add_sync(kFull, (lane < w ? g : 0u) + (lane < rank ? of(lane).all_ge : 0u));
    le = __reduce_add_sync(kFull, (lane > w ? e : 0u) + (lane > rank && lane < kCluster ? of(lane).all_le : 0u));
  }
  __device__ void results(uint32_t& swaps, uint32_t& cut) const {
    block.results(swaps, cut);
    const unsigned lane = threadIdx.x & 31u;
    if (threadIdx.x == 0) {
      block.s.all_swaps = swaps;
      block.s.all_cut = cut;
    }
    sync();
    swaps = __reduce_add_sync(kFull, lane < kCluster ? of(lane).all_swaps : 0u);
    cut = __reduce_min_sync(kFull, lane < kCluster ? of(lane).all_cut : ~0u);
  }
};

// Partitions a[f, l) (more than three elements) about its pivot and returns the first
// place of the right part, in (f, l).  Element i has partner number (elements not
// smaller than the pivot before it) in the left list, or (elements not larger
// behind it) in the right one; lp, rp: room for (l - f) / 2 places each.
template <class Team, class Place>
__device__ __forceinline__ uint32_t partition(const Team& team, Elem* a, uint32_t f, uint32_t l,
                                              Place* lp, Place* rp) {
  const unsigned lane = threadIdx.x & 31u, lt = lt_mask();
  if (team.warp() == 0) {
    const uint32_t mid = f + (l - f) / 2;
    const uint32_t at = median_place(f + 1, a[f + 1].key, mid, a[mid].key, l - 1, a[l - 1].key);
    __syncwarp();
    if (lane == 0) {
      const Elem x = a[f];
      a[f] = a[at];
      a[at] = x;
    }
  }
  team.sync();
  const float p = a[f].key;
  const uint32_t rows = (l - f - 1 + 31) / 32, per = (rows + team.warps() - 1) / team.warps() * 32;
  const uint32_t b = min(f + 1 + team.warp() * per, l), e = min(b + per, l);
  uint32_t nge = 0, nle = 0;
#pragma unroll 4
  for (uint32_t r = b; r < e; r += 32) {
    const float k = a[min(r + lane, e - 1)].key;
    nge += __popc(__ballot_sync(kFull, r + lane < e && !(k < p)));
    nle += __popc(__ballot_sync(kFull, r + lane < e && !(p < k)));
  }
  uint32_t before = nge, behind = nle;
  team.offsets(before, behind);
  behind += nle;
  uint32_t swaps = 0, cut = l;
#pragma unroll 4
  for (uint32_t r = b; r < e; r += 32) {
    const uint32_t i = r + lane;
    const float k = a[min(i, e - 1)].key;
    const bool ge = i < e && !(k < p), le = i < e && !(p < k);
    const unsigned gm = __ballot_sync(kFull, ge), em = __ballot_sync(kFull, le);
    const uint32_t cg = before + __popc(gm & lt);
    const uint32_t cl = behind - __popc(em & lt) - (le ? 1u : 0u);
    const bool left = ge && cl > cg, right = le && cg > cl;
    if (left) lp[cg] = (Place)i;
    if (right) rp[cl] = (Place)i;
    if ((ge && !left) || right) cut = min(cut, i);
    swaps += __popc(__ballot_sync(kFull, left));
    before += __popc(gm);
    behind -= __popc(em);
  }
  cut = __reduce_min_sync(kFull, cut);
  team.results(swaps, cut);
  for (uint32_t m = team.warp() * 32 + lane; m < swaps; m += team.warps() * 32) {
    const uint32_t x = lp[m], y = rp[m];
    const Elem ex = a[x];
    a[x] = a[y];
    a[y] = ex;
  }
  team.sync();
  return cut;
}

// The same of at most 32 elements, lane i holding element i of c; n: the median's
// place.  Goes on until at most three are left or the partitions are used up;
// [f, l) is what is left.
__device__ __forceinline__ void lanes_narrow(Elem& x, uint32_t& f, uint32_t& l, uint32_t nth, int& depth,
                                             uint8_t* place, unsigned lane) {
  const unsigned lt = lt_mask();
  while (l - f > 3 && depth > 0) {
    --depth;
    const uint32_t mid = f + (l - f) / 2;
    const float k1 = __shfl_sync(kFull, x.key, f + 1), k2 = __shfl_sync(kFull, x.key, mid),
                k3 = __shfl_sync(kFull, x.key, l - 1);
    const uint32_t at = median_place(f + 1, k1, mid, k2, l - 1, k3);
    const uint32_t from = lane == f ? at : (lane == at ? f : lane);
    x.key = __shfl_sync(kFull, x.key, from);
    x.id = __shfl_sync(kFull, x.id, from);
    const float p = __shfl_sync(kFull, x.key, f);
    const bool on = lane > f && lane < l;
    const bool ge = on && !(x.key < p), le = on && !(p < x.key);
    const unsigned gm = __ballot_sync(kFull, ge), em = __ballot_sync(kFull, le);
    const int cg = __popc(gm & lt), cl = __popc(em & ~lt) - (le ? 1 : 0);
    const bool left = ge && cl > cg, right = le && cg > cl;
    const unsigned stops = __ballot_sync(kFull, (ge && !left) || right);
    if (left) place[cg] = (uint8_t)lane;
    if (right) place[16 + cl] = (uint8_t)lane;
    __syncwarp();
    const unsigned partner = left ? place[16 + cg] : (right ? place[cl] : lane);
    __syncwarp();
    x.key = __shfl_sync(kFull, x.key, partner);
    x.id = __shfl_sync(kFull, x.id, partner);
    const uint32_t cut = stops ? (uint32_t)__ffs(stops) - 1u : l;
    if (cut <= nth) f = cut;
    else l = cut;
  }
}

// One warp: the selection goes on in a[f, l) with `depth` partitions left.  lp, rp:
// as for partition(); place: 32 bytes of the warp's own.
template <class Place>
__device__ __forceinline__ void warp_select(Elem* a, uint32_t f, uint32_t l, uint32_t nth, int depth,
                                            Place* lp, Place* rp, uint8_t* place) {
  const unsigned lane = threadIdx.x & 31u;
  while (l - f > 32 && depth > 0) {
    --depth;
    const uint32_t cut = partition(WarpTeam{}, a, f, l, lp, rp);
    if (cut <= nth) f = cut;
    else l = cut;
  }
  if (l - f <= 32) {
    const uint32_t c = l - f, base = f;
    Elem x = a[base + min(lane, c - 1)];
    uint32_t lf = 0, ll = c;
    lanes_narrow(x, lf, ll, nth - base, depth, place, lane);
    if (ll - lf <= 3) {  // the rest is sorted by insertion, which keeps equal elements' order
      uint32_t rank = lf;
      for (uint32_t i = lf; i < ll; ++i) {
        const float k = __shfl_sync(kFull, x.key, i);
        rank += k < x.key || (!(x.key < k) && i < lane) ? 1u : 0u;
      }
      if (lane < c) a[base + (lane >= lf && lane < ll ? rank : lane)] = x;
      __syncwarp();
      return;
    }
    if (lane < c) a[base + lane] = x;
    f = base + lf;
    l = base + ll;
    __syncwarp();
  }
  if (lane == 0)  // no partitions left: a heap
    std::__introselect(a + f, a + nth, a + l, 0, __gnu_cxx::__ops::__iter_comp_iter(KeyLess()));
  __syncwarp();
}

// Partitions while more than `most` elements are left and partitions are.
template <class Team, class Place>
__device__ __forceinline__ void narrow(const Team& team, Elem* a, uint32_t& f, uint32_t& l, uint32_t nth,
                                       int& depth, uint32_t most, Place* lp, Place* rp) {
  while (l - f > most && depth > 0) {
    --depth;
    const uint32_t cut = partition(team, a, f, l, lp, rp);
    if (cut <= nth) f = cut;
    else l = cut;
  }
}

// The selection by a team of a block, in shared memory; `refused` is set where a
// heap over more than kMostHeap elements would have to end it.
template <class Place>
__device__ __forceinline__ void team_select(const BlockTeam& team, Elem* a, uint32_t f, uint32_t l,
                                            uint32_t nth, int depth, Place* lp, Place* rp, uint8_t* place,
                                            uint32_t* refused) {
  narrow(team, a, f, l, nth, depth, kWarpRange, lp, rp);
  if (team.warp() == 0) {
    if (l - f > kMostHeap) *refused = 1;
    else warp_select(a, f, l, nth, depth, lp, rp, place);
  }
  team.sync();
}

// ---------------------------------------------------------------------------
// Levels of ranges larger than kShared: all blocks, over tiles of the ranges, as
// many of every range as its level's largest has.
struct Tile {
  uint32_t range, tile;
};
__device__ __forceinline__ Tile tile_of(uint32_t tiles) {
  return Tile{blockIdx.x / tiles, blockIdx.x % tiles};
}

__global__ void __launch_bounds__(kThreads) range_extent(const float* __restrict__ pos,
                                                         const Elem* __restrict__ w, uint32_t n,
                                                         int level, uint32_t tiles, uint32_t* ext) {
  const Tile at = tile_of(tiles);
  __shared__ Extent s_ext[kWarps];
  const Range r = range_of(n, level, at.range);
  const uint32_t b = r.b + at.tile * kTile, e = min(b + kTile, r.e);
  Extent x = no_extent();
#pragma unroll 4
  for (uint32_t i = b + threadIdx.x; i < e; i += kThreads) grow(x, pos, level ? w[i].id : i);
  warp_extent(x);
  if ((threadIdx.x & 31u) == 0) s_ext[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x < 6) {
    uint32_t v = 0;
    for (int k = 0; k < kWarps; ++k)
      v = max(v, threadIdx.x < 3 ? s_ext[k].nlo[threadIdx.x] : s_ext[k].hi[threadIdx.x - 3]);
    atomicMax(ext + 6 * (size_t)at.range + threadIdx.x, v);
  }
}
__device__ __forceinline__ Extent load_extent(const uint32_t* ext, uint32_t s) {
  Extent x;
  for (int a = 0; a < 3; ++a) {
    x.nlo[a] = __ldg(ext + 6 * (size_t)s + a);
    x.hi[a] = __ldg(ext + 6 * (size_t)s + 3 + a);
  }
  return x;
}

__global__ void __launch_bounds__(kThreads) load_keys(const float* __restrict__ pos, Elem* w, uint32_t n,
                                                      int level, uint32_t tiles,
                                                      const uint32_t* __restrict__ ext) {
  const Tile at = tile_of(tiles);
  const Range r = range_of(n, level, at.range);
  const int axis = widest(load_extent(ext, at.range));
  const uint32_t b = r.b + at.tile * kTile, e = min(b + kTile, r.e);
#pragma unroll 4
  for (uint32_t i = b + threadIdx.x; i < e; i += kThreads) {
    const uint32_t id = level ? w[i].id : i;
    w[i] = Elem{split_coord(pos, id, axis), id};
  }
}

// One cluster per range.  lp, rp: a range's lists lie at its own place in them.
__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kBlock)
    split_cluster(Elem* w, uint32_t n, int level, uint32_t* lp, uint32_t* rp, uint32_t* refused) {
  extern __shared__ Elem s_elem[];
  __shared__ TeamShared s_team;
  __shared__ uint8_t s_place[32];
  const unsigned rank = cg::this_cluster().block_rank();
  const BlockTeam block{kBlock / 32, 0, 0, s_team};
  const Range r = range_of(n, level, blockIdx.x / kCluster);
  uint32_t f = r.b, l = r.e;
  int depth = select_depth(r.e - r.b);
  narrow(ClusterTeam{block, rank}, w, f, l, r.m, depth, kShared, lp + r.b, rp + r.b);
  if (rank != 0) return;  // (nothing reads its shared memory any more)
  if (l - f > kShared) {
    if (threadIdx.x == 0) *refused = 1;
    return;
  }
  const uint32_t c = l - f;
  uint16_t* lists = reinterpret_cast<uint16_t*>(s_elem + kShared);
  for (uint32_t i = threadIdx.x; i < c; i += kBlock) s_elem[i] = w[f + i];
  __syncthreads();
  team_select(block, s_elem, 0, c, r.m - f, depth, lists, lists + kShared / 2, s_place, refused);
  for (uint32_t i = threadIdx.x; i < c; i += kBlock) w[f + i] = s_elem[i];
}

// ---------------------------------------------------------------------------
// One block per range of at most `cap` <= kShared photons: one level's split.
__global__ void __launch_bounds__(kBlock) split_block(const float* __restrict__ pos, Elem* w, uint32_t n,
                                                      int level, uint32_t cap, uint32_t* refused) {
  extern __shared__ Elem s_elem[];
  __shared__ TeamShared s_team;
  __shared__ uint8_t s_place[32];
  __shared__ Extent s_ext[kBlock / 32];
  uint16_t* lists = reinterpret_cast<uint16_t*>(s_elem + cap);
  const Range r = range_of(n, level, blockIdx.x);
  const uint32_t c = r.e - r.b;
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  Extent x = no_extent();
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < c; i += blockDim.x) {
    const uint32_t id = level ? w[r.b + i].id : i;
    s_elem[i].id = id;
    grow(x, pos, id);
  }
  warp_extent(x);
  if (lane == 0) s_ext[warp] = x;
  __syncthreads();
  x = lane < (blockDim.x >> 5) ? s_ext[lane] : no_extent();
  warp_extent(x);
  const int axis = widest(x);
#pragma unroll 4
  for (uint32_t i = threadIdx.x; i < c; i += blockDim.x) s_elem[i].key = split_coord(pos, s_elem[i].id, axis);
  __syncthreads();
  team_select(BlockTeam{blockDim.x >> 5, 0, 0, s_team}, s_elem, 0, c, r.m - r.b, select_depth(c), lists,
              lists + cap / 2, s_place, refused);
  for (uint32_t i = threadIdx.x; i < c; i += blockDim.x) w[r.b + i] = s_elem[i];
}

// One block per range of at most kLeafRange photons: every level below `top`, its
// warps in as many teams as the level has ranges, or more than one range to a warp.
// w null: the photons in their own order.  order: the photons of the leaves.
__global__ void __launch_bounds__(kThreads) split_ranges(const float* __restrict__ pos,
                                                         const Elem* __restrict__ w, uint32_t n, int top,
                                                         int depth, uint32_t* order, uint32_t* refused) {
  __shared__ float s_pos[3][kLeafRange];
  __shared__ uint32_t s_id[kLeafRange];
  __shared__ Elem s_elem[kLeafRange];
  __shared__ uint16_t s_lists[kLeafRange];
  __shared__ TeamShared s_team[kWarps / 2];
  __shared__ Extent s_ext[kWarps];
  __shared__ uint8_t s_place[kWarps][32];
  const Range all = range_of(n, top, blockIdx.x);
  const uint32_t c = all.e - all.b;
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  for (uint32_t i = threadIdx.x; i < c; i += kThreads) {
    const uint32_t id = w ? w[all.b + i].id : i;
    s_id[i] = id;
    s_elem[i].id = i;
#pragma unroll
    for (int a = 0; a < 3; ++a) s_pos[a][i] = __ldg(pos + 3 * (size_t)id + a);
  }
  __syncthreads();
  for (int level = top; level < depth; ++level) {
    const uint32_t count = 1u << (level - top);
    const unsigned tw = count < kWarps ? kWarps / count : 1u;  // warps per team
    for (uint32_t s = warp / tw; s < count; s += kWarps / tw) {
      const Range r = range_of(c, level - top, s);
      const unsigned first = warp / tw * tw, tlane = (warp - first) * 32 + lane;
      const BlockTeam team{tw, first, 1 + warp / tw, s_team[tw > 1 ? warp / tw : 0]};
      Extent x = no_extent();
      for (uint32_t i = r.b + tlane; i < r.e; i += 32 * tw) {
        const uint32_t j = s_elem[i].id;
#pragma unroll
        for (int a = 0; a < 3; ++a) grow(x, a, s_pos[a][j]);
      }
      warp_extent(x);
      if (tw > 1) {
        if (lane == 0) s_ext[warp] = x;
        team.sync();
        x = lane < tw ? s_ext[first + lane] : no_extent();
        warp_extent(x);
      }
      const int axis = widest(x);
      for (uint32_t i = r.b + tlane; i < r.e; i += 32 * tw) {
        const float v = s_pos[axis][s_elem[i].id];
        s_elem[i].key = isnan(v) ? INFINITY : v;
      }
      uint16_t *lp = s_lists + r.b, *rp = lp + (r.e - r.b) / 2;
      if (tw > 1) {
        team.sync();
        team_select(team, s_elem, r.b, r.e, r.m, select_depth(r.e - r.b), lp, rp, s_place[warp], refused);
      } else {
        __syncwarp();
        warp_select(s_elem, r.b, r.e, r.m, select_depth(r.e - r.b), lp, rp, s_place[warp]);
      }
    }
    __syncthreads();
  }
  for (uint32_t i = threadIdx.x; i < c; i += kThreads) order[all.b + i] = s_id[s_elem[i].id];
}

// The bounds of a warp's 32 boxes to item j of a level's arrays.  Of equal bounds
// the first lane's is written: a zero's sign is the host build's then.
__device__ __forceinline__ void put_bounds(float (&lo)[3], float (&hi)[3], float* box, uint32_t pad,
                                           uint32_t j, unsigned lane) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    float least = lo[a], most = hi[a];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      least = fminf(least, __shfl_xor_sync(kFull, least, d));
      most = fmaxf(most, __shfl_xor_sync(kFull, most, d));
    }
    lo[a] = __shfl_sync(kFull, lo[a], __ffs(__ballot_sync(kFull, lo[a] == least)) - 1);
    hi[a] = __shfl_sync(kFull, hi[a], __ffs(__ballot_sync(kFull, hi[a] == most)) - 1);
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
// range, its photons' records and their bounds.
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
      const uint32_t s = order ? __ldg(order + b + lane) : b + lane;
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

size_t up256(size_t x) { return (x + 255) / 256 * 256; }
uint32_t most_in_range(size_t n, int level) {
  return (uint32_t)((n + ((size_t)1 << level) - 1) >> level);
}
// Ranges of the last level that split_cluster splits.
size_t cluster_ranges(size_t n) {
  int level = 0;
  while (most_in_range(n, level) > kShared) ++level;
  return (size_t)1 << (level > 0 ? level - 1 : 0);
}

}  // namespace

size_t photon_build_scratch(size_t n) {
  return up256(4 * n) + up256(24 * cluster_ranges(n)) + 256;
}

int build_photon_device(const float* pos, const float* nrm, const float* pw, const DevPhotonMap& d,
                        void* scratch, bool* refused) {
  const uint32_t n = d.n;
  const size_t ranges = cluster_ranges(n);
  // The record arrays, written last, hold the elements and the lists of the
  // partitions (8, 4 and 4 bytes per photon); the order of the records and the
  // tables lie in the scratch.
  Elem* w = reinterpret_cast<Elem*>(d.d_pos4);
  uint32_t* lp = reinterpret_cast<uint32_t*>(w + n);
  uint32_t* rp = lp + n;
  char* base = static_cast<char*>(scratch);
  uint32_t* order = reinterpret_cast<uint32_t*>(base);
  base += up256(4 * (size_t)n);
  uint32_t* ext = reinterpret_cast<uint32_t*>(base);
  uint32_t* flag = reinterpret_cast<uint32_t*>(base + up256(24 * ranges));
  cudaError_t e = cudaMemsetAsync(flag, 0, 4);
  const size_t full = kShared * kElemBytes;
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(split_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)full);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(split_block, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)full);
  if (e != cudaSuccess) return (int)e;
  if (d.depth > 0) {
    int level = 0;
    for (; most_in_range(n, level) > kShared; ++level) {
      const uint32_t c = most_in_range(n, level), count = 1u << level;
      const uint32_t tiles = (c + kTile - 1) / kTile, grid = tiles * count;
      if ((e = cudaMemsetAsync(ext, 0, 24 * (size_t)count)) != cudaSuccess) return (int)e;
      range_extent<<<grid, kThreads>>>(pos, w, n, level, tiles, ext);
      load_keys<<<grid, kThreads>>>(pos, w, n, level, tiles, ext);
      split_cluster<<<count * kCluster, kBlock, full>>>(w, n, level, lp, rp, flag);
    }
    for (; level < d.depth && most_in_range(n, level) > kLeafRange; ++level) {
      const uint32_t cap = (most_in_range(n, level) + 1) / 2 * 2;
      split_block<<<1u << level, kBlock, cap * kElemBytes>>>(pos, w, n, level, cap, flag);
    }
    split_ranges<<<1u << level, kThreads>>>(pos, level ? w : nullptr, n, level, d.depth, order, flag);
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
  e = cudaGetLastError();
  uint32_t bad = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&bad, flag, 4, cudaMemcpyDeviceToHost, 0);
  if (e == cudaSuccess) e = cudaStreamSynchronize(0);
  *refused = bad != 0;
  return (int)e;
}

}  // namespace enc
