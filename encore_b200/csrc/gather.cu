// Photon k-nearest gather and radiance estimate for sm_100a.
//
// One warp per query point.  The warp walks the 32-ary box tree over the
// photon kd leaves (photon.h) with a per-warp stack in shared memory: at an
// inner node each lane tests one child box against the search sphere and the
// children that can hold an accepted photon are pushed together (a leaf as
// its photon range); at a leaf each lane tests one photon, and two sibling
// leaves share one step when their photons fit in the warp (one coalesced
// 16-byte load per lane per array).  A box is pruned by its FP32 squared
// distance to the query, formed with the photon test's own operations on the
// box's clamped coordinates; rounding is monotone, so that distance never
// exceeds the squared distance of a photon inside the box and pruning drops
// nothing the photon test would accept.  Accepted photons are appended to a
// buffer in shared memory; when a step leaves more than `full` of them, the k
// nearest are kept (keep_nearest) and their largest distance becomes the search
// radius; before that it is max_dist^2.  The radius never falls below the k-th
// distance of the photons seen, so at the end the k nearest of the buffer are the
// exact k-nearest set, as in PhotonMap::GetNearestNPhotons
// (PhotonMap.cpp:224-297).
//
// What bounds it is instruction issue, not memory (L2 holds what it reads).  A
// bounded max-heap across the warp's registers, whose maximum every accepted
// photon replaced with two warp reductions, took 916 us for 300,007 queries of
// k = 50 in a room of 400,000 photons, 1,434 us for 100,007 of k = 256, and 7.6 ms
// for 1M of k = 50 that find 600 photons each; the buffer takes 620, 765 us and
// 4.5 ms, and one query at a time per warp where there are few 24 instead of 77
// us for 1,007.  `full` = k + max(16, 3k/4): more photons per selection against
// a radius that shrinks later.  k + 0 / 8 / 16 / 32 / 64 for those: 713 / 666 / 648 /
// 621 / 617, 995 / 901 / 835 / 765 / 764 us, 5.6 / 5.1 / 4.7 / 4.5 / 4.4 ms; for k = 8:
// 373 / 364 / 359 / 368 / 368 us.  Noting the dropped ties (heap_insert) costs 1.4 %.
//
// Acceptance is the reference's: FP32 dist^2 = (x*x + y*y) + z*z with separate
// roundings, dist^2 < r^2, and the stored surface normal equal to the query
// normal component by component unless ENC_GATHER_IGNORE_NORMAL
// (PhotonMap.cpp:239-244).  The estimate follows GetRadianceEstimate
// (PhotonMap.cpp:121-164): r = largest dist^2 found; weight 1 (global map) or
// (r - d)/d (caustic map); density 1 or k / (pi r^2) with pi = 3.14159f
// (Common.h:36); FP32 accumulation.
#include <cuda_runtime.h>

#include <algorithm>

#include "../../include/encore_b200.h"
#include "photon.h"

namespace enc {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kWarpsPerBlock = 8;
constexpr unsigned kMaxSteps = 1u << 24;
// Queries a warp takes from the queue at a time, at most.
constexpr unsigned kQueryChunk = 4;

struct GatherParams {
  const float* box;
  const uint2* leaf;
  int nlevels;
  uint32_t lvl_count[kPhotonMaxLevels];
  uint32_t lvl_off[kPhotonMaxLevels];
  uint32_t lvl_pad[kPhotonMaxLevels];
  const float4* pos4;
  const float4* nrm4;
  const float4* pow4;
  const float* qpos;
  const float* qnrm;
  float* rgb;
  int32_t* idx;
  float* d2;
  int32_t* count;
  uint32_t* status;
  uint32_t* counter;  // this launch's query-queue head, zeroed before it
  uint32_t* visits;   // COUNT: 4 words per query (see gather_kernel)
  unsigned nq;
  unsigned chunk;  // queries a warp takes from the queue at a time; 0: warp w takes query w
  int k;
  int full;        // candidates a step may leave before the k nearest are kept
  float r2max;
  int ignore_normal;
  int caustic;
};

__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }

// Stack entries: (item, squared distance of its box).  An inner-node item is
// level << 28 | index (level 1..7); a leaf item is kLeafEntry | first photon, with
// the leaf's photon count (at most 32) in the low 6 bits of the distance, so a
// leaf step reads its photons without first loading its range.  Those bits only
// lower the distance, by less than 2^-17 of it: a box is then visited that its own
// distance would just have pruned, and its photons are tested one by one.
constexpr uint32_t kLeafEntry = 0x80000000u;
constexpr uint32_t kCountBits = 63u;

// The smallest of a warp's candidates: keeps, of the `count` entries of buf
// (squared distance, photon; count <= 32 S), the k nearest, in their order, and
// returns the k-th distance.  A threshold with exactly k entries below it is
// searched between 0 and the largest: on a surface the number of photons within
// a distance grows with its square, so interpolating the counts finds one in a
// few steps; after kGuesses of them the interval is halved, and entries of equal
// distance at its end are kept in order; *tie is that distance then (some of its
// entries were dropped).  Squared distances are non-negative, so their bit
// patterns order as unsigned integers.
constexpr int kGuesses = 8;
template <int S>
__device__ __forceinline__ float keep_nearest(uint2* buf, int count, int k, int lane, unsigned lt,
                                              uint32_t* tie) {
  uint2 e[S];
  uint32_t top = 0;
#pragma unroll
  for (int s = 0; s < S; ++s) {
    e[s] = s * 32 + lane < count ? buf[s * 32 + lane] : make_uint2(~0u, 0u);
    if (s * 32 + lane < count) top = max(top, e[s].x);
  }
  uint32_t lo = 0, hi = __reduce_max_sync(kFull, top) + 1;  // keys lie in [lo, hi)
  int clo = 0, chi = count;                                 // entries below lo and hi
  int ties = 0;                                             // of value lo that are kept
  for (int i = 0;; ++i) {
    if (hi - lo == 1) {
      ties = k - clo;
      if (lane == 0) *tie = lo;
      break;
    }
    uint32_t t = lo + (hi - lo) / 2;
    if (i < kGuesses) {
      const float flo = __uint_as_float(lo), fhi = __uint_as_float(hi - 1);
      const float g = flo + (fhi - flo) * ((float)(k - clo) + 0.5f) / (float)(chi - clo);
      t = min(max(__float_as_uint(g), lo + 1), hi - 1);
    }
    int c = 0;
#pragma unroll
    for (int s = 0; s < S; ++s) c += __popc(__ballot_sync(kFull, e[s].x < t));
    if (c == k) {
      lo = t;
      break;
    }
    if (c < k) lo = t, clo = c;
    else hi = t, chi = c;
  }
  // entries below lo, and the first `ties` of value lo
  int at = 0;
  uint32_t far = 0;
  __syncwarp();
#pragma unroll
  for (int s = 0; s < S; ++s) {
    bool keep = e[s].x < lo;
    if (ties > 0) {
      const unsigned eq = __ballot_sync(kFull, e[s].x == lo);
      keep = keep || (e[s].x == lo && __popc(eq & lt) < ties);
      ties -= min(ties, __popc(eq));
    }
    const unsigned m = __ballot_sync(kFull, keep);
    if (keep) {
      buf[at + __popc(m & lt)] = e[s];
      far = max(far, e[s].x);
    }
    at += __popc(m);
  }
  __syncwarp();
  return __uint_as_float(__reduce_max_sync(kFull, far));
}

// Bitonic sort of the warp's `count` entries by (first, second) word; n: the
// power of two >= count, the entries between them set to the largest value.
__device__ __forceinline__ void sort_entries(uint2* buf, int count, int n, int lane) {
  for (int i = count + lane; i < n; i += 32) buf[i] = make_uint2(~0u, ~0u);
  __syncwarp();
  for (int size = 2; size <= n; size <<= 1)
    for (int gap = size >> 1; gap > 0; gap >>= 1) {
      for (int j = lane; j < n / 2; j += 32) {
        const int i = 2 * j - (j & (gap - 1));
        const uint2 a = buf[i], b = buf[i + gap];
        const bool less = b.x < a.x || (b.x == a.x && b.y < a.y);
        if (less == ((i & size) == 0)) {
          buf[i] = b;
          buf[i + gap] = a;
        }
      }
      __syncwarp();
    }
}

// Which of several photons at the k-th distance are kept.  Until a query holds k
// photons it takes what it accepts; from then on a nearer photon replaces the
// farthest one held, of equally far ones the one in the highest slot.  The photons
// of one step come in the order of their lanes.  The buffer's selection gives the
// same set unless it drops some of the photons at the k-th distance; such a query
// (one in some 600,000 of a room's) is walked once more with these slots.  The
// photons at the k-th distance that the first walk does not accept come after
// those it does, so neither walk takes them.
__device__ __forceinline__ int heap_insert(uint2* buf, int count, int k, unsigned m, float d2,
                                           unsigned pidx, float& r2, int lane, unsigned lt) {
  auto farthest = [&](uint32_t& far) {  // its slot
    uint32_t v = 0;
    int at = -1;
    for (int i = lane; i < k; i += 32)
      if (at < 0 || buf[i].x >= v) {
        v = buf[i].x;
        at = i;
      }
    far = __reduce_max_sync(kFull, v);
    return (int)__reduce_max_sync(kFull, at >= 0 && v == far ? (uint32_t)at : 0u);
  };
  uint32_t far = 0;
  int slot = 0;
  const int rank = __popc(m & lt), fill = min(__popc(m), k - count);
  if (fill > 0) {
    if (((m >> lane) & 1u) && rank < fill) buf[count + rank] = make_uint2(__float_as_uint(d2), pidx);
    __syncwarp();
    count += fill;
    for (int i = 0; i < fill; ++i) m &= m - 1u;
    if (count < k) return count;
  } else if (m == 0) {
    return count;
  }
  slot = farthest(far);
  for (; m; m &= m - 1u) {
    const int j = __ffs(m) - 1;
    const uint32_t d = __float_as_uint(__shfl_sync(kFull, d2, j));
    const unsigned p = __shfl_sync(kFull, pidx, j);
    if (d >= far) continue;
    __syncwarp();
    if (lane == 0) buf[slot] = make_uint2(d, p);
    __syncwarp();
    slot = farthest(far);
  }
  __syncwarp();
  r2 = __uint_as_float(far);
  return count;
}

// What COUNT records per query: child boxes and photons tested, normals read.
struct Work {
  uint32_t box = 0, pos = 0, nrm = 0;
};
struct Query {
  float x, y, z, nx, ny, nz;
};
__device__ __forceinline__ Query load_query(const GatherParams& P, unsigned q) {
  const float *p = P.qpos + 3 * (size_t)q, *n = P.qnrm + 3 * (size_t)q;
  return Query{__ldg(p), __ldg(p + 1), __ldg(p + 2), __ldg(n), __ldg(n + 1), __ldg(n + 2)};
}

// Walks the tree for one query.  HEAP false: accepted photons go to the buffer, of
// which the k nearest are kept; r2: the search radius, at the end the k-th distance
// if any selection was made.  HEAP true: at most k are held, and an accepted photon
// that finds them full takes the place of the farthest (heap_walk).  Returns the
// photons held, in buf.
template <int S, bool HEAP, bool COUNT>
__device__ __forceinline__ int walk(const GatherParams& P, const Query& q, float& r2, uint2* buf,
                                    uint2* stk, int lane, unsigned lt, uint32_t* tie, Work& work) {
  const int k = P.k, depth = 32 * P.nlevels;  // stack entries of a warp
  const float qx = q.x, qy = q.y, qz = q.z, nx = q.nx, ny = q.ny, nz = q.nz;
  int count = 0;
  // the root: the top level's items are its children
  int sp = 0;
  if (k > 0) {
    if (lane == 0) stk[0] = make_uint2((uint32_t)P.nlevels << 28, 0u);
    sp = 1;
  }
  __syncwarp();
  unsigned steps = 0;
  while (sp > 0) {
    if (++steps > kMaxSteps) {
      if (lane == 0) atomicOr(P.status, 1u);
      break;
    }
    --sp;
    const uint2 top = stk[sp];
    const uint32_t e = top.x;
    if (!(__uint_as_float(top.y & ~kCountBits) < r2)) {  // nothing in it can be accepted
      __syncwarp();
      continue;
    }
    if (!(e & kLeafEntry)) {
      __syncwarp();
      // inner node: lane c tests child 32 * it + c of level lv - 1
      const int cl = (int)(e >> 28) - 1;
      const uint32_t child = 32u * (e & 0x0fffffffu) + (uint32_t)lane;
      bool pass = false;
      float cd = 0.f;
      if (child < P.lvl_count[cl]) {
        const float* b = P.box + P.lvl_off[cl];
        const uint32_t pad = P.lvl_pad[cl];
        const float lx = __ldg(b + child), ly = __ldg(b + pad + child),
                    lz = __ldg(b + 2 * pad + child);
        const float hx = __ldg(b + 3 * pad + child), hy = __ldg(b + 4 * pad + child),
                    hz = __ldg(b + 5 * pad + child);
        const float gx = fmaxf(fmaxf(fs(lx, qx), fs(qx, hx)), 0.f);
        const float gy = fmaxf(fmaxf(fs(ly, qy), fs(qy, hy)), 0.f);
        const float gz = fmaxf(fmaxf(fs(lz, qz), fs(qz, hz)), 0.f);
        cd = fa(fa(fm(gx, gx), fm(gy, gy)), fm(gz, gz));
        pass = cd < r2;
      }
      const unsigned m = __ballot_sync(kFull, pass);
      if (COUNT) work.box += __popc(__ballot_sync(kFull, child < P.lvl_count[cl]));
      const int n = __popc(m);
      if (sp + n > depth) {
        if (lane == 0) atomicOr(P.status, 2u);
        break;
      }
      // Nearest child on top: the passing children are pushed farthest
      // first, so the walk visits them nearest first, the buffer fills with
      // nearer photons and the search radius, once k are kept,
      // shrinks sooner.  A child's place = the passing children farther
      // than it (equal distances: the higher lane counts as farther).
      int farther = 0;
      for (unsigned mm = m; mm; mm &= mm - 1u) {
        const int j = __ffs(mm) - 1;
        const float dj = __shfl_sync(kFull, cd, j);
        farther += (dj > cd || (dj == cd && j > (int)lane)) ? 1 : 0;
      }
      if (pass) {
        const int at = sp + farther;
        uint32_t item = ((uint32_t)cl << 28) | child;
        uint32_t cnt = 0;
        if (cl == 0) {  // a leaf: its photon range goes onto the stack
          const uint2 rng = __ldg(P.leaf + child);
          item = kLeafEntry | rng.x;
          cnt = rng.y - rng.x;
        }
        stk[at] = make_uint2(item, (__float_as_uint(cd) & ~kCountBits) | cnt);
      }
      sp += n;
      __syncwarp();
      continue;
    }
    // leaf: lane j tests photon j of the leaf; when the entry below is a
    // leaf too and both fit in the warp, lanes c0.. test its photons
    const int c0 = (int)(top.y & kCountBits);
    uint32_t b1 = 0;
    int c1 = 0;
    if (sp > 0) {
      const uint2 next = stk[sp - 1];
      const int n1 = (int)(next.y & kCountBits);
      if ((next.x & kLeafEntry) && c0 + n1 <= 32 &&
          __uint_as_float(next.y & ~kCountBits) < r2) {
        b1 = next.x & ~kLeafEntry;
        c1 = n1;
        --sp;
      }
    }
    __syncwarp();
    const unsigned pidx = lane < c0 ? (e & ~kLeafEntry) + (unsigned)lane
                                    : b1 + (unsigned)(lane - c0);
    bool acc = false;
    float d2 = 0.f;
    if (COUNT) {
      work.pos += (uint32_t)(c0 + c1);
    }
    if (lane < c0 + c1) {
      const float4 p = __ldg(P.pos4 + pidx);
      const float x = fs(qx, p.x), y = fs(qy, p.y), z = fs(qz, p.z);
      d2 = fa(fa(fm(x, x), fm(y, y)), fm(z, z));
      acc = d2 < r2;
      if (acc && !P.ignore_normal) {
        const float4 pn = __ldg(P.nrm4 + pidx);
        acc = (pn.x == nx) && (pn.y == ny) && (pn.z == nz);
      }
    }
    if (COUNT && !P.ignore_normal)
      work.nrm += __popc(__ballot_sync(kFull, lane < c0 + c1 && d2 < r2));
    const unsigned m = __ballot_sync(kFull, acc);
    if (HEAP) {
      count = heap_insert(buf, count, k, m, d2, pidx, r2, lane, lt);
      continue;
    }
    if (acc) buf[count + __popc(m & lt)] = make_uint2(__float_as_uint(d2), pidx);
    count += __popc(m);
    __syncwarp();
    if (count > P.full) {
      r2 = keep_nearest<S>(buf, count, k, lane, lt, tie);
      count = k;
    }
  }
  if (!HEAP && count > k) {
    r2 = keep_nearest<S>(buf, count, k, lane, lt, tie);
    count = k;
  }
  return count;
}

// Rare, and kept out of the kernel's own code and registers.
__device__ __noinline__ int heap_walk(const GatherParams& P, unsigned index, uint2* buf, uint2* stk) {
  const int lane = threadIdx.x & 31;
  const Query q = load_query(P, index);
  float r2 = P.r2max;
  Work work;
  return walk<1, true, false>(P, q, r2, buf, stk, lane, (1u << lane) - 1u, nullptr, work);
}

// COUNT: also records per query the work behind the roofline's bytes:
// visits[4q] child boxes tested (24 bytes each), [4q+1] photons tested (a
// 16-byte position each), [4q+2] normals read (16 bytes each), [4q+3]
// photons found (their 16-byte power is read by the estimate).
template <int S, bool NEAREST, bool COUNT = false>
__global__ void __launch_bounds__(256) gather_kernel(const __grid_constant__ GatherParams P) {
  constexpr int kCap = 32 * S;  // candidates a warp holds: k <= kCap - 32
  // per warp: candidates; stack entries, their squared distances, and a leaf
  // entry's photon count
  __shared__ uint2 s_buf[kWarpsPerBlock][kCap];
  __shared__ uint32_t s_tie[kWarpsPerBlock];  // the distance of photons dropped at the k-th place
  extern __shared__ uint2 s_dyn[];
  const int wib = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const int k = P.k;
  uint2* stk = s_dyn + wib * 32 * P.nlevels;
  uint2* buf = s_buf[wib];
  // Each warp takes P.chunk queries at a time from the launch's queue head, so
  // every warp stays busy until the queue is empty (a fixed share per warp left
  // a fifth of the warp slots idle at the end).  The head overshoots nq by at
  // most a chunk per warp: nq < 2^31 keeps it below 2^32.
  unsigned q = 0, qend = 0;
  for (;;) {
    if (q == qend) {
      unsigned b = P.nq;
      if (P.chunk) {
        if (lane == 0) b = atomicAdd(P.counter, P.chunk);
        b = __shfl_sync(kFull, b, 0);
      } else if (qend == 0) {
        b = blockIdx.x * kWarpsPerBlock + wib;
      }
      if (b >= P.nq) break;
      q = b;
      qend = min(b + max(P.chunk, 1u), P.nq);
    }
    const Query query = load_query(P, q);
    if (lane == 0) s_tie[wib] = ~0u;
    float r2 = P.r2max;
    Work work;
    int count = walk<S, false, COUNT>(P, query, r2, buf, stk, lane, lt, &s_tie[wib], work);
    __syncwarp();
    if (count == k && s_tie[wib] == __float_as_uint(r2)) count = heap_walk(P, q, buf, stk);
    __syncwarp();

    if (NEAREST) {
      // by distance, then by the photon's index
      for (int i = lane; i < count; i += 32)
        buf[i].y = (uint32_t)__float_as_int(__ldg(&P.pos4[buf[i].y].w));
      int n = 2;
      while (n < count) n <<= 1;
      sort_entries(buf, count, n, lane);
      for (int p = lane; p < k; p += 32) {
        const uint2 c = p < count ? buf[p] : make_uint2(0u, ~0u);
        P.idx[(size_t)q * k + p] = (int32_t)c.y;
        P.d2[(size_t)q * k + p] = __uint_as_float(c.x);
      }
      if (lane == 0) P.count[q] = count;
      __syncwarp();
    } else {
      float R = 0.f, G = 0.f, B = 0.f;
      if (count > 0) {
        float r = 0.f;
        if (P.caustic) {
          uint32_t far = 0;
          for (int i = lane; i < count; i += 32) far = max(far, buf[i].x);
          r = __uint_as_float(__reduce_max_sync(kFull, far));
        }
        for (int i = lane; i < count; i += 32) {
          const uint2 c = buf[i];
          const float d = __uint_as_float(c.x);
          const float w = P.caustic ? __fdiv_rn(fs(r, d), d) : 1.0f;
          const float4 pw = __ldg(P.pow4 + c.y);
          R = fa(R, fm(pw.x, w));
          G = fa(G, fm(pw.y, w));
          B = fa(B, fm(pw.z, w));
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
          R += __shfl_xor_sync(kFull, R, off);
          G += __shfl_xor_sync(kFull, G, off);
          B += __shfl_xor_sync(kFull, B, off);
        }
        if (P.caustic) {
          const float dens = __fdiv_rn((float)k, fm(fm(3.14159f, r), r));
          R = fm(R, dens);
          G = fm(G, dens);
          B = fm(B, dens);
        }
      }
      if (lane == 0) {
        P.rgb[3 * (size_t)q] = R;
        P.rgb[3 * (size_t)q + 1] = G;
        P.rgb[3 * (size_t)q + 2] = B;
      }
      __syncwarp();
    }
    if (COUNT && lane == 0) {
      P.visits[4 * (size_t)q] = work.box;
      P.visits[4 * (size_t)q + 1] = work.pos;
      P.visits[4 * (size_t)q + 2] = work.nrm;
      P.visits[4 * (size_t)q + 3] = (uint32_t)count;
    }
    ++q;
  }
}

template <bool NEAREST, bool COUNT = false>
int launch_gather(const DevPhotonMap& m, const float* qpos, const float* qnrm, size_t nq, int k,
                  float max_dist, int flags, float* rgb, int32_t* idx, float* d2, int32_t* count,
                  cudaStream_t s, uint32_t* visits = nullptr) {
  if (nq == 0) return 0;
  GatherParams p;
  p.box = m.d_box;
  p.leaf = reinterpret_cast<const uint2*>(m.d_leaf);
  p.nlevels = m.nlevels;
  for (int l = 0; l < kPhotonMaxLevels; ++l) {
    p.lvl_count[l] = m.lvl_count[l];
    p.lvl_off[l] = m.lvl_off[l];
    p.lvl_pad[l] = m.lvl_pad[l];
  }
  p.pos4 = reinterpret_cast<const float4*>(m.d_pos4);
  p.nrm4 = reinterpret_cast<const float4*>(m.d_nrm4);
  p.pow4 = reinterpret_cast<const float4*>(m.d_pow4);
  p.qpos = qpos;
  p.qnrm = qnrm;
  p.rgb = rgb;
  p.idx = idx;
  p.d2 = d2;
  p.count = count;
  p.visits = visits;
  p.status = m.d_status;
  const uint32_t slot = __atomic_fetch_add(const_cast<uint32_t*>(&m.counter_seq), 1u,
                                           __ATOMIC_RELAXED) % kGatherSlots;
  p.counter = m.d_counter + slot;
  p.nq = (unsigned)nq;
  p.k = m.n == 0 ? 0 : k;
  p.r2max = max_dist * max_dist;  // maxDistance*maxDistance in FP32 (PhotonMap.cpp:89)
  p.ignore_normal = (flags & ENC_GATHER_IGNORE_NORMAL) ? 1 : 0;
  p.caustic = m.caustic;
  int S = 0;
  void (*kern)(GatherParams) = nullptr;
  if (k <= 16) S = 2, kern = gather_kernel<2, NEAREST, COUNT>;
  else if (k <= 32) S = 3, kern = gather_kernel<3, NEAREST, COUNT>;
  else if (k <= 64) S = 4, kern = gather_kernel<4, NEAREST, COUNT>;
  else if (k <= 128) S = 6, kern = gather_kernel<6, NEAREST, COUNT>;
  else S = 10, kern = gather_kernel<10, NEAREST, COUNT>;
  p.full = std::min(32 * S - 32, k + std::max(16, 3 * k / 4));
  const size_t smem = (size_t)kWarpsPerBlock * 32 * m.nlevels * sizeof(uint2);
  // One resident wave of persistent warps (the register count allows 5
  // blocks of 256 threads per SM): a larger grid would only queue blocks
  // that find the query queue empty.
  int sms = 148, per_sm = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, m.device);
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 256, smem);
  if (e != cudaSuccess) return (int)e;
  if (per_sm < 1) per_sm = 1;
  const unsigned need = (unsigned)((nq + kWarpsPerBlock - 1) / kWarpsPerBlock);
  unsigned grid = (unsigned)sms * (unsigned)per_sm;
  const size_t warps = (size_t)grid * kWarpsPerBlock;
  if (nq <= warps) {
    p.chunk = 0;  // no more queries than warps: no queue
    grid = need;
  } else {
    p.chunk = (unsigned)std::max<size_t>(1, std::min<size_t>(kQueryChunk, nq / (4 * warps)));
    e = cudaMemsetAsync(p.counter, 0, sizeof(uint32_t), s);
    if (e != cudaSuccess) return (int)e;
  }
  kern<<<grid, 256, smem, s>>>(p);
  return (int)cudaGetLastError();
}

}  // namespace

int launch_radiance(const DevPhotonMap& m, const float* d_qpos, const float* d_qnrm, size_t nq,
                    int k, float max_dist, int flags, float* d_rgb, void* stream) {
  return launch_gather<false>(m, d_qpos, d_qnrm, nq, k, max_dist, flags, d_rgb, nullptr, nullptr,
                              nullptr, static_cast<cudaStream_t>(stream));
}

int launch_radiance_counted(const DevPhotonMap& m, const float* d_qpos, const float* d_qnrm,
                            size_t nq, int k, float max_dist, int flags, float* d_rgb,
                            uint32_t* d_visits, void* stream) {
  return launch_gather<false, true>(m, d_qpos, d_qnrm, nq, k, max_dist, flags, d_rgb, nullptr,
                                    nullptr, nullptr, static_cast<cudaStream_t>(stream), d_visits);
}

int launch_nearest(const DevPhotonMap& m, const float* d_qpos, const float* d_qnrm, size_t nq,
                   int k, float max_dist, int flags, int32_t* d_idx, float* d_d2,
                   int32_t* d_count, void* stream) {
  return launch_gather<true>(m, d_qpos, d_qnrm, nq, k, max_dist, flags, nullptr, d_idx, d_d2,
                             d_count, static_cast<cudaStream_t>(stream));
}

}  // namespace enc
