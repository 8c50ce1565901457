// Ray traversal kernels for sm_100a.
//
//  * wbvh_trace<W, CLAMP, ANY, COUNT, MULTI, LANE, ORD, WAIT>: persistent warps
//    over the quantised wide BVH.  Each warp takes rays from a global atomic queue in
//    chunks and hands them to idle lanes as lanes finish (no lane waits for
//    the slowest ray of a batch).  The traversal stack lives in shared
//    memory, one column per thread.  A visited node continues with its first
//    hit internal child; the others stay on the stack as one group entry.
//    The triangles of its hit leaves are tested in the same step, by the whole
//    warp together (all lanes' triangles, one per lane per round); with LANE by
//    each lane in turn.  Width 8 orders
//    children by octant (the builder places each child in the slot of its
//    octant, so slot k ^ octm for k = 0..7 is roughly front to back for a ray
//    with direction sign bits octm); widths 2 and 4 sort hit children by
//    entry distance.  MULTI launches trace many scenes' batches at once; ORD
//    takes the rays in a given order; WAIT lets lanes at leaves wait for a fuller
//    triangle round.
//  * wbvh_few<CLAMP, ANY>: small batches at width 8, eight lanes per ray.
//  * kd_trace<CLAMP>: the reference's kd-tree walk (Kdtree.cpp:682-784), one
//    lane per ray with the leaves' items tested by the whole warp, over the
//    flattened kd layout.  Bit-exact parity mode.
//
// The triangle test follows TrianglePrim::intersect (TrianglePrim.cpp:204-248)
// operation for operation: every product and sum is a separately rounded FP32
// operation (__fmul_rn / __fadd_rn / __fsub_rn are never contracted into FMA),
// 1/det is an IEEE division, and with CLAMP the Cross() components with
// |c| < 0.001 are set to zero as Vector3::ClampfloatoZero does
// (Vector3.h:148-161, Vector3.cpp:126-140).
//
// Every loop is bounded: a ray that exceeds kMaxSteps work items, or would
// overflow its stack, is stopped, reported as a miss, and sets a bit in the
// accelerator's status word, which the host turns into ENC_ERR_WATCHDOG.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>

#include "engine.h"

// Resident 128-thread blocks per SM that each kernel's register budget is
// fitted to (also the default grid: SMs x this).  The closest-hit kernel
// tests triangles cooperatively across the warp (below).  At 9 blocks it fits
// 56 registers without spilling and ran 1.7 % faster than at 8 (64
// registers) on the 2M-triangle heightfield workload; at 10 blocks (48
// registers) it spills 42 bytes and lost 8 %.  The multi-scene form keeps 8
// blocks: at 9 it spills 78 bytes.  The any-hit kernel has no spill at 9
// either; 1.5M shadow rays in 100,000 random triangles: 667 us, 665 at 8 and 715
// at 10, and 4M over the heightfield 713, 737 and 744.  The per-lane
// closest-hit form, which the host-buffer pipeline runs beside its copies,
// keeps 10 (at 9 the pipeline measured about 1 % slower).
constexpr int kBlocksClosest = 9;
constexpr int kBlocksMulti = 8;
constexpr int kBlocksAny = 9;
constexpr int kBlocksLane = 10;

namespace enc {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr unsigned kMaxSteps = 1u << 22;
constexpr uint32_t kStatusWatchdog = 1u;
constexpr uint32_t kStatusStack = 2u;
constexpr uint32_t kStatusBounds = 4u;

__device__ __forceinline__ float fm(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fa(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fs(float a, float b) { return __fsub_rn(a, b); }

// ClampfloatoZero: (-ENC_EPSILON < x && x < ENC_EPSILON) with the double
// constant 0.001; for a float x this is the same comparison against 0.001f.
__device__ __forceinline__ float clamp_eps(float x) {
  return (x > -0.001f && x < 0.001f) ? 0.0f : x;
}

// Dot(v1, v2) = v1[0]*v2[0] + v1[1]*v2[1] + v1[2]*v2[2], left to right.
__device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by, float bz) {
  return fa(fa(fm(ax, bx), fm(ay, by)), fm(az, bz));
}

// The reference predicate.  a/b/c: the three float4 of a DevTri.
template <bool CLAMP>
__device__ __forceinline__ bool tri_test(const float4 a, const float4 b, const float4 c, float ox,
                                         float oy, float oz, float dx, float dy, float dz,
                                         float tmin, float& t, float& alpha, float& beta) {
  const float e1x = a.w, e1y = b.x, e1z = b.y;
  const float e2x = b.z, e2y = b.w, e2z = c.x;
  // pvec = Cross(dir, edge2)
  float px = fs(fm(dy, e2z), fm(dz, e2y));
  float py = -fs(fm(dx, e2z), fm(dz, e2x));
  float pz = fs(fm(dx, e2y), fm(dy, e2x));
  if (CLAMP) {
    px = clamp_eps(px);
    py = clamp_eps(py);
    pz = clamp_eps(pz);
  }
  const float invdet = __fdiv_rn(1.0f, dot3(e1x, e1y, e1z, px, py, pz));
  // svec = Vector3(v0, origin) = origin - v0
  const float sx = fs(ox, a.x), sy = fs(oy, a.y), sz = fs(oz, a.z);
  // qvec = Cross(svec, edge1)
  float qx = fs(fm(sy, e1z), fm(sz, e1y));
  float qy = -fs(fm(sx, e1z), fm(sz, e1x));
  float qz = fs(fm(sx, e1y), fm(sy, e1x));
  if (CLAMP) {
    qx = clamp_eps(qx);
    qy = clamp_eps(qy);
    qz = clamp_eps(qz);
  }
  alpha = fm(dot3(sx, sy, sz, px, py, pz), invdet);
  beta = fm(dot3(dx, dy, dz, qx, qy, qz), invdet);
  t = fm(dot3(e2x, e2y, e2z, qx, qy, qz), invdet);
  return (alpha >= 0.0f) && (beta >= 0.0f) && (fa(alpha, beta) <= 1.0f) && (t > tmin);
}

// A float's bits made monotone as an unsigned integer (negative values
// below positive ones, order kept within each sign), and back.
__device__ __forceinline__ uint32_t order_key(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float from_order_key(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

struct TraceParams {
  const uint8_t* nodes;
  const float4* tris;  // 3 per triangle
  const float4* rays;  // 2 per ray
  const uint32_t* order;  // null, or: queue index q traces ray order[q] (binned batches)
  void* out;           // enc_hit* (closest) or uint8_t* (any)
  uint32_t* visits;    // COUNT: 2 per ray
  unsigned* counter;
  uint32_t* status;
  unsigned nrays;
  unsigned nnodes;
  unsigned ntris;
  int stack_depth;
  int chunk;
  unsigned share;  // > 0 (at most 32): warp w traces rays [w * share, (w + 1) * share) and
                   // reads no queue
  // multi-scene launches (MULTI = true): per-batch scene and buffers
  const SceneDesc* scenes;
  const BatchDesc* batches;
  const uint32_t* starts;  // nbatches + 1 chunk-aligned queue offsets
  unsigned nbatches;
  uint32_t* batch_status;  // MULTI: one status word per batch, or null (all in *status)
};

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

__device__ __forceinline__ uint32_t byte_of(const uint4* w, int off) {
  const uint32_t* u = reinterpret_cast<const uint32_t*>(w);
  return (u[off >> 2] >> (8 * (off & 3))) & 0xffu;
}

// An 8-bit quantised coordinate as a float: the byte placed under the
// exponent of 2^23 gives 2^23 + q exactly; subtracting 2^23 is exact.
__device__ __forceinline__ float u8f(uint32_t q) {
  return __uint_as_float(0x4B000000u | q) - 8388608.0f;
}

// Box tests use a reciprocal with |d| floored at 1e-20 so that a zero
// direction component (the reference's Normalize clamps small ones to
// exactly 0) gives finite slab distances instead of 0 * inf = NaN,
// which would leave that axis unconstrained.  The triangle predicate
// keeps the exact direction.
// The hardware reciprocal (rcp.approx, within 1 ulp) is enough here:
// an error of an ulp scales one axis's slab distances by 1 +- 2^-23,
// far inside the 1e-5 padding that keeps every accepted hit point off
// its box's faces, and it saves an IEEE division per axis each time a
// lane takes a new ray (measured +2.4 % closest, +3 % any hit).
__device__ __forceinline__ float slab_rcp(float d) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(fabsf(d) > 1e-20f ? d : copysignf(1e-20f, d)));
  return r;
}

template <int W>
struct NodeWords {
  static constexpr int N = WNodeLayout<W>::kBytes / 16;
  uint4 w[N];
};

constexpr uint32_t kNoItem = 0xffffffffu;

// Packed FP32 pairs (sm_100 `add/sub/mul/fma.rn.f32x2`): two floats per
// instruction, each half rounded exactly as the scalar operation, so results
// are bit-identical to the scalar form.  The width-8 slab test computes its
// 48 plane distances as 24 pairs (measured +2 % closest hit and +5 % any hit
// on the 2M-triangle heightfield, identical hits); kPairs = false keeps the
// scalar form.
#ifndef ENC_F32X2
#define ENC_F32X2 1
#endif
#ifndef ENC_GROUP_BOUND
#define ENC_GROUP_BOUND 0
#endif
// Width 8, closest hit: the stack group's lower bound (the smallest entry
// distance among the node's hit internal children) includes the child the
// walk continues into, and the hit found under that child is rarely nearer
// than its entry, so a popped group was culled by it 0.0002 times per ray on
// the 2M-triangle heightfield batch.  Without it such a group's node is
// visited and every child fails the box test against the same closest hit
// (so the hits are identical) and the per-child bound work is saved.
constexpr bool kGroupBound = ENC_GROUP_BOUND != 0;
constexpr bool kPairs = ENC_F32X2 != 0;

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long sub2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b,
                                                   unsigned long long c) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}


// L2 eviction priorities: rays are read once and hits written once, so they
// go in as evict_first, and the nodes, read by every ray, as evict_last; the
// streaming data then displaces less of the node and triangle working set
// (about the L2's size on the 2M-triangle heightfield).  +0.36 % for the
// cooperative closest-hit kernel, identical hits.
__device__ __forceinline__ uint64_t l2_policy_first() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ uint64_t l2_policy_last() {
  uint64_t p;
  asm("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
  return p;
}
__device__ __forceinline__ float4 ldg_hint(const float4* a, uint64_t pol) {
  float4 v;
  asm("ld.global.nc.L2::cache_hint.v4.f32 {%0,%1,%2,%3}, [%4], %5;"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(a), "l"(pol));
  return v;
}
__device__ __forceinline__ uint4 ldg_hint_u(const uint4* a, uint64_t pol) {
  uint4 v;
  asm("ld.global.nc.L2::cache_hint.v4.u32 {%0,%1,%2,%3}, [%4], %5;"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(a), "l"(pol));
  return v;
}
__device__ __forceinline__ void stg_hint(int4* a, int4 v, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.v4.s32 [%0], {%1,%2,%3,%4}, %5;" ::"l"(a), "r"(v.x),
               "r"(v.y), "r"(v.z), "r"(v.w), "l"(pol)
               : "memory");
}

template <int W>
__device__ __forceinline__ void sort_net(float (&k)[W], uint32_t (&v)[W]);

#define ENC_CSWAP(i, j)                   \
  {                                       \
    if (k[j] < k[i]) {                    \
      float tk = k[i];                    \
      k[i] = k[j];                        \
      k[j] = tk;                          \
      uint32_t tv = v[i];                 \
      v[i] = v[j];                        \
      v[j] = tv;                          \
    }                                     \
  }

template <>
__device__ __forceinline__ void sort_net<2>(float (&k)[2], uint32_t (&v)[2]) {
  ENC_CSWAP(0, 1);
}
template <>
__device__ __forceinline__ void sort_net<4>(float (&k)[4], uint32_t (&v)[4]) {
  ENC_CSWAP(0, 1);
  ENC_CSWAP(2, 3);
  ENC_CSWAP(0, 2);
  ENC_CSWAP(1, 3);
  ENC_CSWAP(1, 2);
}
#undef ENC_CSWAP

template <int W, bool CLAMP, bool ANY, bool COUNT, bool MULTI = false, bool LANE = false,
          bool ORD = false, bool WAIT = false>
__global__ void __launch_bounds__(128, ANY    ? kBlocksAny
                                      : LANE ? kBlocksLane
                                             : (MULTI ? kBlocksMulti : kBlocksClosest))
    wbvh_trace(TraceParams P) {
  using L = WNodeLayout<W>;
  // Stack of node groups: one entry per visited node that still has hit
  // internal children, so the depth never exceeds the tree depth.
  //   W == 8: x = child_base, y = remaining hit children as bits k in
  //           octant order (slot = k ^ octm; any hit: slot = k) | internal-slot
  //           mask << 8;
  //           lb = smallest entry distance among the group's hit children.
  //   W < 8:  x = child_base, y = ranks of the remaining children sorted by
  //           entry distance (3 bits each, nearest first) | count << 24;
  //           lb = entry distance of the nearest remaining child.
  // lb is a lower bound for every child still in the group, so a group
  // whose lb exceeds the closest hit so far is dropped whole.
  //   Width-8 entries carry lb in the top 16 bits of y (the float's high
  //   half: rounded toward zero, so never above lb for lb >= 0; a negative
  //   lb is stored as -inf), which keeps an entry at 8 bytes of shared
  //   memory and leaves more of the SM's L1 to node and triangle loads.
  constexpr bool kCompact = W == 8;
  extern __shared__ uint2 s_stack[];
  // The triangles of the lanes' hit leaves are tested as one warp (see below);
  // closest hit with LANE keeps one loop per lane.  Any hit, whose lanes wait
  // for one another in that loop just the same: 811 -> 667 us for 1.5M shadow
  // rays in 100,000 random triangles, half of them blocked, and 801 -> 713 us for
  // 4M over the 2M-triangle heightfield, where few are.
  constexpr bool kCoop = !LANE;
  static_assert(!(ANY && LANE), "any hit has no per-lane form");
  // Any hit stops at the first hit and culls nothing by distance, so its result
  // does not depend on the order of the children; it takes them in slot order
  // and saves the octant permutation (30,000 rays: 96 -> 88 us, 4M: 713 -> 701).
  constexpr bool kOctants = !ANY;
  // Idle lanes a warp waits for before it refills them.  A refill runs some 60
  // instructions for the few lanes that ended in a step (three of 32, at ten
  // visits per ray), so waiting for one more costs less than it saves.  At 1 / 2
  // / 4 / 6 / 8 / 12: the heightfield's 4.18M rays 1,163 / 1,159 / 1,141 / 1,138 /
  // 1,146 / 1,168 us, 1M eye rays on 10,000 triangles 344 / 343 / 342 / 346 / 353 /
  // 371, 16 scenes in one launch 1,157 / 1,143 / 1,134 / 1,143 / 1,160 / 1,211, the
  // shadow rays above 670 / 666 / 663 / 668 / 679 / 703.
  constexpr int kRefill = LANE ? 1 : 4;
  // With WAIT, lanes that stand at leaves wait for their triangle round until
  // kWait of them do, while the others walk on: a round costs about as much as
  // a node visit and listed 10 items of 32.  A lane never walks past a leaf it has
  // not tested, so its walk is the same.  Once the queue is empty no lane waits,
  // for the launch then lasts as long as its longest rays.  At 1 / 3 / 4 / 5 / 6 / 8
  // / 10 / 12 lanes: the heightfield's 4.18M rays 1,155 / 1,138 / 1,116 / 1,099 /
  // 1,089 / 1,084 / 1,094 / 1,119 us (1,142 without WAIT), 4M eye rays on 10,000
  // triangles 1,096 / 1,111 / 1,095 / 1,080 / 1,070 / 1,060 / 1,065 / 1,080 (1,083), 16
  // scenes in one launch 1,136 / 1,147 / 1,135 / 1,124 / 1,115 / 1,105 / 1,108 / 1,131
  // (1,135); any hit at 4 / 6 / 8 / 12 lanes: 2M rays over a field 298 / - / 286 / 290
  // (305 without), 2M on 10,000 triangles - / 723 / 714 / - (721).  The step asks only
  // how many lanes are at leaves: a second ballot, for whether any other walks, took
  // the heightfield's rays 1,079 us (1,066 now) and the 16 scenes 1,100 (1,095).
  static_assert(!WAIT || kCoop, "the per-lane form has no triangle rounds");
  constexpr int kWait = 8;
  static_assert(kWait + kRefill <= 32, "a warp that waits has lanes that walk");
  // the per-lane form keeps the group bound (without it ptxas spills more)
  constexpr bool kBound = kGroupBound || LANE;
  // L2 priorities in the single-scene cooperative closest-hit form only: in
  // any hit they measured 1 % slower, and in the per-lane form, which the
  // host-buffer pipeline runs, the evict_first hits left L2 before their copy
  // out (2 %); the multi-scene form, whose hits the server copies out after
  // each launch, keeps plain loads and stores too
  constexpr bool kL2Hints = kCoop && !MULTI && !ANY;
  __shared__ uint32_t s_coop_tri[kCoop ? 128 : 1];
  __shared__ uint32_t s_coop_own[kCoop ? 128 : 1];
  __shared__ unsigned long long s_coop_key[kCoop ? 128 : 1];
  __shared__ float2 s_coop_uv[kCoop ? 128 : 1];
  __shared__ int s_coop_cnt[kCoop ? 4 : 1];  // per warp: items listed this round
  // Each lane's ray, its reciprocal direction and sign bits, stored when the
  // lane takes the ray: the rounds' workers read their owners' rays here, and
  // with kRayShared the lane itself rereads them at every node instead of
  // holding eleven registers across the traversal loop.
  constexpr bool kRayShared = kCoop;
  __shared__ float4 s_ray[kCoop ? 384 : 1];
  const int B = blockDim.x;
  uint2* stk = s_stack + threadIdx.x;  // entry i at stk[i * B]
  float* slb = reinterpret_cast<float*>(s_stack + (size_t)P.stack_depth * B) + threadIdx.x;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned lt = lanemask_lt();

  // Warp-private ray pool [pool_next, pool_end), refilled in chunks.
  unsigned pool_next = 0, pool_end = 0;
  bool exhausted = false;
  // Binned batches: lane j holds order[pool_base + j] of the current chunk,
  // loaded once when the chunk is taken (one coalesced load per chunk instead
  // of a dependent load per refill); chunks above 32 rays read the rest
  // directly.
  // binned batches (closest hit only): a separate instantiation, so the plain
  // launch carries none of the order handling
  constexpr bool kOrdered = ORD && !MULTI && !ANY;
  unsigned pool_base = 0, ord_reg = 0;
  if (!MULTI && P.share) {
    // a batch that fits the grid at once: a fixed share of rays per warp
    const unsigned w = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    pool_base = pool_next = min(w * P.share, P.nrays);
    pool_end = min(pool_next + P.share, P.nrays);
    if (kOrdered && P.order != nullptr && pool_base + lane < pool_end)
      ord_reg = __ldg(P.order + pool_base + lane);
  }

  int ray = -1;
  float ox = 0, oy = 0, oz = 0, dx = 0, dy = 0, dz = 0, ix = 0, iy = 0, iz = 0, tmin = 0, tmax = 0;
  float best_t = 0, bu = 0, bv = 0;
  int best_id = -1;
  int sp = 0;
  uint32_t node = kNoItem;
  uint32_t octm = 0;  // direction sign bits: bit a set = negative along axis a
  unsigned steps = 0;
  uint32_t nvis = 0, ntest = 0;
  // The scene a lane's ray belongs to (MULTI: per batch, else the launch's).
  const uint8_t* l_nodes = P.nodes;
  const float4* l_tris = P.tris;
  unsigned l_nnodes = P.nnodes, l_ntris = P.ntris;
  void* l_out = P.out;
  unsigned l_idx = 0;          // index of the ray in its output array
  unsigned pool_batch = 0;     // MULTI: batch of the current pool
  uint32_t tmask = 0, tbase = 0;  // untested triangles of the lane's node
  uint32_t* l_status = P.status;  // the status word of the lane's ray (MULTI: its batch's)

  while (true) {
    // ---- refill idle lanes from the warp pool --------------------------
    unsigned need = __ballot_sync(kFull, ray < 0);
    if (__popc(need) < kRefill) need = 0;
    while (need && !exhausted) {
      if (pool_next >= pool_end) {
        if (!MULTI && P.share) {  // the warp's share is all it takes
          exhausted = true;
          break;
        }
        unsigned b = 0;
        if (lane == 0) {
          b = atomicAdd(P.counter, (unsigned)P.chunk);
          // Rays are read once, so every refill would wait on DRAM: bring the
          // chunk one full grid of claims ahead into L2 now (one bulk
          // prefetch; the warp that claims it later finds it in L2).  With the
          // round's atomic listing below: +1.7 % on the 2M-triangle
          // heightfield batch (the listing alone measured -1.2 %).
          if (!MULTI && !kOrdered) {
            const unsigned ahead = gridDim.x * (blockDim.x >> 5) * (unsigned)P.chunk;
            const unsigned pb = b + ahead;
            if (pb > b && pb < P.nrays) {
              const unsigned cnt = min((unsigned)P.chunk, P.nrays - pb);
              asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(P.rays + 2 * (size_t)pb),
                           "r"(cnt * 32u)
                           : "memory");
            }
          }
        }
        b = __shfl_sync(kFull, b, 0);
        if (b >= P.nrays) {
          exhausted = true;
          break;
        }
        pool_next = b;
        pool_base = b;
        if (kOrdered && P.order != nullptr && b + lane < P.nrays) ord_reg = __ldg(P.order + b + lane);
        if constexpr (MULTI) {
          // batch = last start <= b (starts are chunk-aligned, so the whole
          // chunk lies in it); its real rays end before the padding
          unsigned lo = 0, hi = P.nbatches;
          while (hi - lo > 1) {
            const unsigned mid = (lo + hi) >> 1;
            if (__ldg(P.starts + mid) <= b) lo = mid;
            else hi = mid;
          }
          pool_batch = lo;
          pool_end = min(b + (unsigned)P.chunk, __ldg(P.starts + lo) + P.batches[lo].nrays);
        } else {
          pool_end = min(b + (unsigned)P.chunk, P.nrays);
        }
      }
      const unsigned avail = pool_end > pool_next ? pool_end - pool_next : 0u;
      const unsigned rank = __popc(need & lt);
      const unsigned qoff = pool_next - pool_base + rank;  // offset of this lane's ray in the chunk
      const unsigned via = kOrdered ? __shfl_sync(kFull, ord_reg, qoff & 31u) : 0u;
      bool bad_order = false;
      if (((need >> lane) & 1u) && rank < avail) {
        ray = (int)(pool_next + rank);
        if (kOrdered && P.order != nullptr) {
          const unsigned oi = qoff < 32u ? via : __ldg(P.order + pool_next + rank);
          // an order entry outside the batch is skipped and reported
          bad_order = oi >= P.nrays;
          ray = bad_order ? -1 : (int)oi;
        }
      }
      if (bad_order) atomicOr(l_status, kStatusBounds);
      if (ray >= 0 && ((need >> lane) & 1u) && rank < avail) {
        const float4* rp;
        if constexpr (MULTI) {
          const BatchDesc& bd = P.batches[pool_batch];
          const SceneDesc& sd = P.scenes[bd.scene];
          l_idx = (unsigned)ray - bd.start;
          l_out = bd.out;
          l_nodes = sd.nodes;
          l_tris = reinterpret_cast<const float4*>(sd.tris);
          l_nnodes = sd.nnodes;
          l_ntris = sd.ntris;
          if (P.batch_status) l_status = P.batch_status + pool_batch;
          rp = reinterpret_cast<const float4*>(bd.rays) + 2 * (size_t)l_idx;
        } else {
          l_idx = (unsigned)ray;
          rp = P.rays + 2 * (size_t)ray;
        }
        const float4 r0 = kL2Hints ? ldg_hint(rp, l2_policy_first()) : __ldg(rp);
        const float4 r1 = kL2Hints ? ldg_hint(rp + 1, l2_policy_first()) : __ldg(rp + 1);
        ox = r0.x; oy = r0.y; oz = r0.z; tmin = r0.w;
        dx = r1.x; dy = r1.y; dz = r1.z; tmax = r1.w;

        ix = slab_rcp(dx);
        iy = slab_rcp(dy);
        iz = slab_rcp(dz);
        octm = (dx < 0.f ? 1u : 0u) | (dy < 0.f ? 2u : 0u) | (dz < 0.f ? 4u : 0u);
        if (kCoop) {
          s_ray[3 * threadIdx.x] = r0;
          s_ray[3 * threadIdx.x + 1] = r1;
          s_ray[3 * threadIdx.x + 2] = make_float4(ix, iy, iz, __uint_as_float(octm));
        }
        best_t = tmax; best_id = -1; bu = 0.f; bv = 0.f;
        sp = 0;
        node = 0;  // root
        steps = 0;
        nvis = 0; ntest = 0;
      }
      const unsigned took = min(avail, (unsigned)__popc(need));
      pool_next += took;
      need = __ballot_sync(kFull, ray < 0);
    }
    if (__all_sync(kFull, ray < 0)) break;

    bool done = false;
    bool hit_any = false;
    if (!WAIT) tmask = 0;
    if (ray >= 0 && (!WAIT || tmask == 0)) {
      if (++steps > kMaxSteps) {
        atomicOr(l_status, kStatusWatchdog);
        best_id = -1;
        done = true;
      } else if (node >= l_nnodes) {
        atomicOr(l_status, kStatusBounds);
        best_id = -1;
        done = true;
      } else {
        // ---- visit one node: its hit leaves now, its hit internal children
        //      in front-to-back order (one continues, the rest become one
        //      group on the stack) ------------------------------------------
        if (COUNT) ++nvis;
        NodeWords<W> nw;
        const uint4* src = reinterpret_cast<const uint4*>(l_nodes + (size_t)node * L::kBytes);
#pragma unroll
        for (int i = 0; i < NodeWords<W>::N; ++i)
          nw.w[i] = kL2Hints ? ldg_hint_u(src + i, l2_policy_last()) : __ldg(src + i);
        const float px = __uint_as_float(nw.w[0].x);
        const float py = __uint_as_float(nw.w[0].y);
        const float pz = __uint_as_float(nw.w[0].z);
        const uint32_t ew = nw.w[0].w;
        const float sx = __uint_as_float((ew & 0xffu) << 23);
        const float sy = __uint_as_float(((ew >> 8) & 0xffu) << 23);
        const float sz = __uint_as_float(((ew >> 16) & 0xffu) << 23);
        const uint32_t child_base = nw.w[1].x;
        const uint32_t tri_base = nw.w[1].y;
        float vox = ox, voy = oy, voz = oz, vtmin = tmin, vix = ix, viy = iy, viz = iz;
        uint32_t voct = octm;
        if constexpr (kRayShared) {
          const float4 sa = s_ray[3 * threadIdx.x], sc = s_ray[3 * threadIdx.x + 2];
          vox = sa.x; voy = sa.y; voz = sa.z; vtmin = sa.w;
          vix = sc.x; viy = sc.y; viz = sc.z;
          voct = __float_as_uint(sc.w);
        }
        const float bx = (px - vox) * vix, by = (py - voy) * viy, bz = (pz - voz) * viz;
        const float cx = sx * vix, cy = sy * viy, cz = sz * viz;
        // Near and far planes per axis by the ray's direction sign: the
        // near plane of a child box is its lo corner for a positive
        // direction and its hi corner for a negative one.
        const bool nxs = (voct & 1u) != 0, nys = (voct & 2u) != 0, nzs = (voct & 4u) != 0;
        float key[W];
        uint32_t rnk[W];
        uint32_t trimask = 0;
        uint32_t hitk = 0;      // W == 8: hit internal children, bit k = slot k ^ voct
        float lbmin = INFINITY;  // W == 8: smallest entry distance of those
        int nh = 0;
        // Width 8: the six plane arrays are whole words (qlo x at words 8-9,
        // y 10-11, z 12-13, qhi x 14-15, y 16-17, z 18-19), so near/far are
        // chosen once per word and each byte becomes 2^23 + q with one PRMT.
        uint32_t wn[6], wf[6];
        if constexpr (W == 8) {
          const uint32_t* u = reinterpret_cast<const uint32_t*>(nw.w);
          const bool neg[3] = {nxs, nys, nzs};
#pragma unroll
          for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint32_t lo = u[8 + 2 * a + h], hi = u[14 + 2 * a + h];
              wn[2 * a + h] = neg[a] ? hi : lo;
              wf[2 * a + h] = neg[a] ? lo : hi;
            }
        }
        if constexpr (W == 8) {
          // Slab test of the eight children into a hit-slot mask; the header's
          // internal-slot mask splits it into internal and leaf hits.  Empty
          // slots hold an inverted box (lo 255, hi 0), whose near plane lies
          // beyond its far plane for either direction sign, so they never hit
          // (and a leaf entry with meta 0 would contribute no triangles).
          const uint32_t imask = ew >> 24;
          uint32_t hm = 0;
          // pairs: x and y share one pair for the near planes and one for the
          // far planes; z pairs its near and far plane
          const unsigned long long m23 = pack2(-8388608.0f, -8388608.0f);
          // (bx, by) and (cx, cy) as pairs: the node origin, the ray origin and
          // the reciprocal direction already sit in adjacent halves of their
          // 16-byte loads
          const unsigned long long vixy = pack2(vix, viy);
          const unsigned long long bxy = mul2(sub2(pack2(px, py), pack2(vox, voy)), vixy);
          const unsigned long long cxy = mul2(pack2(sx, sy), vixy);
          const unsigned long long czz = pack2(cz, cz), bzz = pack2(bz, bz);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const uint32_t sel = 0x7650u | (uint32_t)(c & 3);
            const int h = c >> 2;
            float tnx, tfx, tny, tfy, tnz, tfz;
            if constexpr (kPairs) {
              // 2^23 + q, minus 2^23, times the scaled reciprocal plus the
              // origin offset, two planes at a time
              auto q2 = [&](uint32_t a, uint32_t b) {
                return add2(pack2(__uint_as_float(__byte_perm(a, 0x4B000000u, sel)),
                                  __uint_as_float(__byte_perm(b, 0x4B000000u, sel))),
                            m23);
              };
              unpack2(fma2(q2(wn[0 + h], wn[2 + h]), cxy, bxy), tnx, tny);
              unpack2(fma2(q2(wf[0 + h], wf[2 + h]), cxy, bxy), tfx, tfy);
              unpack2(fma2(q2(wn[4 + h], wf[4 + h]), czz, bzz), tnz, tfz);
            } else {
              tnx = fmaf(__uint_as_float(__byte_perm(wn[0 + h], 0x4B000000u, sel)) - 8388608.0f, cx, bx);
              tfx = fmaf(__uint_as_float(__byte_perm(wf[0 + h], 0x4B000000u, sel)) - 8388608.0f, cx, bx);
              tny = fmaf(__uint_as_float(__byte_perm(wn[2 + h], 0x4B000000u, sel)) - 8388608.0f, cy, by);
              tfy = fmaf(__uint_as_float(__byte_perm(wf[2 + h], 0x4B000000u, sel)) - 8388608.0f, cy, by);
              tnz = fmaf(__uint_as_float(__byte_perm(wn[4 + h], 0x4B000000u, sel)) - 8388608.0f, cz, bz);
              tfz = fmaf(__uint_as_float(__byte_perm(wf[4 + h], 0x4B000000u, sel)) - 8388608.0f, cz, bz);
            }
            // sm_100's three-input max/min (NaN operands ignored, as fmaxf /
            // fminf do): +0.45 % over the two-input tree
            float tn, tf;
            {
              float m;
              asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(tnx), "f"(tny), "f"(tnz));
              tn = fmaxf(m, vtmin);
              asm("min.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(tfx), "f"(tfy), "f"(tfz));
              tf = fminf(m, best_t);
            }
            if (tn <= tf) {
              hm |= 1u << c;
              // (any hit never culls by distance, so it keeps no bound)
              if (!ANY && kBound && ((imask >> c) & 1u)) lbmin = fminf(lbmin, tn);
            }
          }
          // triangles of the hit leaves (meta = count << 5 | offset)
          // (the meta bytes are words 6 and 7 of the node, bytes 24-31; they
          // are picked by select and shift, not by indexing the node array
          // with the runtime slot c, which would move it to local memory)
          uint32_t lh = hm & ~imask;
          const uint32_t mlo = nw.w[1].z, mhi = nw.w[1].w;
          while (lh) {
            const uint32_t c = __ffs(lh) - 1;
            lh &= lh - 1;
            const uint32_t meta = (((c & 4u) ? mhi : mlo) >> ((c & 3u) * 8u)) & 0xffu;
            trimask |= ((1u << (meta >> 5)) - 1u) << (meta & 31u);
          }
          // hit internal children in octant order: bit k = slot k ^ voct
          uint32_t x = hm & imask;
          if (kOctants) {
            if (voct & 1u) x = ((x & 0x55u) << 1) | ((x >> 1) & 0x55u);
            if (voct & 2u) x = ((x & 0x33u) << 2) | ((x >> 2) & 0x33u);
            if (voct & 4u) x = ((x & 0x0fu) << 4) | ((x >> 4) & 0x0fu);
          }
          hitk = x;
        } else {
#pragma unroll
          for (int c = 0; c < W; ++c) {
            const uint32_t qlx = byte_of(nw.w, L::kQOff + 0 * W + c);
            const uint32_t qly = byte_of(nw.w, L::kQOff + 1 * W + c);
            const uint32_t qlz = byte_of(nw.w, L::kQOff + 2 * W + c);
            const uint32_t qhx = byte_of(nw.w, L::kQOff + 3 * W + c);
            const uint32_t qhy = byte_of(nw.w, L::kQOff + 4 * W + c);
            const uint32_t qhz = byte_of(nw.w, L::kQOff + 5 * W + c);
            const float tnx = fmaf(u8f(nxs ? qhx : qlx), cx, bx);
            const float tfx = fmaf(u8f(nxs ? qlx : qhx), cx, bx);
            const float tny = fmaf(u8f(nys ? qhy : qly), cy, by);
            const float tfy = fmaf(u8f(nys ? qly : qhy), cy, by);
            const float tnz = fmaf(u8f(nzs ? qhz : qlz), cz, bz);
            const float tfz = fmaf(u8f(nzs ? qlz : qhz), cz, bz);
            const float tn = fmaxf(fmaxf(tnx, tny), fmaxf(tnz, vtmin));
            const float tf = fminf(fminf(tfx, tfy), fminf(tfz, best_t));
            const uint32_t meta = byte_of(nw.w, L::kMetaOff + c);
            const bool hit = meta != 0u && tn <= tf;
            const bool leaf = meta >= 32u;
            if (hit && leaf) trimask |= ((1u << (meta >> 5)) - 1u) << (meta & 31u);
            const bool ih = hit && !leaf;
            key[c] = ih ? fminf(tn, 3.0e38f) : INFINITY;  // hits sort before the rest
            rnk[c] = meta - 1u;
            nh += ih ? 1 : 0;
          }
        }
        // ---- next node, and the group of the other hit children ----------
        if constexpr (W == 8) {
          if (hitk) {
            const uint32_t imask = ew >> 24;
            const uint32_t k = __ffs(hitk) - 1;
            const uint32_t slot = kOctants ? k ^ voct : k;
            node = child_base + __popc(imask & ((1u << slot) - 1u));
            const uint32_t rest = hitk & (hitk - 1u);
            if (rest) {
              if (sp >= P.stack_depth) {
                atomicOr(l_status, kStatusStack);
                best_id = -1;
                done = true;
                trimask = 0;
              } else {
                if constexpr (kCompact) {
                  const uint32_t lb16 =
                      (ANY || !kBound) ? 0u
                                            : (lbmin >= 0.0f ? (__float_as_uint(lbmin) >> 16) : 0xff80u);
                  stk[sp * B] = make_uint2(child_base, rest | (imask << 8) | (lb16 << 16));
                } else {
                  stk[sp * B] = make_uint2(child_base, rest | (imask << 8));
                  slb[sp * B] = lbmin;
                }
                ++sp;
              }
            }
          } else {
            node = kNoItem;
          }
        } else {
          if (nh > 0) {
            sort_net<W>(key, rnk);
            node = child_base + rnk[0];
            if (nh > 1) {
              if (sp >= P.stack_depth) {
                atomicOr(l_status, kStatusStack);
                best_id = -1;
                done = true;
                trimask = 0;
              } else {
                uint32_t packed = 0;
#pragma unroll
                for (int c = W - 1; c >= 1; --c)
                  if (c < nh) packed = (packed << 3) | (rnk[c] & 7u);
                stk[sp * B] = make_uint2(child_base, packed | ((uint32_t)(nh - 1) << 24));
                slb[sp * B] = key[1];
                ++sp;
              }
            }
          } else {
            node = kNoItem;
          }
        }
        // ---- triangles of the hit leaves ---------------------------------
        tmask = trimask;
        tbase = tri_base;
        if (kCoop) trimask = 0;  // tested below by the whole warp
        while (!kCoop && trimask) {
          const uint32_t k = __ffs(trimask) - 1;
          trimask &= trimask - 1;
          const uint32_t ti = tri_base + k;
          if (ti >= l_ntris) {
            atomicOr(l_status, kStatusBounds);
            continue;
          }
          const float4* tp = l_tris + 3 * (size_t)ti;
          const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
          if (COUNT) ++ntest;
          float t, u, v;
          if (tri_test<CLAMP>(a, b, c, ox, oy, oz, dx, dy, dz, tmin, t, u, v)) {
            const int id = __float_as_int(c.y);
            if (t < best_t || (t == best_t && id < best_id)) {
              best_t = t;
              best_id = id;
              bu = u;
              bv = v;
            }
          }
        }
      }
    }
    if constexpr (kCoop) {
    // ---- the warp tests all lanes' pending triangles together -------------
    // Each round lists up to 32 (lane, triangle) items in shared memory; lane
    // w tests item w with the owner lane's ray, and the owner's closest hit
    // is the minimum of (t, ID) over its accepted candidates, taken with a
    // 64-bit shared atomicMin on an order-preserving key (t's bits made
    // monotone, then the ID) -- the same choice as the per-lane loop's
    // "t < best_t, or equal t and a lower ID", whatever the order.
    {
      unsigned pend = __ballot_sync(kFull, tmask != 0);
      // (while the queue has rays, fewer than kRefill lanes are idle here, so with
      // fewer than kWait at leaves others still walk)
      if (WAIT && !exhausted && __popc(pend) < kWait) pend = 0;
      const unsigned wib = threadIdx.x >> 5;
      uint32_t* it_tri = s_coop_tri + wib * 32;
      uint32_t* it_own = s_coop_own + wib * 32;
      unsigned long long* key = s_coop_key + wib * 32;
      float2* uv = s_coop_uv + wib * 32;
      while (pend) {
        const int ni = __popc(tmask);
        // each lane with items claims its slots with one shared atomic (the
        // list order does not matter: the closest hit is a minimum)
        if (lane == 0) s_coop_cnt[wib] = 0;
        __syncwarp();
        const int excl = ni ? atomicAdd(&s_coop_cnt[wib], ni) : 0;
        __syncwarp();
        const int total = s_coop_cnt[wib];
        int j = 0;
        while (tmask && excl + j < 32) {
          const uint32_t k = __ffs(tmask) - 1;
          tmask &= tmask - 1;
          it_tri[excl + j] = tbase + k;
          it_own[excl + j] = lane;
          ++j;
        }
        if (COUNT) ntest += j;
        const unsigned long long mykey =
            ANY ? 1ull : ((unsigned long long)order_key(best_t) << 32) | (uint32_t)best_id;
        key[lane] = mykey;
        __syncwarp();
        const int nitems = total < 32 ? total : 32;
        const int own = (int)lane < nitems ? (int)it_own[lane] : (int)lane;
        // the owner's ray, kept in shared memory since its refill (two
        // 16-byte loads instead of seven shuffles; measured +1 %)
        const float4 wr0 = s_ray[3 * (wib * 32 + own)], wr1 = s_ray[3 * (wib * 32 + own) + 1];
        const float wox = wr0.x, woy = wr0.y, woz = wr0.z, wtmin = wr0.w;
        const float wdx = wr1.x, wdy = wr1.y, wdz = wr1.z;
        const float wlim = __shfl_sync(kFull, ANY ? tmax : best_t, own);
        const int wbid = __shfl_sync(kFull, best_id, own);
        const float4* wtris = l_tris;
        unsigned wntris = l_ntris;
        uint32_t* wstatus = P.status;
        if constexpr (MULTI) {
          const unsigned long long tp = __shfl_sync(kFull, (unsigned long long)l_tris, own);
          wtris = reinterpret_cast<const float4*>(tp);
          wntris = __shfl_sync(kFull, l_ntris, own);
          wstatus = reinterpret_cast<uint32_t*>(
              __shfl_sync(kFull, (unsigned long long)l_status, own));
        }
        bool cand = false;
        unsigned long long ckey = 0;
        float cu = 0.f, cv = 0.f;
        if ((int)lane < nitems) {
          const uint32_t ti = it_tri[lane];
          if (ti >= wntris) {
            atomicOr(wstatus, kStatusBounds);
          } else {
            const float4* tp = wtris + 3 * (size_t)ti;
            const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
            float t, u, v;
            if (tri_test<CLAMP>(a, b, c, wox, woy, woz, wdx, wdy, wdz, wtmin, t, u, v)) {
              const int id = __float_as_int(c.y);
              if (ANY) {
                if (t < wlim) key[own] = 0ull;  // any hit: the owner is done
              } else if (t < wlim || (t == wlim && id < wbid)) {
                cand = true;
                ckey = ((unsigned long long)order_key(t) << 32) | (uint32_t)id;
                cu = u;
                cv = v;
                atomicMin(&key[own], ckey);
              }
            }
          }
        }
        __syncwarp();
        if (cand && key[own] == ckey) uv[own] = make_float2(cu, cv);
        __syncwarp();
        const unsigned long long nk = key[lane];
        if (ANY) {
          if (nk == 0ull && ray >= 0) {
            hit_any = true;
            done = true;
            tmask = 0;
          }
        } else if (nk != mykey) {
          best_t = from_order_key((uint32_t)(nk >> 32));
          best_id = (int)(uint32_t)nk;
        }
        __syncwarp();
        pend = __ballot_sync(kFull, tmask != 0);
      }
    }
    }
    if (ray >= 0 && (!WAIT || tmask == 0)) {
      // ---- pop the next group child that can still matter ----------------
      if (!done && node == kNoItem) {
        while (sp > 0) {
          uint2 e;
          if constexpr (kCompact) {
            e = stk[(sp - 1) * B];
            if (!ANY && kBound && __uint_as_float(e.y & 0xffff0000u) > best_t) {
              --sp;
              continue;
            }
          } else {
            if (!ANY && slb[(sp - 1) * B] > best_t) {
              --sp;
              continue;
            }
            e = stk[(sp - 1) * B];
          }
          if constexpr (W == 8) {
            const uint32_t hk = e.y & 0xffu;
            const uint32_t k = __ffs(hk) - 1;
            uint32_t slot = k;
            if (kOctants) slot ^= kRayShared ? __float_as_uint(s_ray[3 * threadIdx.x + 2].w) : octm;
            const uint32_t imask = (e.y >> 8) & 0xffu;
            node = e.x + __popc(imask & ((1u << slot) - 1u));
            const uint32_t rest = hk & (hk - 1u);
            if (rest == 0) {
              --sp;
            } else {
              e.y = (e.y & 0xffff0000u) | rest | (imask << 8);
              stk[(sp - 1) * B] = e;
            }
          } else {
            const uint32_t cnt = e.y >> 24;
            node = e.x + (e.y & 7u);
            if (cnt <= 1) {
              --sp;
            } else {
              e.y = (((e.y & 0xffffffu) >> 3)) | ((cnt - 1) << 24);
              stk[(sp - 1) * B] = e;
            }
          }
          break;
        }
        if (node == kNoItem) done = true;
      }
      if (done) {
        if (ANY) {
          reinterpret_cast<uint8_t*>(l_out)[l_idx] = hit_any ? 1 : 0;
        } else {
          int4 h;
          h.x = best_id;
          h.y = best_id >= 0 ? __float_as_int(best_t) : 0;
          float hu = bu, hv = bv;
          if constexpr (kCoop) {
            // the round that found the hit left its barycentrics in shared memory
            const float2 w = s_coop_uv[threadIdx.x];
            hu = w.x;
            hv = w.y;
          }
          h.z = best_id >= 0 ? __float_as_int(hu) : 0;
          h.w = best_id >= 0 ? __float_as_int(hv) : 0;
          if (kL2Hints)
            stg_hint(reinterpret_cast<int4*>(l_out) + l_idx, h, l2_policy_first());
          else
            reinterpret_cast<int4*>(l_out)[l_idx] = h;
        }
        if (COUNT) {
          P.visits[2 * (size_t)ray] = nvis;
          P.visits[2 * (size_t)ray + 1] = ntest;
        }
        ray = -1;
        node = kNoItem;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Few rays: eight lanes walk one ray, one child box each.
//
// A batch that leaves most of the GPU idle takes as long as its longest ray, and
// a step of wbvh_trace costs a lone warp about 1 us: the node's load, eight slab
// tests, the triangles' load and the triangle round, one after another.  Here
// lane c of a ray's eight tests child c, then the leaf triangles that the step
// reached, eight at a time, while the next node is already on its way (which node
// that is depends on neither).  The stack and the walk are wbvh_trace's for
// width 8, child order, culling and the choice among candidates included, so the
// hits are the same bits.  777 / 5,000 eye and bounce rays in 10,000 triangles: 49
// / 66 us with a share of rays per warp, 32 / 41 us here (39 / 49 with the next
// node fetched after the triangles); 777 shadow rays 58 -> 37, four of them from
// more than 64 registers.  Prefetching the other children hit to L1 made 5,000 rays
// 2 us slower, loading the triangles ahead of the next node 4.

// Position of the r-th set bit of m (r counted from 0, r < popc(m)), by
// halving: keep the low half while it holds more than r set bits.
__device__ __forceinline__ int nth_set_bit(unsigned m, int r) {
  int pos = 0;
#pragma unroll
  for (int b = 16; b >= 1; b >>= 1) {
    const int c = __popc(m & ((1u << b) - 1u));
    if (r >= c) {
      r -= c;
      m >>= b;
      pos += b;
    }
  }
  return pos;
}

template <bool CLAMP, bool ANY>
__global__ void __launch_bounds__(128, 4) wbvh_few(TraceParams P) {
  using L = WNodeLayout<8>;
  extern __shared__ uint2 s_stack[];
  const unsigned lane = threadIdx.x & 31u, grp = lane >> 3, c = lane & 7u;
  uint2* stk = s_stack + (size_t)(threadIdx.x >> 3) * P.stack_depth;
  const unsigned q = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * P.share + grp;
  bool live = grp < P.share && q < P.nrays;
  unsigned ray = q;
  if (live && P.order) {
    ray = __ldg(P.order + q);
    if (ray >= P.nrays) {  // an order entry outside the batch: skipped and reported
      if (c == 0) atomicOr(P.status, kStatusBounds);
      live = false;
    }
  }
  float ox = 0, oy = 0, oz = 0, dx = 0, dy = 0, dz = 0, tmin = 0, tmax = 0;
  if (live) {
    const float4 r0 = __ldg(P.rays + 2 * (size_t)ray), r1 = __ldg(P.rays + 2 * (size_t)ray + 1);
    ox = r0.x; oy = r0.y; oz = r0.z; tmin = r0.w;
    dx = r1.x; dy = r1.y; dz = r1.z; tmax = r1.w;
  }
  const float ix = slab_rcp(dx), iy = slab_rcp(dy), iz = slab_rcp(dz);
  const uint32_t octm = (dx < 0.f ? 1u : 0u) | (dy < 0.f ? 2u : 0u) | (dz < 0.f ? 4u : 0u);
  // the byte of child c in the near and far plane array of each axis
  const unsigned nx = L::kQOff + (octm & 1u ? 24u : 0u) + c, fx = L::kQOff + (octm & 1u ? 0u : 24u) + c;
  const unsigned ny = L::kQOff + (octm & 2u ? 32u : 8u) + c, fy = L::kQOff + (octm & 2u ? 8u : 32u) + c;
  const unsigned nz = L::kQOff + (octm & 4u ? 40u : 16u) + c, fz = L::kQOff + (octm & 4u ? 16u : 40u) + c;
  float best_t = tmax, bu = 0.f, bv = 0.f;
  int best_id = -1;
  bool hit_any = false, lost = false;  // lost: stopped at a bound, reported as a miss
  int sp = 0;
  unsigned steps = 0;
  uint32_t node = live ? 0u : kNoItem;
  // the node to visit: its header and child c's planes
  uint4 h0 = make_uint4(0, 0, 0, 0), h1 = h0;
  uint32_t pnx = 0, pfx = 0, pny = 0, pfy = 0, pnz = 0, pfz = 0;
  auto fetch = [&]() {
    if (node == kNoItem) return;
    if (++steps > kMaxSteps || node >= P.nnodes) {
      if (c == 0) atomicOr(P.status, steps > kMaxSteps ? kStatusWatchdog : kStatusBounds);
      lost = true;
      node = kNoItem;
      return;
    }
    const uint8_t* src = P.nodes + (size_t)node * L::kBytes;
    h0 = __ldg(reinterpret_cast<const uint4*>(src));
    h1 = __ldg(reinterpret_cast<const uint4*>(src) + 1);
    pnx = __ldg(src + nx), pfx = __ldg(src + fx);
    pny = __ldg(src + ny), pfy = __ldg(src + fy);
    pnz = __ldg(src + nz), pfz = __ldg(src + fz);
  };
  fetch();

  while (__any_sync(kFull, node != kNoItem)) {
    const bool on = node != kNoItem;
    bool hit = false;
    if (on) {
      const float sx = __uint_as_float((h0.w & 0xffu) << 23);
      const float sy = __uint_as_float(((h0.w >> 8) & 0xffu) << 23);
      const float sz = __uint_as_float(((h0.w >> 16) & 0xffu) << 23);
      const float bx = (__uint_as_float(h0.x) - ox) * ix, by = (__uint_as_float(h0.y) - oy) * iy,
                  bz = (__uint_as_float(h0.z) - oz) * iz;
      const float cx = sx * ix, cy = sy * iy, cz = sz * iz;
      const float tnx = fmaf(u8f(pnx), cx, bx), tfx = fmaf(u8f(pfx), cx, bx);
      const float tny = fmaf(u8f(pny), cy, by), tfy = fmaf(u8f(pfy), cy, by);
      const float tnz = fmaf(u8f(pnz), cz, bz), tfz = fmaf(u8f(pfz), cz, bz);
      hit = fmaxf(fmaxf(tnx, tny), fmaxf(tnz, tmin)) <= fminf(fminf(tfx, tfy), fminf(tfz, best_t));
    }
    const uint32_t hm = (__ballot_sync(kFull, hit) >> (8 * grp)) & 0xffu;
    const uint32_t imask = h0.w >> 24, tri_base = h1.y;
    // the triangles of the hit leaves: lane c's leaf, then the eight together
    const uint32_t meta = ((c & 4u ? h1.w : h1.z) >> ((c & 3u) * 8u)) & 0xffu;
    uint32_t tris = hit && !((imask >> c) & 1u) ? ((1u << (meta >> 5)) - 1u) << (meta & 31u) : 0u;
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) tris |= __shfl_xor_sync(kFull, tris, d);
    // ---- the next node: the first child hit, else the deferred child pushed
    //      last.  Neither depends on the triangles (a child is culled when its
    //      box is tested), so its data is on its way while they are tested.
    uint32_t x = on ? hm & imask : 0u;
    if (!ANY) {
      if (octm & 1u) x = ((x & 0x55u) << 1) | ((x >> 1) & 0x55u);
      if (octm & 2u) x = ((x & 0x33u) << 2) | ((x >> 2) & 0x33u);
      if (octm & 4u) x = ((x & 0x0fu) << 4) | ((x >> 4) & 0x0fu);
    }
    const bool pop = on && x == 0 && sp > 0;
    const uint2 e = pop ? stk[sp - 1] : make_uint2(h1.x, x | (imask << 8));
    __syncwarp();  // all eight have read it
    if (on) {
      node = kNoItem;
      const uint32_t hk = e.y & 0xffu;
      if (hk) {
        const uint32_t k = __ffs(hk) - 1, slot = ANY ? k : k ^ octm, rest = hk & (hk - 1u);
        node = e.x + __popc((e.y >> 8) & ((1u << slot) - 1u));
        if (pop) --sp;
        if (rest && sp >= P.stack_depth) {
          if (c == 0) atomicOr(P.status, kStatusStack);
          lost = true;
          node = kNoItem;
        } else if (rest) {
          if (c == 0) stk[sp] = make_uint2(e.x, (e.y & ~0xffu) | rest);
          ++sp;
        }
      }
    }
    fetch();
    // ---- triangles, eight at a time ---------------------------------------
    while (__any_sync(kFull, tris != 0)) {
      const int n = __popc(tris);
      unsigned long long key = ~0ull;
      float u = 0.f, v = 0.f;
      if ((int)c < n) {
        const uint32_t ti = tri_base + (uint32_t)nth_set_bit(tris, (int)c);
        if (ti >= P.ntris) {
          atomicOr(P.status, kStatusBounds);
        } else {
          const float4* tp = P.tris + 3 * (size_t)ti;
          const float4 ta = __ldg(tp), tb = __ldg(tp + 1), tc = __ldg(tp + 2);
          float t;
          if (tri_test<CLAMP>(ta, tb, tc, ox, oy, oz, dx, dy, dz, tmin, t, u, v)) {
            const int id = __float_as_int(tc.y);
            if (t < best_t || (!ANY && t == best_t && id < best_id))
              key = ((unsigned long long)order_key(t) << 32) | (uint32_t)id;
          }
        }
      }
      const unsigned cand = __ballot_sync(kFull, key != ~0ull);
      if (ANY) {
        if ((cand >> (8 * grp)) & 0xffu) {
          hit_any = true;
          node = kNoItem;
          tris = 0;
        }
      } else if (cand) {
        unsigned long long low = key;
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) {
          const unsigned long long o = __shfl_xor_sync(kFull, low, d);
          low = o < low ? o : low;
        }
        // (two triangles of one ID cannot occur: IDs are a permutation)
        const uint32_t from = (__ballot_sync(kFull, key == low) >> (8 * grp)) & 0xffu;
        const int src = (int)(8 * grp) + __ffs(from) - 1;
        const float wu = __shfl_sync(kFull, u, src), wv = __shfl_sync(kFull, v, src);
        if (low != ~0ull) {
          best_t = from_order_key((uint32_t)(low >> 32));
          best_id = (int)(uint32_t)low;
          bu = wu;
          bv = wv;
        }
      }
      if (n <= 8) {
        tris = 0;
      } else {
        for (int i = 0; i < 8; ++i) tris &= tris - 1u;
      }
    }
    __syncwarp();  // the stack entries written above
  }
  if (lost) best_id = -1, hit_any = false;
  if (live && c == 0) {
    if (ANY) {
      reinterpret_cast<uint8_t*>(P.out)[ray] = hit_any ? 1 : 0;
    } else {
      reinterpret_cast<int4*>(P.out)[ray] =
          best_id >= 0 ? make_int4(best_id, __float_as_int(best_t), __float_as_int(bu),
                                   __float_as_int(bv))
                       : make_int4(-1, 0, 0, 0);
    }
  }
}

// ---------------------------------------------------------------------------
// kd-tree walk in the reference's order (Kdtree.cpp:682-784).

struct KdParams {
  const KdNode* nodes;
  const uint32_t* items;
  const float4* tris;  // triangle-ID order
  const float4* rays;
  const uint32_t* order;  // null, or: queue index q walks ray order[q] (binned batches)
  void* out;
  uint32_t* status;
  unsigned* counter;
  unsigned share;  // > 0: warp w walks queue indices [w * share, (w + 1) * share)
  unsigned nrays, nnodes, nitems, ntris;
  float lo[3], hi[3];  // root box min corner and pos + size
};

// The walk alternates between two phases, each with most of the warp's lanes
// at work.  One thread per ray that tested its own leaves ran 5.8 lanes per
// instruction: a lane at a leaf looped over its items while the others waited
// (3.69 G warp instructions for 1M rays on a 524,288-triangle field).
//   1. Every lane steps through inner nodes and empty leaves until it stands
//      at a leaf with items; the phase ends once kKdLeave or fewer lanes are
//      still walking (they go on next time).
//   2. The items of all those leaves form one list that the warp tests 32 at
//      a time, lane w testing item w with its owner's ray.  The reference tests
//      a leaf's items in order and keeps t < best; the smallest (t, position in
//      the list) below the owner's best is the same item.
// Lanes whose walk is over take new rays once kKdRefill of them are idle, so
// the set-up's six divisions run for several lanes at a time.
// Measured on that batch: 5,190 us one thread per ray, 2,114 us with every leaf
// in the list (1.60 G warp instructions at 25 lanes), 1,923 with long leaves by
// themselves (from 24 / 32 / 48 / 96 items: 1,944 / 1,937 / 1,924 / 1,922); with the
// list, kKdLeave 4 / 8 / 12 / 20 / 24: 2,308 / 2,210 /
// 2,152 / 2,155 / 2,260; kKdRefill 1 / 4 / 16: within 1 %; 6 / 7 / 9 / 10 blocks
// per SM: 2,441 / 2,253 / 2,200 / 2,560.  What bounds it now: issue (73 %
// active) and the latency of its dependent node, item and triangle loads (L2 hit
// rate 99 %).
constexpr int kKdBlocks = 8;
constexpr int kKdLeave = 16;
constexpr int kKdRefill = 8;
constexpr unsigned kKdChunk = 32;  // rays a warp takes from the queue at a time
// Deferred far children of the walk: at most one per level.  The first entries
// live in shared memory, which most rays never leave; deeper ones in local
// memory.
constexpr int kKdShared = 12;
constexpr int kKdStack = 64;
// A leaf of so many items or more is tested by itself, with no list and no
// shared-memory minimum per round: cells at the tree's depth limit hold hundreds
// (5 % of the field's leaves held 70 % of the tests, 362 items each).
constexpr uint32_t kKdLong = 64;

template <bool CLAMP, bool ANY>
__global__ void __launch_bounds__(128, kKdBlocks) kd_trace(KdParams P) {
  __shared__ uint2 s_stack[kKdShared][128];
  __shared__ float s_o[3][128], s_inv[3][128];  // for the walk: by axis
  __shared__ float4 s_from[128], s_dir[128];    // for the tests: o, tmin; d, tmax
  __shared__ unsigned long long s_key[128];  // best candidate of the lane's leaf
  __shared__ float4 s_hit[128];              // t, u, v, ID of the ray's closest hit so far
  __shared__ uint8_t s_own[128];             // r-th lane of the warp that has leaf items
  uint2 deep[kKdStack - kKdShared];               // stack entries beyond the shared ones
  const unsigned tid = threadIdx.x, lane = tid & 31u, wbase = tid & ~31u;
  const unsigned lt = lanemask_lt();

  unsigned pool_next = 0, pool_end = 0;
  bool exhausted = false;
  if (P.share) {
    const unsigned w = blockIdx.x * (blockDim.x >> 5) + (tid >> 5);
    pool_next = min(w * P.share, P.nrays);
    pool_end = min(pool_next + P.share, P.nrays);
  }

  bool active = false;
  unsigned ray = 0, steps = 0;
  uint32_t node = 0;
  uint32_t cnt = 0, beg = 0;  // pending leaf (cnt > 0): its items
  int sp = 0;
  float tmin = 0.f, tmax = 0.f, tend = 0.f, best_t = INFINITY;

  while (true) {
    // ---- refill idle lanes ------------------------------------------------
    unsigned idle = __ballot_sync(kFull, !active);
    if (idle && !exhausted && (idle == kFull || __popc(idle) >= kKdRefill)) {
      bool fresh = false;
      while (idle && !exhausted) {
        if (pool_next >= pool_end) {
          unsigned b = P.nrays;
          if (!P.share) {
            if (lane == 0) b = atomicAdd(P.counter, kKdChunk);
            b = __shfl_sync(kFull, b, 0);
          }
          if (b >= P.nrays) {
            exhausted = true;
            break;
          }
          pool_next = b;
          pool_end = min(b + kKdChunk, P.nrays);
        }
        const unsigned avail = pool_end - pool_next;
        const unsigned rank = __popc(idle & lt);
        if (((idle >> lane) & 1u) && rank < avail) {
          ray = pool_next + rank;
          active = fresh = true;
          if (P.order) {
            ray = __ldg(P.order + ray);
            if (ray >= P.nrays) {  // an order entry outside the batch: skipped and reported
              atomicOr(P.status, kStatusBounds);
              active = fresh = false;
            }
          }
        }
        pool_next += min(avail, (unsigned)__popc(idle));
        idle = __ballot_sync(kFull, !active);
      }
      if (fresh) {
        const float4 r0 = __ldg(P.rays + 2 * (size_t)ray);
        const float4 r1 = __ldg(P.rays + 2 * (size_t)ray + 1);
        const float o[3] = {r0.x, r0.y, r0.z};
        const float d[3] = {r1.x, r1.y, r1.z};
        // m_Bounds.Intersect(r, tmin, tmax)  (AABB.cpp:117-143)
        float t0 = 0.f, t1 = INFINITY;
        bool in = true;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          s_o[i][tid] = o[i];
          s_inv[i][tid] = __fdiv_rn(1.f, d[i]);
          if (in) {
            float tin = __fdiv_rn(fs(P.lo[i], o[i]), d[i]);
            float tout = __fdiv_rn(fs(P.hi[i], o[i]), d[i]);
            if (tin > tout) {
              const float tt = tin;
              tin = tout;
              tout = tt;
            }
            t0 = tin > t0 ? tin : t0;
            t1 = tout < t1 ? tout : t1;
            if (t0 > t1) in = false;
          }
        }
        s_from[tid] = r0;
        s_dir[tid] = r1;
        s_hit[tid] = make_float4(INFINITY, 0.f, 0.f, __int_as_float(-1));
        best_t = INFINITY;
        tmin = t0;
        tmax = tend = t1;
        sp = 0;
        node = 0;
        steps = 0;
        cnt = 0;
        if (!in) node = kNoItem;  // no walk: ends below as a miss
      }
      __syncwarp();  // the other lanes read a fresh ray and write its hit (a ballot orders no memory)
    }
    if (__ballot_sync(kFull, active) == 0) break;

    // The walk returns to the far child deferred last.  The interval it was
    // deferred with ended where the one below it on the stack begins (or at
    // the root box's exit): a push sets tmax to the new entry's tplane and a
    // pop restores the value before it, so an entry needs no tmax of its own.
    auto entry = [&](int i) { return i < kKdShared ? s_stack[i][tid] : deep[i - kKdShared]; };
    auto pop = [&]() {
      if (sp == 0) return false;
      --sp;
      const uint2 e = entry(sp);
      node = e.x;
      tmin = __uint_as_float(e.y);
      tmax = sp > 0 ? __uint_as_float(entry(sp - 1).y) : tend;
      return true;
    };

    // ---- walk until the lanes stand at leaves -----------------------------
    bool fin = active && node == kNoItem;  // the ray's walk is over
    bool lost = false;                     // stopped at a bound: reported as a miss
    while (true) {
      const bool walking = active && !fin && cnt == 0;
      const unsigned wm = __ballot_sync(kFull, walking);
      const unsigned at_leaf = __ballot_sync(kFull, cnt != 0);
      if (wm == 0 || (at_leaf != 0 && __popc(wm) <= kKdLeave)) break;
      if (!walking) continue;
      if (++steps > kMaxSteps) {
        atomicOr(P.status, kStatusWatchdog);
        fin = lost = true;
      } else if (best_t < tmin) {
        fin = true;
      } else if (node >= P.nnodes) {
        atomicOr(P.status, kStatusBounds);
        fin = lost = true;
      } else {
        const uint2 n = __ldg(reinterpret_cast<const uint2*>(P.nodes) + node);
        const uint32_t axis = n.x & 3u;
        if (axis != 3u) {
          float split = __uint_as_float(n.x);
          split = (split > -0.001f && split < 0.001f) ? 0.0f : split;
          const float oa = s_o[axis][tid], ia = s_inv[axis][tid];
          const float tplane = fm(fs(split, oa), ia);
          const bool below = oa <= split;
          const uint32_t first = below ? n.y : n.y + 1;
          const uint32_t second = below ? n.y + 1 : n.y;
          if (tplane == 0.0f) {
            node = ia > 0.0f ? second : first;
          } else if (tplane >= tmax || tplane < 0.0f) {
            node = first;
          } else if (tplane <= tmin) {
            node = second;
          } else if (sp >= kKdStack) {
            atomicOr(P.status, kStatusStack);
            fin = lost = true;
          } else {
            const uint2 e = make_uint2(second, __float_as_uint(tplane));
            if (sp < kKdShared) s_stack[sp][tid] = e;
            else deep[sp - kKdShared] = e;
            ++sp;
            node = first;
            tmax = tplane;
          }
        } else {
          cnt = n.x >> 2;
          beg = n.y;
          if ((size_t)beg + cnt > P.nitems) {
            atomicOr(P.status, kStatusBounds);
            cnt = 0;
            fin = lost = true;
          } else if (cnt == 0 && !pop()) {  // an empty leaf
            fin = true;
          }
        }
      }
    }

    // ---- the warp tests the items of its lanes' leaves together -----------
    // Long leaves one by one: all lanes test the same ray, lane l items l, l + 32,
    // ..., and keep the first nearest of theirs.
    for (unsigned big = __ballot_sync(kFull, cnt >= kKdLong); big; big &= big - 1u) {
      const int src = __ffs(big) - 1;
      const unsigned ot = wbase + (unsigned)src;
      const uint32_t n = __shfl_sync(kFull, cnt, src);
      const uint32_t* items = P.items + __shfl_sync(kFull, beg, src);
      const float4 o = s_from[ot], d = s_dir[ot];
      float4 near = make_float4(__shfl_sync(kFull, best_t, src), 0.f, 0.f, __int_as_float(-1));
      uint32_t at = ~0u;
      for (uint32_t k = lane; k < n; k += 32) {
        const uint32_t id = __ldg(items + k);
        if (id >= P.ntris) {
          atomicOr(P.status, kStatusBounds);
          continue;
        }
        const float4* tp = P.tris + 3 * (size_t)id;
        float t, u, v;
        if (tri_test<CLAMP>(__ldg(tp), __ldg(tp + 1), __ldg(tp + 2), o.x, o.y, o.z, d.x, d.y, d.z,
                            o.w, t, u, v) &&
            t < near.x) {
          near = make_float4(t, u, v, __int_as_float((int)id));
          at = k;
        }
      }
      // the smallest t, then the first in the list (-0 and +0 are one distance)
      const uint32_t key = at != ~0u ? order_key(near.x == 0.0f ? 0.0f : near.x) : ~0u;
      const uint32_t low = __reduce_min_sync(kFull, key);
      const uint32_t first = __reduce_min_sync(kFull, key == low ? at : ~0u);
      if (first != ~0u && at == first) s_hit[ot] = near;
      __syncwarp();
      if ((int)lane == src) {
        if (first != ~0u) best_t = s_hit[ot].x;
        cnt = 0;
        if (!pop()) fin = true;
      }
    }
    const unsigned leaves = __ballot_sync(kFull, cnt != 0);
    if (leaves) {
      uint32_t excl = cnt;  // becomes the lane's first item in the warp's list
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, excl, d);
        if ((int)lane >= d) excl += v;
      }
      const uint32_t total = __shfl_sync(kFull, excl, 31);
      excl -= cnt;
      if (cnt) s_own[wbase + __popc(leaves & lt)] = (uint8_t)lane;
      s_key[tid] = ~0ull;
      __syncwarp();
      for (uint32_t base = 0; base < total; base += 32) {
        // the owner of item base + lane: the last lane whose list starts at
        // or before it
        const bool starts = cnt && excl >= base && excl < base + 32;
        const uint32_t first = __reduce_or_sync(kFull, starts ? 1u << (excl - base) : 0u);
        const unsigned before = __popc(__ballot_sync(kFull, cnt && excl < base));
        const unsigned own = s_own[wbase + before + __popc(first & (lt | (1u << lane))) - 1];
        const uint32_t oexcl = __shfl_sync(kFull, excl, own);
        const uint32_t obeg = __shfl_sync(kFull, beg, own);
        const float obest = __shfl_sync(kFull, best_t, own);
        const unsigned ot = wbase + own;
        bool cand = false;
        unsigned long long key = 0;
        float t = 0.f, u = 0.f, v = 0.f;
        uint32_t id = 0;
        if (base + lane < total) {
          const uint32_t k = base + lane - oexcl;
          id = __ldg(P.items + obeg + k);
          if (id >= P.ntris) {
            atomicOr(P.status, kStatusBounds);
          } else {
            const float4* tp = P.tris + 3 * (size_t)id;
            const float4 o = s_from[ot], d = s_dir[ot];
            if (tri_test<CLAMP>(__ldg(tp), __ldg(tp + 1), __ldg(tp + 2), o.x, o.y, o.z, d.x, d.y,
                                d.z, o.w, t, u, v) &&
                t < obest) {
              cand = true;
              // -0 and +0 are one distance: the first of them in the list wins
              key = ((unsigned long long)order_key(t == 0.0f ? 0.0f : t) << 32) | k;
              atomicMin(&s_key[ot], key);
            }
          }
        }
        __syncwarp();
        if (cand && s_key[ot] == key) s_hit[ot] = make_float4(t, u, v, __int_as_float((int)id));
        __syncwarp();
      }
      if (cnt) {
        if (s_key[tid] != ~0ull) best_t = s_hit[tid].x;
        cnt = 0;
        if (!pop()) fin = true;
      }
    }

    // ---- finished rays ----------------------------------------------------
    if (fin) {
      // IsInShadow form: closest hit && t < distance; closest: hits at or
      // beyond the ray's tmax are reported as misses.
      const float4 h = s_hit[tid];
      const int id = lost ? -1 : __float_as_int(h.w);
      const bool hit = id >= 0 && h.x < s_dir[tid].w;
      if (ANY) {
        reinterpret_cast<uint8_t*>(P.out)[ray] = hit ? 1 : 0;
      } else {
        reinterpret_cast<int4*>(P.out)[ray] =
            hit ? make_int4(id, __float_as_int(h.x), __float_as_int(h.y), __float_as_int(h.z))
                : make_int4(-1, 0, 0, 0);
      }
      active = false;
      node = 0;
      cnt = 0;
    }
    __syncwarp();
  }
}

// Shared memory per stack entry: width 8 packs lb into the 8-byte entry;
// widths 2 and 4 keep it in a separate float array.
constexpr size_t stack_entry_bytes(int W) {
  return W == 8 ? sizeof(uint2) : sizeof(uint2) + sizeof(float);
}

// The largest batch that wbvh_few takes, in warps of four rays per SM (28,416
// rays on 148 SMs): at 28,000 rays it took 82 us against 94 in 10,000 random
// triangles, 47 against 59 on a 131,072-triangle field and 83 against 107 for
// shadow rays in 100,000 triangles, at 38,000 rays 96 against 92, 62 against 70 and
// 100 against 99.  A caller's choice of chunk, block or blocks per SM is one of
// wbvh_trace's shape.
constexpr int kFewWarps = 48;
bool few_rays(const Launch& L, size_t n, int sms) {
  return !L.fixed_chunk && !L.fixed_shape && n <= (size_t)sms * kFewWarps * 4;
}
// Whether WAIT pays: a launch of six chunks of 32 rays per resident warp or more
// (1,022,976 rays), in a tree with fewer than kFewTests triangle tests per node
// visit.  At 300,000 / 524,288 / 1M / 2M / 4M eye rays on 10,000 random triangles
// (0.34 tests) it took 315 / 225 / 340 / 580 / 1,056 us against 305 / 222 / 343 / 592 /
// 1,083 without.  Where a visit tests more, rounds are fuller anyway: 1.84M bounce
// rays on 100,000 random triangles (1.05) took 480 us against 468, 4M on 1M (2.1)
// 6,210 against 6,049; fields of 20,000 to 2M triangles lie at 0.36 to 0.51 and gain
// 1.4 to 6 %.  The line lies where neither form loses: from 600,000 to 1M rays closest
// hit gains 0 to 3 % on those trees, but any hit loses 0.7 to 3.5 % on 10,000 random
// triangles, 1 % at 1M still, and gains 1 to 3 % on the fields from 700,000 on.
// Any hit, at 9 blocks per SM too: 4M / 2M / 1M rays over fields 666 ->
// 609 / 305 -> 288 / 164 -> 160 us, 2M on 2,000 / 10,000 / 20,000 random triangles
// 446 -> 434 / 721 -> 714 / 757 -> 753, 1.5M on 100,000 656 -> 669; 300,000 rays 62 ->
// 64; where no ray is blocked and most leave the field at once (4.18M toward a light
// above it) 237 -> 242.  The multi-scene form, whose 64 registers hold the waiting lanes'
// state at no cost, gains up to kFewTestsMulti: 3M rays over two scenes 721 -> 685
// us on a 131,072-triangle field, 1,234 -> 1,197 / 1,441 -> 1,404 / 1,869 -> 1,851 on
// 10,000 / 30,000 / 100,000 random triangles, 4,920 -> 5,015 on 1M.
bool many_rays(size_t n, int blocks, int threads) {
  return n >= (size_t)blocks * (size_t)threads * 6;
}

// A launch gets 48 KB of shared memory per block without asking for more, and the
// traversal's own arrays (9.2 KB) are part of it beside the stacks.
template <class Kernel>
cudaError_t allow_shared(Kernel k, size_t stacks) {
  if (stacks <= 36 * 1024) return cudaSuccess;
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)stacks);
}

template <bool CLAMP, bool ANY>
int launch_few(TraceParams p, size_t n, int sms, cudaStream_t s) {
  const size_t warps = (size_t)sms * kSpreadWarps;
  p.share = (unsigned)std::min<size_t>(4, (n + warps - 1) / warps);  // rays per warp
  if (n == 0) p.share = 1;  // a warm-up launch: one block that finds no ray
  const size_t smem = (size_t)16 * p.stack_depth * sizeof(uint2);  // 16 rays per block
  const unsigned grid = (unsigned)std::max<size_t>(1, (n + 4 * p.share - 1) / (4 * p.share));
  wbvh_few<CLAMP, ANY><<<grid, 128, smem, s>>>(p);
  return (int)cudaGetLastError();
}

template <int W, bool CLAMP, bool ANY, bool COUNT>
int launch_w(const DevAccel& a, const float* rays, size_t n, void* out, uint32_t* visits,
             const Launch& L, cudaStream_t s, const uint32_t* order) {
  TraceParams p{};
  p.nodes = static_cast<const uint8_t*>(a.d_nodes);
  p.tris = reinterpret_cast<const float4*>(a.d_tris);
  p.rays = reinterpret_cast<const float4*>(rays);
  p.order = order;
  p.out = out;
  p.visits = visits;
  const uint32_t slot =
      __atomic_fetch_add(const_cast<uint32_t*>(&a.counter_seq), 1u, __ATOMIC_RELAXED) % kQueueSlots;
  p.counter = a.d_counter + slot;
  p.status = a.d_status;
  p.nrays = (unsigned)n;
  p.nnodes = a.nnodes;
  p.ntris = a.ntris;
  // Each visited node leaves at most one group entry, so tree_depth - 1
  // entries always suffice; 0 selects that bound.
  p.stack_depth = L.stack > 0 ? L.stack : (a.tree_depth > 8 ? a.tree_depth : 8);
  p.chunk = L.chunk;
  const int sms = device_sm_count(a.device);
  if constexpr (W == 8 && !COUNT) {
    if (few_rays(L, n, sms)) return launch_few<CLAMP, ANY>(p, n, sms, s);
  }
  size_t smem = (size_t)p.stack_depth * L.block * stack_entry_bytes(W);
  const bool lane = !ANY && L.per_lane;
  // Binned (ordered) launches use their own instantiation (closest hit
  // only); without the order handling the plain cooperative kernel ran 1.6 %
  // faster.  The per-lane form, which the host-buffer pipeline runs beside
  // its copies, keeps it whatever the order: leaner, it ran faster but slowed
  // the concurrent copies more (the whole call 4 % slower).
  const bool ord = !ANY && order != nullptr;
  auto k = wbvh_trace<W, CLAMP, ANY, COUNT>;
  if constexpr (!ANY) {
    if (lane) k = wbvh_trace<W, CLAMP, false, COUNT, false, true, true>;
    else if (ord) k = wbvh_trace<W, CLAMP, false, COUNT, false, false, true>;
  }
  if constexpr (W == 8 && !COUNT) {
    const int blocks =
        sms * (L.blocks_per_sm > 0 ? L.blocks_per_sm : (ANY ? kBlocksAny : kBlocksClosest));
    if (!lane && a.tests_per_visit < kFewTests && many_rays(n, blocks, L.block)) {
      k = wbvh_trace<W, CLAMP, ANY, false, false, false, false, true>;
      if constexpr (!ANY) {
        if (ord) k = wbvh_trace<W, CLAMP, false, false, false, false, true, true>;
      }
    }
  }
  if (const cudaError_t e = allow_shared(k, smem); e != cudaSuccess) return (int)e;
  int grid = sms * (L.blocks_per_sm > 0
                        ? L.blocks_per_sm
                        : (ANY ? kBlocksAny : (lane ? kBlocksLane : kBlocksClosest)));
  p.share = ray_share(L, n, sms, &grid);
  if (p.share == 0) {
    cudaError_t e = cudaMemsetAsync(p.counter, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return (int)e;
  }
  k<<<grid, L.block, smem, s>>>(p);
  return (int)cudaGetLastError();
}

template <bool ANY, bool COUNT>
int dispatch_w(const DevAccel& a, const float* rays, size_t n, void* out, uint32_t* visits,
               const Launch& L, cudaStream_t s, const uint32_t* order = nullptr) {
  const bool clamp = a.predicate == ENC_PRED_REFERENCE;
  switch (a.width) {
    case 2:
      return clamp ? launch_w<2, true, ANY, COUNT>(a, rays, n, out, visits, L, s, order)
                   : launch_w<2, false, ANY, COUNT>(a, rays, n, out, visits, L, s, order);
    case 4:
      return clamp ? launch_w<4, true, ANY, COUNT>(a, rays, n, out, visits, L, s, order)
                   : launch_w<4, false, ANY, COUNT>(a, rays, n, out, visits, L, s, order);
    default:
      return clamp ? launch_w<8, true, ANY, COUNT>(a, rays, n, out, visits, L, s, order)
                   : launch_w<8, false, ANY, COUNT>(a, rays, n, out, visits, L, s, order);
  }
}

template <bool ANY>
int launch_kd(const DevAccel& a, const float* rays, size_t n, void* out, cudaStream_t s,
              const uint32_t* order = nullptr) {
  KdParams p;
  p.nodes = a.d_kd;
  p.items = a.d_kd_items;
  p.tris = reinterpret_cast<const float4*>(a.d_tris);
  p.rays = reinterpret_cast<const float4*>(rays);
  p.order = order;
  p.out = out;
  p.status = a.d_status;
  p.nrays = (unsigned)n;
  p.nnodes = a.nnodes;
  p.nitems = a.kd_nitems;
  p.ntris = a.ntris;
  for (int i = 0; i < 3; ++i) {
    p.lo[i] = a.kd_root_lo[i];
    p.hi[i] = a.kd_root_hi[i];
  }
  const uint32_t slot =
      __atomic_fetch_add(const_cast<uint32_t*>(&a.counter_seq), 1u, __ATOMIC_RELAXED) % kQueueSlots;
  p.counter = a.d_counter + slot;
  const int sms = device_sm_count(a.device);
  int grid = sms * kKdBlocks;
  p.share = ray_share(Launch(), n, sms, &grid);
  if (p.share == 0) {
    cudaError_t e = cudaMemsetAsync(p.counter, 0, sizeof(unsigned), s);
    if (e != cudaSuccess) return (int)e;
  }
  if (a.predicate == ENC_PRED_REFERENCE) kd_trace<true, ANY><<<grid, 128, 0, s>>>(p);
  else kd_trace<false, ANY><<<grid, 128, 0, s>>>(p);
  return (int)cudaGetLastError();
}

}  // namespace

int device_sm_count(int device) {
  static int cache[64] = {0};
  if (device < 0 || device >= 64) return 148;
  if (cache[device] == 0) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || v <= 0)
      v = 148;
    cache[device] = v;
  }
  return cache[device];
}

int launch_closest(const DevAccel& a, const float* d_rays, size_t n, enc_hit* d_hits,
                   const Launch& L, void* stream, uint32_t* d_visits, const uint32_t* d_order) {
  if (n == 0) return 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (a.kind == ENC_ACCEL_KDTREE) return launch_kd<false>(a, d_rays, n, d_hits, s, d_order);
  if (d_visits) return dispatch_w<false, true>(a, d_rays, n, d_hits, d_visits, L, s, d_order);
  return dispatch_w<false, false>(a, d_rays, n, d_hits, nullptr, L, s, d_order);
}

int launch_any(const DevAccel& a, const float* d_rays, size_t n, uint8_t* d_occ, const Launch& L,
               void* stream) {
  if (n == 0) return 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (a.kind == ENC_ACCEL_KDTREE) return launch_kd<true>(a, d_rays, n, d_occ, s);
  return dispatch_w<true, false>(a, d_rays, n, d_occ, nullptr, L, s);
}

namespace {

// Closest hit over the wide BVH with the queue head and status word supplied
// by the caller instead of taken from the accelerator.
template <int W, bool CLAMP>
int launch_w_external(const DevAccel& a, const float* rays, size_t n, enc_hit* hits,
                      const Launch& L, cudaStream_t s, uint32_t* counter, uint32_t* status) {
  TraceParams p{};
  p.nodes = static_cast<const uint8_t*>(a.d_nodes);
  p.tris = reinterpret_cast<const float4*>(a.d_tris);
  p.rays = reinterpret_cast<const float4*>(rays);
  p.out = hits;
  p.visits = nullptr;
  p.counter = counter;
  p.status = status;
  p.nrays = (unsigned)n;
  p.nnodes = a.nnodes;
  p.ntris = a.ntris;
  p.stack_depth = L.stack > 0 ? L.stack : (a.tree_depth > 8 ? a.tree_depth : 8);
  p.chunk = L.chunk;
  const int sms = device_sm_count(a.device);
  if constexpr (W == 8) {  // the warm-up launch (n = 0) runs both kernels
    if (few_rays(L, n, sms)) {
      const int e = launch_few<CLAMP, false>(p, n, sms, s);
      if (e != 0 || n > 0) return e;
    }
  }
  size_t smem = (size_t)p.stack_depth * L.block * stack_entry_bytes(W);
  auto k = wbvh_trace<W, CLAMP, false, false>;
  if (const cudaError_t e = allow_shared(k, smem); e != cudaSuccess) return (int)e;
  int grid = sms * (L.blocks_per_sm > 0 ? L.blocks_per_sm : kBlocksClosest);
  if (n > 0) p.share = ray_share(L, n, sms, &grid);
  k<<<grid, L.block, smem, s>>>(p);
  return (int)cudaGetLastError();
}

}  // namespace

int warm_closest_kernel(const DevAccel& a, uint32_t* counter, uint32_t* status) {
  // (not fixed_shape: the small-batch kernel is warmed with the other)
  // An empty batch: every warp finds the queue exhausted at once.  The launch
  // loads the kernel's module and sizes the context's local memory for it.
  Launch L = resolve_launch(nullptr, a.kind, a.width);
  L.blocks_per_sm = 1;
  int e = 0;
  const bool clamp = a.predicate == ENC_PRED_REFERENCE;
  float* no_rays = nullptr;
  switch (a.width) {
    case 2:
      e = clamp ? launch_w_external<2, true>(a, no_rays, 0, nullptr, L, 0, counter, status)
                : launch_w_external<2, false>(a, no_rays, 0, nullptr, L, 0, counter, status);
      break;
    case 4:
      e = clamp ? launch_w_external<4, true>(a, no_rays, 0, nullptr, L, 0, counter, status)
                : launch_w_external<4, false>(a, no_rays, 0, nullptr, L, 0, counter, status);
      break;
    default:
      e = clamp ? launch_w_external<8, true>(a, no_rays, 0, nullptr, L, 0, counter, status)
                : launch_w_external<8, false>(a, no_rays, 0, nullptr, L, 0, counter, status);
  }
  if (e != 0) return e;
  return (int)cudaStreamSynchronize(0);
}

int launch_closest_external_scratch(const DevAccel& a, const float* d_rays, size_t n,
                                    enc_hit* d_hits, const Launch& L, void* stream,
                                    uint32_t* counter, uint32_t* status) {
  if (n == 0) return 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool clamp = a.predicate == ENC_PRED_REFERENCE;
  switch (a.width) {
    case 2:
      return clamp ? launch_w_external<2, true>(a, d_rays, n, d_hits, L, s, counter, status)
                   : launch_w_external<2, false>(a, d_rays, n, d_hits, L, s, counter, status);
    case 4:
      return clamp ? launch_w_external<4, true>(a, d_rays, n, d_hits, L, s, counter, status)
                   : launch_w_external<4, false>(a, d_rays, n, d_hits, L, s, counter, status);
    default:
      return clamp ? launch_w_external<8, true>(a, d_rays, n, d_hits, L, s, counter, status)
                   : launch_w_external<8, false>(a, d_rays, n, d_hits, L, s, counter, status);
  }
}

}  // namespace enc

namespace enc {
namespace {

template <int W, bool CLAMP, bool ANY>
int launch_multi_w(const MultiLaunch& m, const Launch& L, cudaStream_t s) {
  TraceParams p{};
  p.counter = m.d_counter;
  p.status = m.d_status;
  p.nrays = m.total;
  p.stack_depth = L.stack > 0 ? L.stack : (m.stack_depth > 8 ? m.stack_depth : 8);
  p.chunk = L.chunk;
  p.scenes = m.d_scenes;
  p.batches = m.d_batches;
  p.starts = m.d_starts;
  p.nbatches = m.nbatches;
  p.batch_status = m.d_batch_status;
  size_t smem = (size_t)p.stack_depth * L.block * stack_entry_bytes(W);
  auto k = wbvh_trace<W, CLAMP, ANY, false, true>;
  if constexpr (W == 8 && !ANY) {
    const int blocks = device_sm_count(m.device) *
                       (L.blocks_per_sm > 0 ? L.blocks_per_sm : kBlocksMulti);
    if (m.wait && many_rays(m.total, blocks, L.block))
      k = wbvh_trace<W, CLAMP, false, false, true, false, false, true>;
  }
  if (const cudaError_t e = allow_shared(k, smem); e != cudaSuccess) return (int)e;
  cudaError_t e = cudaMemsetAsync(m.d_counter, 0, sizeof(unsigned), s);
  if (e != cudaSuccess) return (int)e;
  int grid = device_sm_count(m.device) *
             (L.blocks_per_sm > 0 ? L.blocks_per_sm : (ANY ? kBlocksAny : kBlocksMulti));
  k<<<grid, L.block, smem, s>>>(p);
  return (int)cudaGetLastError();
}

template <bool ANY>
int launch_multi(const MultiLaunch& m, const Launch& L, void* stream) {
  if (m.total == 0 || m.nbatches == 0) return 0;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool clamp = m.predicate == ENC_PRED_REFERENCE;
  switch (m.width) {
    case 2:
      return clamp ? launch_multi_w<2, true, ANY>(m, L, s) : launch_multi_w<2, false, ANY>(m, L, s);
    case 4:
      return clamp ? launch_multi_w<4, true, ANY>(m, L, s) : launch_multi_w<4, false, ANY>(m, L, s);
    default:
      return clamp ? launch_multi_w<8, true, ANY>(m, L, s) : launch_multi_w<8, false, ANY>(m, L, s);
  }
}

}  // namespace

int launch_multi_closest(const MultiLaunch& m, const Launch& L, void* stream) {
  return launch_multi<false>(m, L, stream);
}

int launch_multi_any(const MultiLaunch& m, const Launch& L, void* stream) {
  return launch_multi<true>(m, L, stream);
}

}  // namespace enc
