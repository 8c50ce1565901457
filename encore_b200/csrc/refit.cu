// Refit of a wide BVH on the device (Bvh::update, BVH.cpp:52-121): the
// triangles' new positions are uploaded and every box of the tree is formed
// again, bottom-up, and quantised.  Same results as the host refit
// (wbvh_build.cpp:refit_wbvh) bit for bit: minima and maxima do not depend on
// their order, a padded minimum is the minimum of padded values (rounding is
// monotone), and the grid arithmetic is the host's in FP64.
//
//   refit_bounds   scene bounds of the new vertices, and whether all are finite;
//   refit_tris     one thread per triangle: its record (DevTri) and its box, at
//                  its place in leaf order;
//   refit_levels   W lanes per node, one child box each, level by level from
//                  the deepest (the nodes lie in breadth-first order); the
//                  levels of at most kTopNodes nodes in one launch of one block.
//
// Bytes: 36 per triangle over PCIe and read twice from HBM, 48 + 24 written per
// triangle and 24 read back, 24 + a node per node; the upload is nearly all of
// the time.  A 524,288-triangle field, refit alone: 121 ms on the host, 1.07 ms
// here, of which the upload of 18.9 MB from pageable memory takes about 0.9.
#include <cuda_runtime.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstring>

#include "engine.h"

namespace enc {
namespace {

constexpr unsigned kFull = 0xffffffffu;
// A level of so many nodes takes one block of 1024 threads two passes at most,
// less than a launch of its own.
constexpr uint32_t kTopNodes = 256;

// A finite float as an unsigned key of the same order, and back.
__device__ __forceinline__ uint32_t key_of(float f) {
  const uint32_t b = __float_as_uint(f);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
float of_key(uint32_t k) {
  const uint32_t b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  float f;
  std::memcpy(&f, &b, 4);
  return f;
}

// out[0..2]: keys of the smallest x, y, z; out[3..5]: of the largest; out[6]:
// not 0 if a coordinate is infinite or NaN.
__global__ void __launch_bounds__(256) refit_bounds(const float* __restrict__ v, size_t nverts,
                                                    uint32_t* out) {
  __shared__ uint32_t s_red[8][7];
  uint32_t lo[3] = {~0u, ~0u, ~0u}, hi[3] = {0u, 0u, 0u}, bad = 0;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nverts;
       i += (size_t)gridDim.x * blockDim.x) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float x = __ldg(v + 3 * i + a);
      bad |= isfinite(x) ? 0u : 1u;
      const uint32_t k = key_of(x);
      lo[a] = min(lo[a], k);
      hi[a] = max(hi[a], k);
    }
  }
  const unsigned lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    lo[a] = __reduce_min_sync(kFull, lo[a]);
    hi[a] = __reduce_max_sync(kFull, hi[a]);
  }
  bad = __reduce_or_sync(kFull, bad);
  if (lane == 0) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      s_red[warp][a] = lo[a];
      s_red[warp][3 + a] = hi[a];
    }
    s_red[warp][6] = bad;
  }
  __syncthreads();
  if (threadIdx.x < 7) {
    uint32_t r = s_red[0][threadIdx.x];
    for (unsigned w = 1; w < blockDim.x / 32; ++w) {
      const uint32_t x = s_red[w][threadIdx.x];
      r = threadIdx.x < 3 ? min(r, x) : (threadIdx.x < 6 ? max(r, x) : (r | x));
    }
    if (threadIdx.x < 3) atomicMin(out + threadIdx.x, r);
    else if (threadIdx.x < 6) atomicMax(out + threadIdx.x, r);
    else if (r) atomicOr(out + 6, r);
  }
}

// A box: three float2 (lo.x lo.y | lo.z hi.x | hi.y hi.z), 24 bytes.
struct Box6 {
  float lo[3], hi[3];
};
__device__ __forceinline__ Box6 load_box(const float2* b, size_t i) {
  const float2 p = b[3 * i], q = b[3 * i + 1], r = b[3 * i + 2];
  return Box6{{p.x, p.y, q.x}, {q.y, r.x, r.y}};
}
__device__ __forceinline__ void store_box(float2* b, size_t i, const Box6& x) {
  b[3 * i] = make_float2(x.lo[0], x.lo[1]);
  b[3 * i + 1] = make_float2(x.lo[2], x.hi[0]);
  b[3 * i + 2] = make_float2(x.hi[1], x.hi[2]);
}

__global__ void __launch_bounds__(256) refit_tris(const float* __restrict__ v, uint32_t n,
                                                  const uint32_t* __restrict__ tri_pos,
                                                  float4* tris, float2* boxes) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t slot = __ldg(tri_pos + i);
    if (slot >= n) continue;
    float t[9];
#pragma unroll
    for (int k = 0; k < 9; ++k) t[k] = __ldg(v + 9 * (size_t)i + k);
    float4* d = tris + 3 * (size_t)slot;
    d[0] = make_float4(t[0], t[1], t[2], __fsub_rn(t[3], t[0]));
    d[1] = make_float4(__fsub_rn(t[4], t[1]), __fsub_rn(t[5], t[2]), __fsub_rn(t[6], t[0]),
                       __fsub_rn(t[7], t[1]));
    d[2] = make_float4(__fsub_rn(t[8], t[2]), __int_as_float((int)i), 0.f, 0.f);
    Box6 b;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      b.lo[a] = fminf(fminf(t[a], t[3 + a]), t[6 + a]);
      b.hi[a] = fmaxf(fmaxf(t[a], t[3 + a]), t[6 + a]);
    }
    store_box(boxes, slot, b);
  }
}

// Smallest e >= -126 with 255 * 2^e >= ext and 2^e >= the float spacing above
// mag (quantize_node's grid step).  ext: a non-negative difference of floats;
// mag: finite and below FLT_MAX.
__device__ __forceinline__ int grid_exponent(double ext, float mag) {
  int e = -126;
  if (ext > 0.0) {
    // ext = m * 2^k with 1 <= m < 2; 255 = 1.9921875 * 2^7
    const long long b = __double_as_longlong(ext);
    const int k = (int)((b >> 52) & 0x7ff) - 1023;
    const long long m255 = __double_as_longlong(1.9921875) & 0xfffffffffffffll;
    e = max(e, k - 7 + ((b & 0xfffffffffffffll) > m255 ? 1 : 0));
  }
  const int me = (int)(__float_as_uint(mag) >> 23);  // spacing: 2^(me - 150), 2^-149 below 2^-126
  return max(e, (me > 0 ? me : 1) - 150);
}

struct Levels {
  uint32_t start[65];  // nodes of level l: [start[l], start[l + 1])
};

// Levels hi_level down to lo_level; more than one only in a launch of one block.
template <int W>
__global__ void __launch_bounds__(1024)
    refit_levels(Levels lv, int hi_level, int lo_level, uint8_t* nodes,
                 const float2* tri_boxes, float2* node_boxes, float pad) {
  using L = WNodeLayout<W>;
  const unsigned c = threadIdx.x % W;
  for (int l = hi_level; l >= lo_level; --l) {
    const uint32_t s = lv.start[l], e = lv.start[l + 1];
    const uint32_t per = gridDim.x * (blockDim.x / W);
    // every lane of a warp runs the same passes, for the shuffles
    const uint32_t passes = (e - s + per - 1) / per;
    for (uint32_t p = 0; p < passes; ++p) {
      const uint32_t node = s + p * per + (blockIdx.x * blockDim.x + threadIdx.x) / W;
      const bool on = node < e;
      uint8_t* raw = nodes + (size_t)(on ? node : s) * L::kBytes;
      const uint4 h1 = *reinterpret_cast<const uint4*>(raw + 16);
      const uint32_t child_base = h1.x, tri_base = h1.y;
      const uint32_t m = on ? raw[L::kMetaOff + c] : 0u;
      Box6 b{{INFINITY, INFINITY, INFINITY}, {-INFINITY, -INFINITY, -INFINITY}};
      if (m >= 32u) {
        const uint32_t first = tri_base + (m & 31u);
        for (uint32_t k = 0; k < (m >> 5); ++k) {
          const Box6 t = load_box(tri_boxes, first + k);
#pragma unroll
          for (int a = 0; a < 3; ++a) {
            b.lo[a] = fminf(b.lo[a], t.lo[a]);
            b.hi[a] = fmaxf(b.hi[a], t.hi[a]);
          }
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          b.lo[a] = __fsub_rn(b.lo[a], pad);
          b.hi[a] = __fadd_rn(b.hi[a], pad);
        }
      } else if (m != 0u) {
        b = load_box(node_boxes, child_base + m - 1u);
      }
      Box6 nb = b;
#pragma unroll
      for (int o = 1; o < W; o <<= 1)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          nb.lo[a] = fminf(nb.lo[a], __shfl_xor_sync(kFull, nb.lo[a], o));
          nb.hi[a] = fmaxf(nb.hi[a], __shfl_xor_sync(kFull, nb.hi[a], o));
        }
      if (!on) continue;  // no shuffle follows in this pass
      uint32_t ew = 0;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double plo = (double)nb.lo[a];
        const int ex = grid_exponent((double)nb.hi[a] - plo,
                                     fmaxf(fabsf(nb.lo[a]), fabsf(nb.hi[a])));
        ew |= (uint32_t)(ex + 127) << (8 * a);
        uint32_t qlo = 255u, qhi = 0u;  // an empty slot: an inverted box
        if (m != 0u) {
          // dividing by the step 2^ex is exact, and so is multiplying by 2^-ex
          const double inv = __longlong_as_double((long long)(1023 - ex) << 52);
          qlo = (uint32_t)floor(((double)b.lo[a] - plo) * inv);
          qhi = (uint32_t)ceil(((double)b.hi[a] - plo) * inv);
        }
        raw[L::kQOff + a * W + c] = (uint8_t)qlo;
        raw[L::kQOff + (3 + a) * W + c] = (uint8_t)qhi;
      }
      if (c == 0) {
        store_box(node_boxes, node, nb);
        uint4* h0 = reinterpret_cast<uint4*>(raw);
        const uint32_t imask = h0->w & 0xff000000u;
        *h0 = make_uint4(__float_as_uint(nb.lo[0]), __float_as_uint(nb.lo[1]),
                         __float_as_uint(nb.lo[2]), ew | imask);
      }
    }
    if (l > lo_level) __syncthreads();
  }
}

template <int W>
cudaError_t run_levels(const Levels& lv, int nlevels, uint8_t* nodes, const float2* tri_boxes,
                       float2* node_boxes, float pad) {
  int l = nlevels - 1;
  while (l >= 0) {
    const uint32_t count = lv.start[l + 1] - lv.start[l];
    if (count > kTopNodes) {
      const uint32_t grid = (uint32_t)(((uint64_t)count * W + 255) / 256);
      refit_levels<W><<<grid, 256>>>(lv, l, l, nodes, tri_boxes, node_boxes, pad);
      --l;
    } else {
      int lo = l;
      while (lo > 0 && lv.start[lo] - lv.start[lo - 1] <= kTopNodes) --lo;
      refit_levels<W><<<1, 1024>>>(lv, l, lo, nodes, tri_boxes, node_boxes, pad);
      l = lo - 1;
    }
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// A bound of zero has the sign of the axis' first zero, as the host's minima and
// maxima leave it.  The keys put -0 below +0, so a minimum of +0 or a maximum of -0
// says that there is no other, and the vertices need not be looked through.
float zero_bound(const float* v, size_t nverts, int axis, float bound, bool largest) {
  if (bound != 0.f || std::signbit(bound) == largest) return bound;
  for (size_t i = 0; i < nverts; ++i)
    if (v[3 * i + axis] == 0.f) return v[3 * i + axis];
  return bound;
}

struct Scratch {
  void* p = nullptr;
  bool pooled = false;
  ~Scratch() {
    if (p) pool_free(p, pooled);
  }
};

}  // namespace

int refit_device(const DevAccel& d, const WBVHHost& host, RefitPlan* r, const float* tri_verts,
                 float lo[3], float hi[3], bool* done) {
  *done = false;
  if (!r->planned) {
    r->planned = true;
    r->usable = refit_levels_of(host, r->level_start);
  }
  if (!r->usable) return 0;
  const size_t nt = d.ntris, nn = d.nnodes;
  auto up = [](size_t x) { return (x + 255) / 256 * 256; };
  const size_t o_box = up(36 * nt), o_node = o_box + up(24 * nt), o_out = o_node + up(24 * nn);
  const size_t need = o_out + 256;
  // Taken for this call alone: on the legacy default stream, as all that uses it.
  Scratch mem;
  if (pool_alloc(&mem.p, need, d.device, &mem.pooled) != cudaSuccess) {
    cudaGetLastError();  // no room for the scratch: the host refit needs none
    mem.p = nullptr;
    return 0;
  }
  char* base = static_cast<char*>(mem.p);
  float* verts = reinterpret_cast<float*>(base);
  float2* tri_boxes = reinterpret_cast<float2*>(base + o_box);
  float2* node_boxes = reinterpret_cast<float2*>(base + o_node);
  uint32_t* out = reinterpret_cast<uint32_t*>(base + o_out);
  cudaError_t e = cudaMemcpy(verts, tri_verts, 36 * nt, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemsetAsync(out, 0xff, 12);
  if (e == cudaSuccess) e = cudaMemsetAsync(out + 3, 0, 16);
  if (e != cudaSuccess) return (int)e;
  const int sms = device_sm_count(d.device);
  const size_t wave = (size_t)sms * 8;
  auto blocks = [&](size_t n) { return (unsigned)std::min((n + 255) / 256, wave); };
  refit_bounds<<<blocks(3 * nt), 256>>>(verts, 3 * nt, out);
  uint32_t k[7];
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(k, out, sizeof(k), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return (int)e;
  if (k[6]) return 0;  // the host refit says what such coordinates give
  for (int a = 0; a < 3; ++a) {
    lo[a] = zero_bound(tri_verts, 3 * nt, a, of_key(k[a]), false);
    hi[a] = zero_bound(tri_verts, 3 * nt, a, of_key(k[3 + a]), true);
  }
  float maxabs = 0.f;
  for (int a = 0; a < 3; ++a) maxabs = std::max(maxabs, std::max(std::fabs(lo[a]), std::fabs(hi[a])));
  const float pad = box_pad(lo, hi, maxabs);
  for (int a = 0; a < 3; ++a)  // a grid needs a float above every corner
    if (!(lo[a] - pad > -FLT_MAX) || !(hi[a] + pad < FLT_MAX)) return 0;
  // From here on nothing can be refused, so the accelerator is written in place.
  refit_tris<<<blocks(nt), 256>>>(verts, (uint32_t)nt, d.d_tri_pos,
                                  reinterpret_cast<float4*>(d.d_tris), tri_boxes);
  e = cudaGetLastError();
  Levels lv{};
  const int nlevels = (int)r->level_start.size() - 1;
  for (int l = 0; l <= nlevels; ++l) lv.start[l] = r->level_start[l];
  uint8_t* nodes = static_cast<uint8_t*>(d.d_nodes);
  if (e == cudaSuccess)
    e = d.width == 2   ? run_levels<2>(lv, nlevels, nodes, tri_boxes, node_boxes, pad)
        : d.width == 4 ? run_levels<4>(lv, nlevels, nodes, tri_boxes, node_boxes, pad)
                       : run_levels<8>(lv, nlevels, nodes, tri_boxes, node_boxes, pad);
  if (e == cudaSuccess) e = cudaStreamSynchronize(0);
  *done = e == cudaSuccess;
  return (int)e;
}

}  // namespace enc
