// forceManyBody on the GPU: the d3 Barnes-Hut tree, built every tick and walked per point.
//
// The tree is exactly the one d3-octree / d3-quadtree / d3-binarytree build for
// src/manyBody.js (cube = floor(min) with a power-of-two size, midpoint splits, children in the
// order bit k = coordinate k above the midpoint), cut at LEVELS levels (21 in 3D, 24 in 1D/2D):
//
//   morton     the d3 cube from the bounding box, each point's cell at the finest level (exact),
//              interleaved into a left-aligned Morton key in d3's child order; the sort's digit
//              histograms are counted in the same pass
//   sort       onesweep radix sort of (key, node) over the top 31 (3D) / 32 (2D) key bits, then
//              the run fix-up that orders keys equal in those bits by the rest (sort.cu)
//   build      Karras (2012) binary radix tree over the sorted keys; each internal node's d3
//              depth = common prefix bits / DIMS; the sorted (position, strength) of the points,
//              and each point's d3 leaf depth (from the deeper of its two neighbour prefixes)
//   heads      a binary node whose depth is deeper than its parent's heads a d3 cell (the binary
//              nodes below it at the same depth are splits inside that cell); its d3 children
//              are counted, and child slots are allocated by a scan (every cell's children are
//              contiguous, so the walk reads them in one sweep)
//   cells      each cell's value and centre of mass as manyBody.js accumulate() defines them
//              (value = sqrt(4 / 2^DIMS) times the sum of the children's values; centroid
//              weighted by the children's |value|). When the strengths share one sign this
//              recursion has a closed form, value(D) = sum_p s_p c^(leafDepth_p - D) and centroid
//              weights |s_p| c^leafDepth_p, so every cell is a range sum of exact int64
//              fixed-point prefix sums over the sorted points. With strengths of both signs the
//              recursion itself runs over the d3 cells, from the deepest up through the child
//              slots, with atomic arrival counts: d3's FP64 values bit for bit (so cells that
//              cancel are skipped as d3 skips them), FP64 centroid sums for the top levels.
//   slots      each cell writes its children (position or centroid, value at own depth, and for
//              a child cell its child range and depth) into its slots
//   walk       a warp walks the union of the d3 traversals of 32 (or 16) consecutive sorted
//              points: rounds of up to 32 children are gathered from the group's stack in shared
//              memory, classified lane-parallel against the group's bounding box, and every lane
//              applies apply() of manyBody.js for its own point, two children per step in packed
//              FP32 pairs: a cell is approximated at the first (widest) depth of its chain where
//              w^2 / theta^2 < l, points are summed exactly, distanceMin / distanceMax as d3;
//              cells that some point must open are pushed with the mask of those points.
//
// Up to 6,144 points, morton to slots are one launch (k_small_tree).
//
// Points with the same code at the finest level share the deepest cell as its children.
#include <cooperative_groups.h>
#include <math.h>

#include <atomic>
#include <cuda/atomic>
#include <cmath>
#include <type_traits>

#include "kernels.h"

namespace {

constexpr uint32_t kLeaf = 0x80000000u;
constexpr uint32_t kIndex = 0x7fffffffu;
constexpr uint32_t kLeafMark = 0x7fffffffu;  // meta word of a point (a cell's is count | depth << 26)
constexpr uint32_t kCountMask = (1u << 26) - 1;
constexpr uint32_t kNoParent = 0xffffffffu;  // a point alone in its graph (batches)
constexpr uint8_t kGapDepth = 0xff;          // an internal index between two graphs (batches)
constexpr int kThreads = 256;

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

struct alignas(32) D4 {  // four exact fixed-point sums
  long long x, y, z, w;
};
__host__ __device__ __forceinline__ D4 mk4(long long a, long long b, long long c, long long d) {
  return {a, b, c, d};
}

__device__ __forceinline__ uint64_t spread3(uint64_t x) {  // 21 bits -> every third bit
  x &= 0x1fffffull;
  x = (x | x << 32) & 0x1f00000000ffffull;
  x = (x | x << 16) & 0x1f0000ff0000ffull;
  x = (x | x << 8) & 0x100f00f00f00f00full;
  x = (x | x << 4) & 0x10c30c30c30c30c3ull;
  x = (x | x << 2) & 0x1249249249249249ull;
  return x;
}
__device__ __forceinline__ uint64_t spread2(uint64_t x) {  // 32 bits -> every other bit
  x &= 0xffffffffull;
  x = (x | x << 16) & 0x0000ffff0000ffffull;
  x = (x | x << 8) & 0x00ff00ff00ff00ffull;
  x = (x | x << 4) & 0x0f0f0f0f0f0f0f0full;
  x = (x | x << 2) & 0x3333333333333333ull;
  x = (x | x << 1) & 0x5555555555555555ull;
  return x;
}

__device__ __forceinline__ int levels_of(int ndim) { return ndim == 3 ? 21 : 24; }

// c^k with c = sqrt(4 / 2^DIMS) (the per-level scale of manyBody.js accumulate()): c is a power
// of sqrt(2), c^k = 2^(k (2 - DIMS) / 2), so it is an exact power of two, times sqrt(2) when the
// exponent is odd.
__device__ __forceinline__ float damp(int ndim, int k) {
  const int e2 = k * (2 - ndim);  // |e2| <= 2 * 24 (levels): the power of two is a normal float
  const float odd = (e2 & 1) ? 1.41421356237309515f : 1.f;
  return odd * __int_as_float((127 + (e2 >> 1)) << 23);
}

// Conversions between FP32 and 64-bit integers in integer arithmetic: the hardware's 64-bit
// conversions issue on the FP64 pipe, a small fraction of the FP32 rate on this part.
// f2ll_rn: round to nearest even, |v| < 2^63 (above 2^24 a float is an integer: its significand
// shifted into place; below, the 32-bit conversion rounds).
__device__ __forceinline__ long long f2ll_rn(float v) {
  const uint32_t b = __float_as_uint(v);
  const int e = (int)((b >> 23) & 255u) - 150;  // |v| = significand * 2^e
  if (e < 0) return (long long)__float2int_rn(v);
  const long long m = (long long)((b & 0x7fffffu) | 0x800000u) << e;
  return (b >> 31) ? -m : m;
}
// ll2f_rn: the nearest float (ties to even) to a 64-bit integer.
__device__ __forceinline__ float ll2f_rn(long long v) {
  const unsigned long long u = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  float r;
  if (u < (1ull << 24)) {
    r = (float)(uint32_t)u;
  } else {
    const int lz = __clzll((long long)u);
    const unsigned long long w = u << lz;  // top bit at 63
    uint32_t m = (uint32_t)(w >> 40);      // 24 significant bits
    const unsigned long long rest = w & ((1ull << 40) - 1);
    if (rest > (1ull << 39) || (rest == (1ull << 39) && (m & 1u))) ++m;
    r = (float)m * __int_as_float((127 + 40 - lz) << 23);  // m <= 2^24, 2^(40 - lz): exact
  }
  return v < 0 ? -r : r;
}

// (x - o) * 2^F as an exact integer: x - o is rounded once in FP32 and its rounding error
// recovered exactly (Knuth's TwoSum); both parts scale exactly by the power of two 2^F.
__device__ __forceinline__ long long fx_offset(float x, float o, float scaleF) {
  const float s = x - o;
  const float bb = s - x;
  const float e = (x - (s - bb)) + (-o - bb);
  const long long d = f2ll_rn(s * scaleF) + f2ll_rn(e * scaleF);
  return d < 0 ? 0 : d;
}
// floor(W * D / 2^62) for W, D >= 0 (the 128-bit product's bits 62..125)
__device__ __forceinline__ long long mulhi62(long long W, long long D) {
  const unsigned long long hi = __umul64hi((unsigned long long)W, (unsigned long long)D);
  const unsigned long long lo = (unsigned long long)W * (unsigned long long)D;
  return (long long)((hi << 2) | (lo >> 62));
}
// 2^F of the fixed-point offsets: u = (x - origin) / size = offset / 2^62, F = 62 - log2(size)
__device__ __forceinline__ float offset_scale(const float* cube) {
  int F = 62 - (int)cube[4];
  F = F < -100 ? -100 : F > 100 ? 100 : F;
  return __int_as_float((F + 127) << 23);
}

// 4^-k as an exact float (k <= 31)
__device__ __forceinline__ float pow4neg(uint32_t k) { return __int_as_float((127 - 2 * (int)k) << 23); }

// floor((floor(x) - origin) * 2^e) for e < 0, in FP64 where every step is exact. Not inlined:
// inlined, the compiler predicates it into the common path, which then pays its FP64 work.
__device__ __noinline__ float cell_of_wide(float x, float origin, int e) {
  return (float)floor(ldexp(floor((double)x) - (double)origin, e));
}

// The cell index of x at the finest level, floor((x - origin) * 2^e), in exact arithmetic:
// e >= 0: floor(x * 2^e) and origin * 2^e are exact floats, and so is their difference, an
// integer below 2^24; e < 0 (cubes wider than 2^LEVELS): cell_of_wide.
__device__ __forceinline__ uint64_t cell_of(float x, float origin, int e, uint32_t top) {
  float c;
  if (e >= 0) {
    const float s = __int_as_float((e + 127) << 23);
    c = floorf(x * s) - origin * s;
  } else {
    c = cell_of_wide(x, origin, e);
  }
  c = fminf(fmaxf(c, 0.f), (float)top);
  return (uint64_t)(uint32_t)c;  // below 2^24: a 32-bit conversion (the 64-bit one is FP64-pipe)
}

// d3 cover() of a bounding box (d3-octree): origin = floor(min); a power-of-two size doubled
// until max < origin + size (FP64). cube5 = origin x, y, z, size, log2 size. WARP: every lane of the
// warp calls it for one box, tries a size of its own, and lane 0 writes: one thread's chain of FP64 sums
// and compares took 3,600 clocks for 11 doublings, at the start of every tick. Otherwise by one thread.
template <bool WARP>
__device__ __forceinline__ void d3_cover(const FlReduce* red, int ndim, float* cube5) {
  double lo0 = 0, lo1 = 0, lo2 = 0, hi0 = 0, hi1 = 0, hi2 = 0;
  lo0 = floor((double)fl::unordered(~red->lo[0])), hi0 = (double)fl::unordered(red->hi[0]);
  if (ndim > 1) lo1 = floor((double)fl::unordered(~red->lo[1])), hi1 = (double)fl::unordered(red->hi[1]);
  if (ndim > 2) lo2 = floor((double)fl::unordered(~red->lo[2])), hi2 = (double)fl::unordered(red->hi[2]);
  const auto holds = [&](double size) {
    return hi0 < lo0 + size && (ndim < 2 || hi1 < lo1 + size) && (ndim < 3 || hi2 < lo2 + size);
  };
  if (!WARP) {
    double size = 1;
    int lg = 0;
    while (lg < 1100 && !holds(size)) size *= 2, ++lg;
    cube5[0] = (float)lo0, cube5[1] = (float)lo1, cube5[2] = (float)lo2;
    cube5[3] = (float)size, cube5[4] = (float)lg;
    return;
  }
  // lane k tries the size 2^(base + k); past 2^1023 doubling gives infinity
  const auto size_of = [](int k) { return k < 1024 ? __longlong_as_double((long long)(k + 1023) << 52) : (double)INFINITY; };
  int lg = 1100;
  for (int base = 0; base < 1100; base += 32) {
    const int k = base + (int)fl::lane_id();
    const uint32_t fits = __ballot_sync(FL_FULL, k < 1100 && holds(size_of(k)));
    if (fits) {
      lg = base + __ffs(fits) - 1;
      break;
    }
  }
  if (fl::lane_id() == 0) {
    cube5[0] = (float)lo0, cube5[1] = (float)lo1, cube5[2] = (float)lo2;
    cube5[3] = (float)size_of(lg), cube5[4] = (float)lg;
  }
}

// The left-aligned Morton key of p in the cube with the given origin, e = LEVELS - log2(size).
__device__ __forceinline__ uint64_t morton_key(float4 p, const float* origin, int e, int ndim) {
  const int L = levels_of(ndim), bits = L * ndim;
  const uint32_t top = (1u << L) - 1;
  const uint64_t qx = cell_of(p.x, origin[0], e, top);
  uint64_t key;
  if (ndim == 3)
    key = spread3(qx) | spread3(cell_of(p.y, origin[1], e, top)) << 1 |
          spread3(cell_of(p.z, origin[2], e, top)) << 2;
  else if (ndim == 2)
    key = spread2(qx) | spread2(cell_of(p.y, origin[1], e, top)) << 1;
  else
    key = qx;
  return key << (64 - bits);
}

// Bounding box -> d3 cube -> keys; digit histograms of the sort passes in the same read.
constexpr int kMortonThreads = 1024;

__global__ void __launch_bounds__(kMortonThreads) k_morton(const float4* __restrict__ pos, int n,
                                                     int ndim, const FlReduce* red,
                                                     uint64_t* __restrict__ keys,
                                                     uint32_t* __restrict__ vals,
                                                     uint32_t* __restrict__ hist, int lo_bit,
                                                     float* cube_out) {
  __shared__ float s_cube[5];
  __shared__ uint32_t sh[8 * 256];
  const int passes = (64 - lo_bit + 7) / 8;
  if (threadIdx.x < 32) {
    d3_cover<true>(red, ndim, s_cube);
    if (blockIdx.x == 0 && threadIdx.x == 0)
      for (int k = 0; k < 5; ++k) cube_out[k] = s_cube[k];
  }
  for (int i = threadIdx.x; i < 8 * 256; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const int e = levels_of(ndim) - (int)s_cube[4];
  const int stride = gridDim.x * blockDim.x;
  for (int base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const int i = base + threadIdx.x;
    const bool ok = i < n;
    uint64_t key = 0;
    if (ok) {
      key = morton_key(pos[i], s_cube, e, ndim);
      keys[i] = key;
      vals[i] = (uint32_t)i;
    }
    for (int p = 0; p < passes; ++p)
      fl::hist_add(sh + p * 256, (uint32_t)(key >> (lo_bit + 8 * p)) & 255u, ok);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * 256; i += blockDim.x)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// ---- batches of graphs: the per-graph tick values, the keys, and the sort by graph

// One warp per graph (WARP) or one thread: the graph's d3 cube from its bounding box, the walk's threshold, its
// distances, this tick's alpha, its velocity multiplier and its centre force's shift.
template <bool WARP>
__global__ void __launch_bounds__(128) k_bgraph(int graphs, int ndim, const int32_t* __restrict__ off,
                                        const FlReduce* __restrict__ red,
                                        const FlBatchParams* __restrict__ prm,
                                        const double* __restrict__ alpha,
                                        FlGraph* __restrict__ gr) {
  const int g = (blockIdx.x * blockDim.x + threadIdx.x) / (WARP ? 32 : 1);
  if (g >= graphs) return;  // WARP: the whole warp
  FlGraph o;
  const int first = off[g], count = off[g + 1] - off[g];
  if (count > 0) {
    d3_cover<WARP>(red + g, ndim, o.origin);
  } else {
    o.origin[0] = o.origin[1] = o.origin[2] = 0.f, o.size = 1.f, o.lg = 0.f;
  }
  if (WARP && fl::lane_id()) return;
  const FlBatchParams p = prm[g];
  o.T0 = (float)((double)o.size * (double)o.size / p.theta2);
  o.dmin2 = (float)p.dmin2;
  o.dmax2 = p.dmax2 > 3e38 ? INFINITY : (float)p.dmax2;
  o.alpha = (float)alpha[g];
  o.decay = (float)p.decay;
  const double c[3] = {p.cx, p.cy, p.cz};
  for (int k = 0; k < 3; ++k) {
    const double d = k < ndim && count > 0 && p.cstrength != 0 ? (fl::sum_of(red[g], k) / count - c[k]) * p.cstrength : 0.0;
    const float h = (float)d;
    o.shift[k] = make_float2(h, (float)(d - (double)h));
  }
  o.first = first, o.count = count;
  o.frozen = alpha[g] < 0.0 ? 1 : 0;
  o.fx = p.fx;
  o.tick0 = p.tick0;
  o.citer = p.citer, o.cinv = p.cinv, o.cstr = p.cstr;
  o.pad = 0u;
  gr[g] = o;
}

// Morton keys of a batch, each point in its own graph's cube; histograms as k_morton.
__global__ void __launch_bounds__(kMortonThreads) k_bmorton(const float4* __restrict__ pos, int n,
                                                      int ndim, const uint32_t* __restrict__ gid,
                                                      const FlGraph* __restrict__ gr,
                                                      uint64_t* __restrict__ keys,
                                                      uint32_t* __restrict__ vals,
                                                      uint32_t* __restrict__ hist, int lo_bit) {
  __shared__ uint32_t sh[8 * 256];
  const int passes = (64 - lo_bit + 7) / 8;
  for (int i = threadIdx.x; i < 8 * 256; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const int stride = gridDim.x * blockDim.x;
  for (int base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const int i = base + threadIdx.x;
    const bool ok = i < n;
    uint64_t key = 0;
    if (ok) {
      const FlGraph& g = gr[gid[i]];
      key = morton_key(pos[i], g.origin, levels_of(ndim) - (int)g.lg, ndim);
      keys[i] = key;
      vals[i] = (uint32_t)i;
    }
    for (int p = 0; p < passes; ++p)
      fl::hist_add(sh + p * 256, (uint32_t)(key >> (lo_bit + 8 * p)) & 255u, ok);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * 256; i += blockDim.x)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// The graph of node `node`: the last g with off[g] <= node (graph offsets in shared memory).
__device__ __forceinline__ uint32_t graph_of(const int32_t* s_off, int graphs, uint32_t node) {
  int lo = 0, hi = graphs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if ((uint32_t)s_off[mid] <= node) lo = mid;
    else hi = mid - 1;
  }
  return (uint32_t)lo;
}
// The second sort's input: the graph of each point in Morton order, in the top `passes` bytes of the
// key, and the point's Morton-order position; with the histograms of those digits.
constexpr int kGidSearchMax = 8192;  // graphs whose offsets the key kernel searches in shared memory

__global__ void __launch_bounds__(kMortonThreads) k_bgidkey(int n, const uint32_t* __restrict__ mperm,
                                                      const uint32_t* __restrict__ gid,
                                                      const int32_t* __restrict__ off, int graphs,
                                                      int passes, uint64_t* __restrict__ keys,
                                                      uint32_t* __restrict__ vals,
                                                      uint32_t* __restrict__ hist) {
  __shared__ uint32_t sh[2 * 256];
  __shared__ int32_t s_off[kGidSearchMax];
  const bool search = graphs <= kGidSearchMax;
  for (int i = threadIdx.x; i < 2 * 256; i += blockDim.x) sh[i] = 0;
  if (search)
    for (int i = threadIdx.x; i < graphs; i += blockDim.x) s_off[i] = off[i];
  __syncthreads();
  const int stride = gridDim.x * blockDim.x;
  for (int base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const int i = base + threadIdx.x;
    const bool ok = i < n;
    uint64_t key = 0;
    if (ok) {
      // a node's graph: from the offsets (a search in shared memory) rather than a random read
      const uint32_t node = mperm[i];
      key = (uint64_t)(search ? graph_of(s_off, graphs, node) : gid[node]) << (64 - 8 * passes);
      keys[i] = key;
      vals[i] = (uint32_t)i;
    }
    for (int p = 0; p < passes; ++p)
      fl::hist_add(sh + p * 256, (uint32_t)(key >> (64 - 8 * (passes - p))) & 255u, ok);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 2 * 256; i += blockDim.x)
    if (sh[i]) atomicAdd(&hist[i], sh[i]);
}

// The order by (graph, Morton code): position j takes the Morton-order point at order2[j].
__global__ void __launch_bounds__(kThreads) k_bgather(int n, const uint32_t* __restrict__ order2,
                                                      const uint64_t* __restrict__ mkeys,
                                                      const uint32_t* __restrict__ mperm,
                                                      const uint32_t* __restrict__ gid,
                                                      uint64_t* __restrict__ skeys,
                                                      uint32_t* __restrict__ perm,
                                                      uint32_t* __restrict__ gid_pos) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  const uint32_t v = order2[j];
  const uint32_t node = mperm[v];
  skeys[j] = mkeys[v];
  perm[j] = node;
  // graph g's points take sorted positions [off[g], off[g + 1]), the same range its nodes have
  gid_pos[j] = gid[j];
}

// Common prefix of sorted keys i and j (index tie-break), -1 outside [lo, hi] (one graph's range)
__device__ __forceinline__ int kdelta(const uint64_t* __restrict__ k, int lo, int hi, uint64_t ki,
                                      int i, int j) {
  if (j < lo || j > hi) return -1;
  uint64_t kj = k[j];
  return ki != kj ? __clzll(ki ^ kj) : 64 + __clz(i ^ j);
}

// Modular (wrapping) 64-bit arithmetic: in a batch, the prefix over all graphs' records may pass
// 2^63 (each graph has its own scale); the difference of two prefix values within one graph is
// still its exact sum, which that graph's scale keeps below 2^62.
__device__ __forceinline__ long long wadd(long long a, long long b) {
  return (long long)((unsigned long long)a + (unsigned long long)b);
}
__device__ __forceinline__ long long wsub(long long a, long long b) {
  return (long long)((unsigned long long)a - (unsigned long long)b);
}
__device__ __forceinline__ D4 add4(D4 a, D4 b) {
  return mk4(wadd(a.x, b.x), wadd(a.y, b.y), wadd(a.z, b.z), wadd(a.w, b.w));
}
__device__ __forceinline__ D4 shfl_up4(D4 v, int o) {
  return mk4(__shfl_up_sync(FL_FULL, v.x, o), __shfl_up_sync(FL_FULL, v.y, o),
             __shfl_up_sync(FL_FULL, v.z, o), __shfl_up_sync(FL_FULL, v.w, o));
}

// Inclusive prefix of one D4 per thread over a 256-thread block: written to out[i] (i >= 0),
// the block's total to tot[blockIdx.x]. Every thread of the block must call it.
__device__ void block_prefix4(D4 v, D4* out, D4* tot, int i) {
  __shared__ D4 s_warp[kThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    D4 y = shfl_up4(v, o);
    if (lane >= o) v = add4(v, y);
  }
  if (lane == 31) s_warp[warp] = v;
  __syncthreads();
  if (warp) {
    D4 b = s_warp[0];
    for (int w = 1; w < warp; ++w) b = add4(b, s_warp[w]);
    v = add4(v, b);
  }
  if (i >= 0) out[i] = v;
  if (threadIdx.x == kThreads - 1) tot[blockIdx.x] = v;
}

// A sorted point's record for the closed-form cell sums: (|a|, |a| u_x, |a| u_y, |a| u_z) with
// a = strength * c^leafDepth and u = (p - origin) / size in [0, 1) the position in the d3 cube, as
// exact fixed point (scale 2^fe, chosen so that no sum over all points overflows). up, dn: the common
// prefixes with the points after and before.
__device__ __forceinline__ D4 point_record(float4 p, int up, int dn, int ndim, const float* cb, int fe) {
  const int L = levels_of(ndim), bits = L * ndim;
  const int dmx = up > dn ? up : dn;
  const int lD = (dmx >= bits ? L : dmx / ndim) + 1;  // the point's d3 leaf depth
  const float sF = offset_scale(cb);
  const long long W = f2ll_rn(fabsf(p.w * damp(ndim, lD)) * __int_as_float((fe + 127) << 23));
  return mk4(W, mulhi62(W, fx_offset(p.x, cb[0], sF)), ndim > 1 ? mulhi62(W, fx_offset(p.y, cb[1], sF)) : 0,
             ndim > 2 ? mulhi62(W, fx_offset(p.z, cb[2], sF)) : 0);
}

// Internal node i of the graph at sorted positions [lo, hi], lo < hi (i == hi: an index of no tree).
// Karras (2012), "Maximizing parallelism in the construction of BVHs, octrees, and k-d trees": node i
// covers a sorted range [first, last] and splits it where the common prefix grows.
// Returns first, last and the d3 depth of the node's cell.
// A search step asks whether a common prefix is longer than d bits: whether the keys' exclusive or is at
// most its largest value then, a compare instead of a count of leading zeros.
__device__ __forceinline__ uint64_t prefix_mask(int d) { return d < 63 ? ~0ull >> (d + 1) : 0ull; }
// WIDE: 12 and then 7 probes at once, for a few warps an SM, which wait for each probe's latency: 5,300
// clocks for 7,400 at 1,000 points (4 blocks of 256), a tick up to 4 % shorter from 500 to 2,048. Blocks of
// 512 show no difference; with 24 warps an SM, or a chip full of them, the probes' work counts and one at
// a time is faster (10,300 clocks for 11,600 at 5,000 points).
template <bool WIDE>
__device__ __forceinline__ uint3 karras_node(const uint64_t* __restrict__ k, int lo, int hi, uint64_t ki,
                                             int up, int dn, int i, int ndim, uint32_t* left,
                                             uint32_t* right, uint32_t* parent, uint32_t* leaf_parent,
                                             uint32_t* range, uint8_t* depth) {
  const int L = levels_of(ndim), bits = L * ndim;
  if (i == hi) {  // the last point of a graph: this internal index belongs to no tree
    left[i] = right[i] = kNoParent;
    range[2 * i] = range[2 * i + 1] = (uint32_t)i;
    depth[i] = kGapDepth;
    return make_uint3((uint32_t)i, (uint32_t)i, (uint32_t)kGapDepth);
  }
  if (i == lo) parent[i] = (uint32_t)i;  // a graph's root is its own parent
  const int d = up > dn ? 1 : -1;
  const int dmin = up > dn ? dn : up;
  // whether the prefix of keys i and j is longer than `than` bits, m its mask (equal keys: the
  // indices' bits follow)
  const auto longer = [&](int j, int than, uint64_t m) {
    if (WIDE) {  // read in any case: no branch to diverge at
      const int in = min(max(j, lo), hi);
      const uint64_t x = ki ^ k[in];
      return (bool)((in == j) & (x <= m) & ((than < 64) | (64 + __clz(i ^ j) > than)));
    }
    if (j < lo || j > hi) return false;
    const uint64_t x = ki ^ k[j];
    return x <= m && (than < 64 || 64 + __clz(i ^ j) > than);
  };
  const uint64_t mmin = prefix_mask(dmin);
  // the most l with longer(i + l d) (it falls as l grows, and holds for from): below from + w, w a
  // power of two
  const auto farthest = [&](int from, int w, int than, uint64_t m) {
    int l = from;
    if (WIDE) {
      while (w > 1) {
        const int q = w > 8 ? w >> 3 : 1;
        int hits = 0;
#pragma unroll
        for (int e = 1; e < 8; ++e) hits += longer(i + (l + e * q) * d, than, m);
        l += hits * q;
        w = q;
      }
    } else {
      for (int t = w >> 1; t >= 1; t >>= 1)
        if (longer(i + (l + t) * d, than, m)) l += t;
    }
    return l;
  };
  int lmax = 1;  // below 2^28, as the indices are
  if (WIDE) {
    int hits = 0;
#pragma unroll
    for (int e = 1; e < 13; ++e) hits += longer(i + d * (1 << e), dmin, mmin);  // kSmallTreeMax < 2^13
    lmax = 1 << hits;
  } else {
    while (longer(i + 2 * lmax * d, dmin, mmin)) lmax *= 2;
  }
  const int len = farthest(lmax, lmax, dmin, mmin);
  const int j = i + len * d;
  const int dnode = kdelta(k, lo, hi, ki, i, j);
  const int s = farthest(0, 1 << (32 - __clz(len)), dnode, prefix_mask(dnode));
  const int split = i + s * d + (d < 0 ? -1 : 0);
  const int first = i < j ? i : j, last = i < j ? j : i;
  uint32_t l = first == split ? (kLeaf | (uint32_t)split) : (uint32_t)split;
  uint32_t r = last == split + 1 ? (kLeaf | (uint32_t)(split + 1)) : (uint32_t)(split + 1);
  left[i] = l, right[i] = r;
  if (l & kLeaf) leaf_parent[l & kIndex] = (uint32_t)i;
  else parent[l] = (uint32_t)i;
  if (r & kLeaf) leaf_parent[r & kIndex] = (uint32_t)i;
  else parent[r] = (uint32_t)i;
  range[2 * i] = (uint32_t)first, range[2 * i + 1] = (uint32_t)last;
  int dep = dnode >= bits ? L : dnode / ndim;
  dep = dep > L ? L : dep;
  depth[i] = (uint8_t)dep;
  return make_uint3((uint32_t)first, (uint32_t)last, (uint32_t)dep);
}

// The binary radix tree over the sorted keys (karras_node): thread i takes internal node i, or gathers
// sorted point i and, for the closed-form cell sums, its record (point_record), prefix-summed within
// the block. Integer sums are exact, and cheap where FP64 is not.
// PART: 1, the points (sorted leaves, records, their block prefix); 2, the internal nodes.
// 6 blocks per SM (40 registers): the points' half 28.1 -> 26.5 us at 1M nodes, the heads (below)
// 30.3 -> 28.5; 8 blocks (32 registers) spill, 26.8 and 30.2.
constexpr int kTreeBlocks = 6;
template <int PART>
__global__ void __launch_bounds__(kThreads, kTreeBlocks) k_build(
    const uint64_t* __restrict__ k, const uint32_t* __restrict__ perm,
    const float4* __restrict__ pos, const float* __restrict__ strength, int n, int ndim,
    uint32_t* __restrict__ left, uint32_t* __restrict__ right, uint32_t* __restrict__ parent,
    uint32_t* __restrict__ leaf_parent, uint32_t* __restrict__ range, uint8_t* __restrict__ depth,
    uint32_t* __restrict__ omask, float4* __restrict__ leaf, D4* __restrict__ wsum, D4* __restrict__ wtot,
    const float* __restrict__ cube, int fx_exp, FlSegs seg) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  // the sorted range of this point's graph (a batch), and that graph's cube
  int lo = 0, hi = n - 1;
  const float* cb = cube;
  int fe = fx_exp;
  if (seg.graphs && i < n) {
    const uint32_t g = seg.gid_pos[i];
    lo = seg.off[g], hi = seg.off[g + 1] - 1;
    cb = seg.g[g].origin;
    fe = seg.g[g].fx;
  }
  const uint64_t ki = i < n ? k[i] : 0;
  const int up = i < n ? kdelta(k, lo, hi, ki, i, i + 1) : -1;
  const int dn = i < n ? kdelta(k, lo, hi, ki, i, i - 1) : -1;
  if (PART == 1 && i < n && lo == hi) leaf_parent[i] = kNoParent;  // alone in its graph: no tree
  D4 wrec = mk4(0, 0, 0, 0);
  if (PART == 1 && i < n) {
    const uint32_t node = perm[i];
    float4 p = pos[node];
    p.w = strength[node];
    leaf[i] = p;
    if (wsum) wrec = point_record(p, up, dn, ndim, cb, fe);
  }
  if (PART == 1 && wsum)  // block-uniform
    block_prefix4(wrec, wsum, wtot, i < n ? i : -1);
  if (PART == 1 || i >= n - 1) return;
  omask[i] = 0u;  // k_frontier marks the octants
  karras_node<false>(k, lo, hi, ki, up, dn, i, ndim, left, right, parent, leaf_parent, range, depth);
}

// Every binary node below the root that is a d3 child (a point, or an internal node deeper than
// its parent: the first node of another cell) finds the head of its parent's cell, climbing the
// binary nodes of equal depth, and marks its octant (its keys' digit at the parent's depth) in
// the head's octant mask. Returns head | octant << 27 | 1 << 31 for the slots, 0 for other nodes.
// pt: x is a point (sorted order), else an internal node.
// p: its binary parent; first_of(): its first point.
template <class First>
__device__ __forceinline__ uint32_t frontier_of(bool pt, uint32_t x, uint32_t p, First first_of, int ndim,
                                                const uint64_t* skeys, const uint32_t* parent,
                                                const uint8_t* depth, uint32_t* omask, uint32_t* err) {
  // the parent cell's binary node: none for a graph's root, an index between two graphs, or a
  // point alone in its graph
  if (p == kNoParent || (!pt && (p == x || depth[x] == kGapDepth))) return 0u;
  const int Dp = depth[p];
  if (!pt && depth[x] <= Dp) return 0u;
  uint32_t h = p;
  for (int guard = 0;; ++guard) {  // equal depths: splits inside one cell
    const uint32_t up = parent[h];
    if (up == h || depth[up] < Dp) break;
    h = up;
    if (guard > 64) {
      atomicOr(err, FL_ERR_TREE);
      break;
    }
  }
  uint32_t oct = 0;
  if (Dp < levels_of(ndim)) {
    const uint64_t k = skeys[first_of()];
    oct = (uint32_t)(k >> (64 - ndim * (Dp + 1))) & ((1u << ndim) - 1u);
    atomicOr(omask + h, (1u << oct) | (pt ? 0u : 1u << (16 + oct)));  // cells also above
  }
  return h | (oct << 27) | 0x80000000u;
}

// Threads [0, n-1) take the internal nodes, [n-1, 2n-1) the points.
__global__ void __launch_bounds__(kThreads) k_frontier(
    int n, int ndim, const uint64_t* __restrict__ skeys, const uint32_t* __restrict__ parent,
    const uint32_t* __restrict__ leaf_parent, const uint32_t* __restrict__ range,
    const uint8_t* __restrict__ depth, uint32_t* __restrict__ omask,
    uint32_t* __restrict__ head_of, uint32_t* err) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 2 * n - 1) return;
  const bool pt = t >= n - 1;
  const uint32_t x = pt ? (uint32_t)(t - (n - 1)) : (uint32_t)t;
  head_of[t] = frontier_of(pt, x, pt ? leaf_parent[x] : parent[x], [&] { return pt ? x : range[2 * x]; }, ndim,
                           skeys, parent, depth, omask, err);
}

// Exclusive prefix of the block totals, in place, by one block of kTopThreads: each thread sums
// a run of consecutive totals, a warp-shuffle scan of the threads' sums (two levels) gives each
// run its start, and the thread rewrites its run. For the child counts (u32) and the
// fixed-point point records (D4).
constexpr int kTopThreads = 1024;
__device__ __forceinline__ uint32_t top_add(uint32_t a, uint32_t b) { return a + b; }
__device__ __forceinline__ D4 top_add(D4 a, D4 b) { return add4(a, b); }
__device__ __forceinline__ uint32_t top_up(uint32_t v, int o) { return __shfl_up_sync(FL_FULL, v, o); }
__device__ __forceinline__ D4 top_up(D4 v, int o) { return shfl_up4(v, o); }

template <typename T>
__device__ __forceinline__ void top_scan(T* tot, int nb, T zero) {
  __shared__ T s_warp[kTopThreads / 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (nb + kTopThreads - 1) / kTopThreads, a = threadIdx.x * per;
  const int b = a + per < nb ? a + per : nb;
  T sum = zero;
#pragma unroll 8
  for (int t = a; t < b; ++t) sum = top_add(sum, tot[t]);
  T x = sum;  // inclusive scan within the warp
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = top_up(x, o);
    if (lane >= o) x = top_add(x, y);
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {  // inclusive scan of the warp totals
    T w = s_warp[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const T y = top_up(w, o);
      if (lane >= o) w = top_add(w, y);
    }
    s_warp[lane] = w;
  }
  __syncthreads();
  T run = warp ? s_warp[warp - 1] : zero;
  const T y = top_up(x, 1);  // exclusive within the warp: the previous lane's inclusive sum
  if (lane) run = top_add(run, y);
#pragma unroll 8
  for (int t = a; t < b; ++t) {
    const T v = tot[t];
    tot[t] = run;
    run = top_add(run, v);
  }
}

__global__ void __launch_bounds__(kTopThreads) k_top_u32(uint32_t* tot, int nb) {
  top_scan<uint32_t>(tot, nb, 0u);
}

__global__ void __launch_bounds__(kTopThreads) k_top4(D4* tot, int nb) {
  top_scan<D4>(tot, nb, mk4(0, 0, 0, 0));
}

// first child slot of head x: slots [0, roots) hold the roots (one per graph), children follow
// in head order
__device__ __forceinline__ uint32_t first_slot(const uint32_t* first, const uint32_t* ctot,
                                               uint32_t x, uint32_t roots) {
  return roots + first[x] + ctot[x >> 8];
}

// The cell of a head of depth D in closed form (strengths of one sign, `sign`): its centroid and its
// value at its own depth. hi, lo: the prefix sums up to its last point and before its first, p0; in
// fixed point, exact.
__device__ __forceinline__ float4 closed_cell(D4 hi, D4 lo, float4 p0, int D, int ndim, float sign,
                                              const float* __restrict__ cube, int fe) {
  const long long W = wsub(hi.x, lo.x);
  float4 out;
  if (W > 0) {
    // centroid = p0 + size * sum(w (u - u0)) / sum(w), about the range's first point p0: the
    // integer sums give the offsets exactly, so FP32 keeps the precision of the cell, not the cube
    const float fW = ll2f_rn(W);
    const float sF = offset_scale(cube), r = cube[3] / fW;
    out.x = p0.x + ll2f_rn(wsub(wsub(hi.y, lo.y), mulhi62(W, fx_offset(p0.x, cube[0], sF)))) * r;
    out.y = ndim > 1 ? p0.y + ll2f_rn(wsub(wsub(hi.z, lo.z), mulhi62(W, fx_offset(p0.y, cube[1], sF)))) * r : 0.f;
    out.z = ndim > 2 ? p0.z + ll2f_rn(wsub(wsub(hi.w, lo.w), mulhi62(W, fx_offset(p0.z, cube[2], sF)))) * r : 0.f;
    out.w = sign * fW * __int_as_float((127 - fe) << 23) * damp(ndim, -D);
  } else {
    out = p0;
    out.w = 0.f;
  }
  return out;
}

// Whether internal node i of depth D, binary parent pa, heads a d3 cell: a graph's root, or the first
// node of a deeper cell.
__device__ __forceinline__ bool is_head(uint32_t i, int D, uint32_t pa, const uint8_t* depth) {
  return D != kGapDepth && (pa == i || depth[pa] < D);
}
// The d3 children of a head's cell: its occupied octants; at the deepest level, where the keys are
// equal, its points.
__device__ __forceinline__ uint32_t children_of(int D, int ndim, uint32_t om, uint32_t points) {
  return D >= levels_of(ndim) ? points : (uint32_t)__popc(om & 0xffffu);
}

// Every head's count of children; the counts' exclusive prefix within the block (first[]) and the block's total (ctot[]), for the slots. CLOSED (strengths
// of one sign): a head's cell from the prefix sums too (closed_cell), into cell[].
template <bool CLOSED>
__global__ void __launch_bounds__(kThreads, kTreeBlocks) k_heads(int n, int ndim,
                                                    const uint32_t* __restrict__ parent,
                                                    const uint32_t* __restrict__ range,
                                                    const uint8_t* __restrict__ depth,
                                                    const uint32_t* __restrict__ omask,
                                                    uint32_t* __restrict__ count,
                                                    uint32_t* __restrict__ first,
                                                    uint32_t* __restrict__ ctot, float sign,
                                                    const D4* __restrict__ P,
                                                    const D4* __restrict__ Ptot,
                                                    const float4* __restrict__ leaf,
                                                    const float* __restrict__ cube, int fx_exp,
                                                    float4* __restrict__ cell,
                                                    uint32_t* __restrict__ arrive, FlSegs seg) {
  __shared__ uint32_t s_warp[kThreads / 32];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t c = 0;
  if (i < n - 1) {
    const int D = depth[i];
    if (is_head((uint32_t)i, D, parent[i], depth)) {
      const uint32_t a = range[2 * i], b = range[2 * i + 1];
      c = children_of(D, ndim, omask[i], b - a + 1);
      if (CLOSED && c) {
        const FlGraph* gr = seg.graphs ? seg.g + seg.gid_pos[a] : nullptr;
        // prefix sums: within the 256-point block, plus the blocks before it
        cell[i] = closed_cell(add4(P[b], Ptot[b >> 8]), a ? add4(P[a - 1], Ptot[(a - 1) >> 8]) : mk4(0, 0, 0, 0),
                              leaf[a], D, ndim, sign, gr ? gr->origin : cube, gr ? gr->fx : fx_exp);
      }
    }
    count[i] = c;
    if (!CLOSED) arrive[i] = 0u;  // the recursion's arrivals
  }
  uint32_t x = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(FL_FULL, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  uint32_t before = 0;
  for (int w = 0; w < warp; ++w) before += s_warp[w];
  if (i < n - 1) first[i] = before + x - c;
  if (threadIdx.x == kThreads - 1) ctot[blockIdx.x] = before + x;
}

// The recursion itself (strengths of both signs), over the d3 cells from the deepest up, reading
// each head's children from its slots (k_slots has written the points and every slot's meta).
// A warp owns kUpNodes consecutive binary nodes and starts with its heads without child cells. A
// finished cell writes itself into its slot among its parent's children and counts itself in at the
// parent; the last of the parent's child cells to arrive (their octants are the high half of the
// parent's octant mask) puts the parent on its warp's queue in shared memory, and the warp works
// through the queue a round at a time, one head per lane, until it is empty. The binary nodes of
// a cell over the sorted points [a, b] lie in a .. b (its own is a or b), so a parent whose points
// lie in the warp's range has all its cells there: they count in shared memory, ordered by the
// rounds. Only the cells above count in global memory, by a device-wide acquire-release, which
// waits for the stores before it to reach L2.
// So the chain of dependent steps is the d3 depth, and a round's heads sit on consecutive lanes: FP64
// runs at 2 lanes per clock per SM, and a warp instruction costs its 16 clocks however few of its
// lanes are active. Bound by that and by the chain of loads, counts and rounds: 300,000 points took
// 114 us with one list of starts, every count in global memory and rounds of whole blocks, and take
// 94 (ncu); a tick alone 499 -> 476 us.
// A head combines its children as accumulate() does (src/manyBody.js:42-71). With
// fp64_depth > 0 every value is d3's FP64 number bit for bit: the children's values summed in
// slot order, which is d3's octant order (z << 2 | y << 1 | x), a chain of one-child cells
// scaled by c once per level, the sum scaled by c (c1, d3's Math.sqrt(4 / 2^dims), correctly
// rounded); each cell's FP64 value rides in slot64 beside its slot (a point's strength too,
// converted by k_slots on full warps). So a cell whose children cancel is skipped
// (`!quad.value`, src/manyBody.js:74) exactly when d3 skips it: a cancellation can leave d3 an
// FP64 residual, a value that d3 opens like any other. Centroids are weighted by the FP32
// values, summed in FP64 above fp64_depth and in FP32 below. fp64_depth 0 runs all of it in
// FP32 (values within 2^-20 of their children's |values| count as 0), for precision
// comparisons.
constexpr uint32_t kNoHead = 0xffffffffu;
// Nodes per warp: 256, with eight children's slots loaded together, takes 87 us alone, but its 120
// registers slow the tick beside others' (316 us for 312).
constexpr int kUpThreads = 128, kUpWarps = kUpThreads / 32, kUpNodes = 128;

// One head of the recursion: combine its children into its cell, write the cell into its slot
// and count it in at its parent. Returns the parent when this was its last child cell to
// arrive, else kNoHead (also after a graph's root, and on a malformed tree).
__device__ __forceinline__ uint32_t cells_up_one(
    uint32_t h, int n, int ndim, const uint32_t* __restrict__ head_of,
    const uint32_t* __restrict__ omask, const uint8_t* __restrict__ depth,
    const uint32_t* __restrict__ count, const uint32_t* __restrict__ first,
    const uint32_t* __restrict__ ctot, const uint32_t* __restrict__ range,
    uint32_t* __restrict__ arrive, uint32_t* s_arrive, uint32_t lo, float4* cdata,
    const uint2* __restrict__ cmeta, double* slot64, int fp64_depth, double c1, uint32_t* err,
    const FlSegs& seg) {
  const uint32_t roots = seg.graphs ? (uint32_t)seg.graphs : 1u;
  const uint32_t nslots = 2u * (uint32_t)n + 1u;
  const bool exact = fp64_depth > 0;
  const int D = depth[h];
  const uint32_t cnt = count[h], fs = first_slot(first, ctot, h, roots);
  // the parent's record: its loads overlap the children's
  const uint32_t rec = head_of[h];
  const bool root = !(rec & 0x80000000u);
  const uint32_t p = rec & kCountMask, oct = (rec >> 27) & 15u;
  uint32_t pcnt = 0, pfirst = 0, ptot = 0, pmask = 0;
  uint2 prange = make_uint2(0u, 0u);
  if (!root) {
    pcnt = count[p], pfirst = first[p], ptot = ctot[p >> 8], pmask = omask[p];
    prange = reinterpret_cast<const uint2*>(range)[p];
  }
  if (fs + cnt > nslots) {  // a malformed tree
    atomicOr(err, FL_ERR_TREE);
    return kNoHead;
  }
  const bool wide = D < fp64_depth;
  double sv = 0, sa = 0, sx = 0, sy = 0, sz = 0;
  float fv = 0, fa = 0, fx = 0, fy = 0, fz = 0;
  float4 firstpos = make_float4(0, 0, 0, 0);
  for (uint32_t j = 0; j < cnt; ++j) {
    const uint2 m = cmeta[fs + j];
    const float4 q = __ldcg(cdata + fs + j);
    double v = exact ? __ldcg(slot64 + fs + j) : 0.0;  // a point's strength, as k_slots wrote it, or a cell's value
    float v32 = q.w;  // the centroid weight's value
    if (m.y != kLeafMark) {
      // the chain of one-child cells from D + 1 down to the child's depth scales by c
      const int cd = (int)(m.y >> 26);
      v32 *= damp(ndim, cd - D - 1);
      if (exact)
        for (int l = cd - D - 1; l > 0; --l) v *= c1;
    }
    if (j == 0) firstpos = q;
    const float a = fabsf(v32);
    if (exact) {
      // d3 skips children whose value is 0 (or NaN): tested on the bits
      const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
      if (b == 0 || b > 0x7ff0000000000000ull) continue;
      sv += v;
    } else {
      if (!(a > 0.f)) continue;
      fv += v32;
    }
    fa += a;
    if (wide) sa += a, sx += (double)a * q.x, sy += (double)a * q.y, sz += (double)a * q.z;
    else fx += a * q.x, fy += a * q.y, fz += a * q.z;
  }
  float4 out;
  if (wide)
    out = sa > 0 ? make_float4((float)(sx / sa), (float)(sy / sa), (float)(sz / sa), 0.f) : firstpos;
  else
    out = fa > 0.f ? make_float4(fx / fa, fy / fa, fz / fa, 0.f) : firstpos;
  double val = 0;
  if (exact) {
    val = sv * c1;
    out.w = (float)val;
    // a residual below FP32's range stays a value the walk does not skip
    if (val != 0 && out.w == 0.f) out.w = copysignf(1.17549435e-38f, (float)val);
  } else {
    out.w = fabsf(fv) <= fa * 0x1p-20f ? 0.f : (float)((double)fv * c1);
  }
  if (root) {  // a graph's root: its own slot
    cdata[seg.graphs ? seg.gid_pos[h] : 0u] = out;
    return kNoHead;
  }
  const uint32_t pfs = roots + pfirst + ptot;
  const uint32_t rank = (uint32_t)__popc(pmask & ((1u << oct) - 1u)), slot = pfs + rank;
  if (rank >= pcnt || pfs + pcnt > nslots) {  // a malformed tree
    atomicOr(err, FL_ERR_TREE);
    return kNoHead;
  }
  cdata[slot] = out;
  if (exact) slot64[slot] = val;
  if (prange.x >= lo && prange.y < lo + kUpNodes)  // all its binary nodes are the warp's
    return atomicAdd(&s_arrive[p - lo], 1u) + 1u == (uint32_t)__popc(pmask >> 16) ? p : kNoHead;
  // acquire-release: each arrival publishes its cell; the last sees all of them
  const uint32_t w = cuda::atomic_ref<uint32_t, cuda::thread_scope_device>(arrive[p])
                         .fetch_add(1u, cuda::memory_order_acq_rel);
  return w + 1u == (uint32_t)__popc(pmask >> 16) ? p : kNoHead;
}

__global__ void __launch_bounds__(kUpThreads) k_cells_up(
    int n, int ndim, const uint32_t* __restrict__ head_of, const uint32_t* __restrict__ omask,
    const uint8_t* __restrict__ depth, const uint32_t* __restrict__ count,
    const uint32_t* __restrict__ first, const uint32_t* __restrict__ ctot,
    const uint32_t* __restrict__ range, uint32_t* __restrict__ arrive, float4* cdata,
    const uint2* __restrict__ cmeta, double* slot64, int fp64_depth, double c1, uint32_t* err,
    FlSegs seg) {
  // per warp: this round's heads and the next one's, and the arrivals at its own cells
  __shared__ uint32_t s_queue[kUpWarps][2][kUpNodes];
  __shared__ uint32_t s_arrive[kUpWarps][kUpNodes];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t below_me = (1u << lane) - 1u;
  const uint32_t lo = (blockIdx.x * kUpWarps + warp) * kUpNodes;
  uint32_t len = 0;
  for (uint32_t k = 0; k < kUpNodes; k += 32) {
    const uint32_t i = lo + k + lane;
    s_arrive[warp][k + lane] = 0u;
    const bool start = i < (uint32_t)(n - 1) && count[i] && (depth[i] >= levels_of(ndim) || !(omask[i] >> 16));
    const uint32_t b = __ballot_sync(FL_FULL, start);
    if (start) s_queue[warp][0][len + __popc(b & below_me)] = i;
    len += __popc(b);
  }
  for (int round = 0; len; ++round) {
    if (round > 64) {  // deeper than any d3 tree: a malformed tree
      if (lane == 0) atomicOr(err, FL_ERR_TREE);
      return;
    }
    __syncwarp();
    const uint32_t* now = s_queue[warp][round & 1];
    uint32_t* later = s_queue[warp][~round & 1];
    uint32_t more = 0;
    for (uint32_t k = 0; k < len; k += 32) {
      uint32_t next = kNoHead;
      if (k + lane < len)
        next = cells_up_one(now[k + lane], n, ndim, head_of, omask, depth, count, first, ctot, range, arrive,
                            s_arrive[warp], lo, cdata, cmeta, slot64, fp64_depth, c1, err, seg);
      const uint32_t b = __ballot_sync(FL_FULL, next != kNoHead);
      if (next != kNoHead) later[more + __popc(b & below_me)] = next;
      more += __popc(b);
    }
    len = more;
  }
}

// Child x (frontier record rec) writes itself into its slot of its head's cell: the head's first slot
// plus the child's rank (occupied octants before its own; at the deepest level, its place in the
// range). l: the point, or the cell (CELL: its own; else the recursion writes it later).
template <bool CELL>
__device__ __forceinline__ void write_slot(bool pt, uint32_t x, uint32_t rec, int n, int ndim, uint32_t roots,
                                           const uint32_t* omask, const uint32_t* range,
                                           const uint8_t* depth, const uint32_t* count,
                                           const uint32_t* first, const uint32_t* ctot, const float4* l,
                                           float4* cdata, uint2* cmeta, double* slot64, uint32_t* err) {
  if (!(rec & 0x80000000u)) return;
  const uint32_t h = rec & kCountMask, oct = (rec >> 27) & 15u;
  const uint32_t rank = depth[h] >= levels_of(ndim)
                            ? (pt ? x : range[2 * x]) - range[2 * h]
                            : (uint32_t)__popc(omask[h] & ((1u << oct) - 1u));
  const uint32_t slot = first_slot(first, ctot, h, roots) + rank;
  if (rank >= count[h] || slot >= 2u * (uint32_t)n + 1u) {  // a malformed tree
    atomicOr(err, FL_ERR_TREE);
    return;
  }
  if (pt) {
    const float4 p = *l;
    cdata[slot] = p;
    // the recursion's FP64 value of the point, converted here on full warps
    if (slot64) slot64[slot] = (double)p.w;
    cmeta[slot] = make_uint2(x, kLeafMark);
  } else {
    if (CELL) cdata[slot] = *l;
    cmeta[slot] = make_uint2(first_slot(first, ctot, x, roots), count[x] | ((uint32_t)depth[x] << 26));
  }
}

// Every d3 child into its slot; a root also fills its own. Threads as in k_frontier.
__global__ void __launch_bounds__(kThreads) k_slots(
    int n, int ndim, const uint32_t* __restrict__ head_of, const uint32_t* __restrict__ omask,
    const uint32_t* __restrict__ parent,
    const uint32_t* __restrict__ range, const uint8_t* __restrict__ depth,
    const uint32_t* __restrict__ count, const uint32_t* __restrict__ first,
    const uint32_t* __restrict__ ctot, const float4* __restrict__ cell,
    const float4* __restrict__ leaf, float4* __restrict__ cdata, uint2* __restrict__ cmeta,
    uint32_t* err, FlSegs seg, bool cells_later, double* __restrict__ slot64) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 2 * n - 1) return;
  const bool pt = t >= n - 1;
  const uint32_t x = pt ? (uint32_t)(t - (n - 1)) : (uint32_t)t;
  const uint32_t roots = seg.graphs ? (uint32_t)seg.graphs : 1u;
  if (!pt && depth[x] != kGapDepth && parent[x] == x) {  // a graph's root: its own slot
    const uint32_t rs = seg.graphs ? seg.gid_pos[x] : 0u;
    if (!cells_later) cdata[rs] = cell[x];
    cmeta[rs] = make_uint2(first_slot(first, ctot, x, roots), count[x] | ((uint32_t)depth[x] << 26));
  }
  const uint32_t rec = head_of[t];
  const float4* l = pt ? leaf + x : cell + x;
  if (cells_later)
    write_slot<false>(pt, x, rec, n, ndim, roots, omask, range, depth, count, first, ctot, l, cdata, cmeta,
                      slot64, err);
  else
    write_slot<true>(pt, x, rec, n, ndim, roots, omask, range, depth, count, first, ctot, l, cdata, cmeta,
                     slot64, err);
}

// The whole tree of a layout of up to kSmallTreeMax points in one launch: one cluster of up to 8
// blocks, a point per thread, a cluster barrier where the passes of a large layout are launches
// (the bodies are theirs, and so are the arrays left in global memory). Blocks own kSmallRun * k
// consecutive points (by input, then by sorted order).
//   keys    each run of 256 sorted by a bitonic network (shuffles below a warp), the runs of a block
//           merged by binary searches among each other, then the blocks' slices the same way: a
//           pair's place is its place in its slice plus the pairs before it in the others (equal
//           keys: those of earlier inputs, which keeps the order of a stable sort)
//   nodes   Karras' searches on all the sorted keys in shared memory
// The rest reads what other blocks wrote after a cluster barrier (release / acquire).
// Bound by the chain of dependent steps, not by work: a launch, and an L2 round trip per pass. Against
// eight launches and two memsets (the keys, a sort by counting, the tree's passes) a tick went from
// 20.5 to 14.3 us at 1,000 points and from 44.9 to 34.3 at 5,000 (2D, with collide).
constexpr int kSmallRun = 256, kSmallMaxThreads = 768, kSmallBlocks = 8;
static_assert(kSmallTreeMax == kSmallMaxThreads * kSmallBlocks, "a point per thread");
struct SmallTree {
  const float4* pos;
  const float* strength;
  const FlReduce* red;
  FlReduce* zero;  // a record to clear, or null
  uint64_t *tmp, *keys;
  uint32_t *vtmp, *perm;
  float* cube;
  uint32_t* err;
  FlTreeBufs t;
  float sign;
  int fx_exp;
  bool slots64;
};

// the keys among sorted a[0, len) before key: the smaller ones, and the equal ones with ties
__device__ __forceinline__ int keys_before(const uint64_t* a, int len, uint64_t key, bool ties, int top) {
  int at = 0;
  for (int step = top; step; step >>= 1) {
    const int q = at + step;
    if (q <= len) {
      const uint64_t o = a[q - 1];
      if (o < key || (ties && o == key)) at = q;
    }
  }
  return at;
}

__host__ __device__ constexpr int small_align(int n) { return (n + 15) & ~15; }  // entries, to whole vectors
// bytes of global memory into shared memory by a whole block, 16 at a time (the arrays' ends are padded)
__device__ __forceinline__ void to_shared(void* dst, const void* src, int bytes) {
  for (int j = threadIdx.x; j * 16 < bytes; j += blockDim.x)
    reinterpret_cast<uint4*>(dst)[j] = reinterpret_cast<const uint4*>(src)[j];
}

template <bool CLOSED>
__global__ void __launch_bounds__(kSmallMaxThreads) k_small_tree(const SmallTree a) {
  // a slice's pairs in exchange; then every sorted key, and every node's parent and depth
  extern __shared__ __align__(16) uint64_t s_key[];
  uint32_t* s_parent = reinterpret_cast<uint32_t*>(s_key + small_align(a.t.n));
  uint8_t* s_depth = reinterpret_cast<uint8_t*>(s_parent + small_align(a.t.n));
  __shared__ float s_cube[5];
  __shared__ D4 s_warp4[kSmallMaxThreads / 32];
  __shared__ uint32_t s_warp[kSmallMaxThreads / 32];
  __shared__ D4 s_base4[kSmallTreeMax / 256];
  __shared__ uint32_t s_base[kSmallTreeMax / 256];
  namespace cg = cooperative_groups;
  const int n = a.t.n, ndim = a.t.ndim, S = blockDim.x, C = gridDim.x, c = blockIdx.x;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int i = c * S + tid;  // this thread's point, sorted point and internal node
  const bool ok = i < n, node = i < n - 1;
  const int used = (n + S - 1) / S;  // blocks with points
  auto sync = [&] {
    if (C > 1) cg::this_cluster().sync();
    else __syncthreads();
  };
  const uint32_t idx0 = (uint32_t)i;
  float4 p = ok ? a.pos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  if (warp == 0) {
    d3_cover<true>(a.red, ndim, s_cube);
    if (c == 0 && lane == 0)
      for (int k = 0; k < 5; ++k) a.cube[k] = s_cube[k];
  }
  if (a.zero && c == C - 1)
    for (int k = tid; k < (int)(sizeof(FlReduce) / 4); k += S) reinterpret_cast<uint32_t*>(a.zero)[k] = 0u;
  __syncthreads();
  // ---- keys, sorted by (key, input)
  uint64_t key = ok ? morton_key(p, s_cube, levels_of(ndim) - (int)s_cube[4], ndim) : ~0ull;
  uint32_t idx = idx0;  // past the end: the largest key and input of all, so they end last
  uint32_t* s_idx = reinterpret_cast<uint32_t*>(s_key + S);
  const int r = tid & (kSmallRun - 1);
  for (int k = 2; k <= kSmallRun; k <<= 1)
    for (int j = k >> 1; j; j >>= 1) {
      uint64_t ko;
      uint32_t io;
      if (j >= 32) {  // block-uniform
        __syncthreads();
        s_key[tid] = key, s_idx[tid] = idx;
        __syncthreads();
        ko = s_key[tid ^ j], io = s_idx[tid ^ j];
      } else {
        ko = __shfl_xor_sync(FL_FULL, key, j), io = __shfl_xor_sync(FL_FULL, idx, j);
      }
      const bool greater = key > ko || (key == ko && idx > io);
      if (((r & j) == 0) == ((r & k) == 0) ? greater : !greater) key = ko, idx = io;
    }
  if (S > kSmallRun) {  // the block's runs into its slice's order
    __syncthreads();
    s_key[tid] = key;
    __syncthreads();
    int at = r;
    for (int q = 0; q < S; q += kSmallRun)
      if (q != tid - r) at += keys_before(s_key + q, kSmallRun, key, q < tid - r, kSmallRun);
    __syncthreads();
    s_key[at] = key, s_idx[at] = idx;
    __syncthreads();
    key = s_key[tid], idx = s_idx[tid];
  }
  if (ok) {
    p = a.pos[idx];
    p.w = a.strength[idx];
  }
  if (C > 1) {
    if (ok) a.tmp[i] = key;
    sync();
    to_shared(s_key, a.tmp, 8 * n);
    __syncthreads();
  }
  if (ok) {
    int place = tid;
    for (int q = 0; q < used; ++q)
      if (q != c) place += keys_before(s_key + q * S, min(S, n - q * S), key, q < c, S >= 512 ? 512 : 256);
    a.keys[place] = key;
    a.perm[place] = idx;
    a.t.leaf[place] = p;
  }
  sync();
  if (ok) p = a.t.leaf[i];
  to_shared(s_key, a.keys, 8 * n);
  __syncthreads();
  // ---- the binary tree, and the points' records
  key = ok ? s_key[i] : 0;
  const int up = ok ? kdelta(s_key, 0, n - 1, key, i, i + 1) : -1;
  const int dn = ok ? kdelta(s_key, 0, n - 1, key, i, i - 1) : -1;
  if (CLOSED) {
    D4 v = mk4(0, 0, 0, 0);
    if (ok) v = point_record(p, up, dn, ndim, s_cube, a.fx_exp);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const D4 y = shfl_up4(v, o);
      if (lane >= o) v = add4(v, y);
    }
    if (lane == 31) s_warp4[warp] = v;
    __syncthreads();
    for (int w = 0; w < warp; ++w) v = add4(v, s_warp4[w]);
    if (ok) reinterpret_cast<D4*>(a.t.wsum)[i] = v;
    if (tid == S - 1 && c < used) reinterpret_cast<D4*>(a.t.wtiles)[c] = v;
  }
  uint3 me = make_uint3(0u, 0u, (uint32_t)kGapDepth);  // the node's first and last point, its depth
  if (node) {
    a.t.omask[i] = 0u;
    if (!CLOSED) a.t.flag[i] = 0u;
    if (S == kSmallRun)
      me = karras_node<true>(s_key, 0, n - 1, key, up, dn, i, ndim, a.t.left, a.t.right, a.t.parent,
                             a.t.leaf_parent, a.t.range, a.t.depth);
    else
      me = karras_node<false>(s_key, 0, n - 1, key, up, dn, i, ndim, a.t.left, a.t.right, a.t.parent,
                              a.t.leaf_parent, a.t.range, a.t.depth);
  }
  sync();
  // ---- the heads of the children's cells, and the heads' cells
  const uint32_t up_point = ok ? a.t.leaf_parent[i] : kNoParent;
  const D4* P = reinterpret_cast<const D4*>(a.t.wsum);
  D4 hi = mk4(0, 0, 0, 0), lo = mk4(0, 0, 0, 0);
  float4 p0 = make_float4(0.f, 0.f, 0.f, 0.f);
  if (CLOSED && node) {  // for its cell, if it heads one: loads on their way beside the copies
    hi = P[me.y], p0 = a.t.leaf[me.x];
    if (me.x) lo = P[me.x - 1];
  }
  to_shared(s_parent, a.t.parent, 4 * (n - 1));
  to_shared(s_depth, a.t.depth, n - 1);
  if (CLOSED && tid < (n + 255) / 256) {  // the records of the blocks before, per 256 points
    D4 b = mk4(0, 0, 0, 0);
    for (int q = 0; q < tid * 256 / S; ++q) b = add4(b, reinterpret_cast<const D4*>(a.t.wtiles)[q]);
    s_base4[tid] = b;
  }
  __syncthreads();
  const uint32_t nrec = node ? frontier_of(false, i, s_parent[i], [&] { return me.x; }, ndim, s_key, s_parent,
                                           s_depth, a.t.omask, a.err) : 0u;
  const uint32_t prec = ok ? frontier_of(true, i, up_point, [&] { return (uint32_t)i; }, ndim, s_key, s_parent,
                                         s_depth, a.t.omask, a.err) : 0u;
  if (!CLOSED && node) a.t.head_of[i] = nrec;
  const bool head = node && is_head((uint32_t)i, (int)me.z, s_parent[i], s_depth);
  float4 cell = make_float4(0.f, 0.f, 0.f, 0.f);
  if (CLOSED && head)
    cell = closed_cell(add4(hi, s_base4[me.y >> 8]), me.x ? add4(lo, s_base4[(me.x - 1) >> 8]) : lo, p0,
                       (int)me.z, ndim, a.sign, s_cube, a.fx_exp);
  sync();
  // ---- the heads' children counted, and their first slots
  const uint32_t cnt = head ? children_of((int)me.z, ndim, a.t.omask[i], me.y - me.x + 1) : 0u;
  if (node) a.t.count[i] = cnt;
  uint32_t x = cnt;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(FL_FULL, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  for (int w = 0; w < warp; ++w) x += s_warp[w];
  if (node) a.t.first[i] = x - cnt;
  if (tid == S - 1) a.vtmp[c] = x;  // the block's children
  sync();
  if (tid < (n + 255) / 256) {
    uint32_t b = 0;
    for (int q = 0; q < tid * 256 / S; ++q) b += a.vtmp[q];
    s_base[tid] = b;
    if (!CLOSED && c == 0) static_cast<uint32_t*>(a.t.scan_scratch)[tid] = b;
  }
  __syncthreads();
  // ---- the slots
  double* slot64 = a.slots64 ? a.t.slot64 : nullptr;
  if (i == 0) {  // the root's own slot
    if (CLOSED) a.t.child_data[0] = cell;
    a.t.child_meta[0] = make_uint2(first_slot(a.t.first, s_base, 0u, 1u), cnt | (me.z << 26));
  }
  if (node)
    write_slot<CLOSED>(false, i, nrec, n, ndim, 1u, a.t.omask, a.t.range, s_depth, a.t.count, a.t.first,
                       s_base, &cell, a.t.child_data, a.t.child_meta, slot64, a.err);
  if (ok) {
    write_slot<CLOSED>(true, i, prec, n, ndim, 1u, a.t.omask, a.t.range, s_depth, a.t.count, a.t.first,
                       s_base, &p, a.t.child_data, a.t.child_meta, slot64, a.err);
  }
}

constexpr int kWalkThreads = 128;
constexpr int kWalkWarps = kWalkThreads / 32;
constexpr int kStack = 96;  // entries per group in shared memory; deeper entries spill to global
// A group's stack never holds more than (levels + 1) * 32 entries: every round pushes at most 32
// entries (the cells its points open), and the entries on the stack form layers, one per round
// whose pushes are not yet consumed, holding cells of strictly increasing depth.
__host__ __device__ constexpr int kWalkStackLayers(int ndim) { return (ndim == 3 ? 21 : 24) + 1; }
constexpr int kWalkSpillPerWarp = 704;  // max over dims of 32 (levels + 1) - kStack
// Blocks per SM the walk's registers are held to: at 1M nodes 8 (64 registers) measured 740 us a
// launch, 9 (56) 746, 7 (72) 766.
constexpr int kWalkMinBlocks = 8;
constexpr int kWalkBlocksPerSm = 10;    // blocks of the persistent walk grid per SM
// the largest layout whose walk runs one point per warp by default (FL_TUNE_WALK_GROUP 0)
constexpr int kLaneWalkMaxNodes = 32768;

// Packed FP32 pairs (the f32x2 arithmetic of sm_100 and later): two children per instruction.
__device__ __forceinline__ uint64_t pk2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 up2(uint64_t x) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
  return r;
}
__device__ __forceinline__ uint64_t sub2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ float rcp_approx(float x) {  // the reciprocal __fdividef multiplies by
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

constexpr int kSeenWords = 64;  // a group's coordinate filter: 2,048 bits per axis
// A warp's walk state. The round's children are kept as pairs (2j, 2j + 1) in the packed layout
// that the f32x2 arithmetic reads.
struct WalkShared {
  uint4 stack[kStack];  // first child slot, count, top depth, the points that test the children
  float4 a[16];         // {x, x', y, y'}
  float4 b[16];         // {z, z', value, value'}: at the chain's top depth, times alpha
  float4 t[16];         // {theta threshold, ', uncommon cases' bound, '}
  uint32_t mask[32];    // the points that test each child
  uint32_t opens[32];   // the points that open each child
  uint32_t seen[3][kSeenWords];
  float4 lo, hi;        // the group's bounding box
};

// The less common cases of apply() (src/manyBody.js:73-115) for one child: a chain of cells
// whose widest cell is too close (the child is approximated at the first, widest, depth of the
// chain that passes the theta test), a zero component of the displacement (d3 replaces it with
// a jiggle) and distanceMin. `va` arrives as the value at the chain's top depth.
// The jiggle's ids of a pair are the graph's own, so that a layout draws the same jiggles alone
// or in any batch: a point's node index less its graph's first node (`first`), and for a cell
// the graph's node count `ng` plus the cell's first child slot counted from the graph's first
// (`cellbase`: the slot before it). Outside a batch: first 0, ng = n, cellbase 0.
template <int NDIM>
__device__ __forceinline__ void rare_case(uint32_t meta, uint32_t top, uint32_t idx, float T0,
                                          float dmin2, uint32_t myid, uint32_t first,
                                          uint32_t ng, uint32_t cellbase,
                                          const uint32_t* __restrict__ perm, int n, uint32_t step,
                                          uint32_t seed, float& va, float& dx, float& dy,
                                          float& dz, float& l) {
  if (meta != kLeafMark) {
    const uint32_t D = (meta >> 26) & 31u;
    if (top < D && T0 * pow4neg(top) >= l) {
      uint32_t k = top + 1;
      while (k < D && T0 * pow4neg(k) >= l) ++k;
      va *= damp(NDIM, (int)top - (int)k);  // value(k) = value(top) c^(top - k)
    }
  }
  if (dx == 0.f || (NDIM > 1 && dy == 0.f) || (NDIM > 2 && dz == 0.f)) {
    const uint32_t other =
        meta == kLeafMark
            ? perm[idx < (uint32_t)n ? idx : 0] - first
            : ng + (idx - cellbase);
    myid -= first;
    if (dx == 0.f) dx = fl::jiggle(myid, other, 0, step, seed), l += dx * dx;
    if (NDIM > 1 && dy == 0.f) dy = fl::jiggle(myid, other, 1, step, seed), l += dy * dy;
    if (NDIM > 2 && dz == 0.f) dz = fl::jiggle(myid, other, 2, step, seed), l += dz * dz;
  }
  if (l < dmin2) l = sqrtf(dmin2 * l);
}

__device__ __forceinline__ float below(float d2) {  // l < d2 <=> l <= below(d2), for l >= 0
  return d2 > 0.f ? __uint_as_float(__float_as_uint(d2) - 1u) : -1.f;
}
// 1 << i, 0 for i >= 32.
__device__ __forceinline__ uint32_t bit_at(uint32_t i) {
  uint32_t r;
  asm("shl.b32 %0, 1, %1;" : "=r"(r) : "r"(i));
  return r;
}
// The warp's inclusive prefix sum (shfl.up's predicate says whether the lane below exists).
__device__ __forceinline__ uint32_t inclusive_sum(uint32_t v) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .u32 t;\n\t"
        "shfl.sync.up.b32 t|p, %0, %1, 0, 0xffffffff;\n\t"
        "@p add.u32 %0, %0, t;\n\t}"
        : "+r"(v) : "r"(o));
  return v;
}
// A coordinate's bit of the filter (a multiplicative hash, 2^32 / golden ratio times 2): the sign
// is left out, so that 0 and -0 share a bit.
__device__ __forceinline__ uint32_t seen_bit(float x) {
  return (__float_as_uint(x) * 0x3c6ef362u) >> 21;
}
__device__ __forceinline__ bool maybe_seen(const uint32_t* seen, float x) {
  const uint32_t h = seen_bit(x);
  return seen[h >> 5] >> (h & 31u) & 1u;
}

// The walk of P consecutive sorted points by a warp: P = 32, a point per lane, or P = 16, two
// lanes per point that take every other pair of children (fewer points share, and pay for, one
// union of traversals).
//
// Per round the warp gathers 32 children, one per lane, and each lane decides from the group's
// bounding box what its child can need. The displacement, its square and their sum round
// monotonically, so the box's nearest squared distance bounds every point's own:
//   far    no point opens it and none takes an uncommon case: it is only applied
//   plain  some points may open it, but none takes an uncommon case
//   odd    distanceMin, a chain's widest cell or a coordinate that one of the points may share (a
//          zero component, which d3 jiggles) can occur
// A shared coordinate is looked for in a filter of the group's coordinates, 2,048 bits per axis,
// and only where the child lies within the box on that axis. Then every lane takes the children
// in order, two per step, with the tests that the pair's classes ask for: the same FP32 sums, in
// the same order, as testing every pair for everything.
//
// The pass is bound by instruction issue (79 % of the issue slots). At 1M nodes in 3D a group meets
// 687 children in 24.4 rounds, of which a point's own traversal needs 43 %; 61 % are far, 22 %
// plain. Measured with events, testing every pair for everything -> this: 791 -> 740 us a launch
// (1M nodes, 3D), 292 -> 259 (300k, distanceMax), 99 -> 92 (200k, 2D), 117 -> 113 (100k, 3D). Two
// far steps at once, not one (765 us) nor four (777). Applying the far children later, 32 at a
// time without tests, took 613 us, but adds each point's terms in another order.
//
// stats (STATS): [0] child tests (P per child), [1] tests a point's own traversal needed,
// [2] deepest stack, [3] points that opened a cell, [4] points that applied a cell or point,
// [5] pair steps that took the uncommon-case branch.
// BATCH: the points belong to a batch of graphs (segs): a group is up to 32 points of one graph,
// with its tree (root slot = its index), cube, theta, distances and alpha.
template <int NDIM, int P, bool STATS, bool DMAX, bool BATCH>
__global__ void __launch_bounds__(kWalkThreads, kWalkMinBlocks) k_walk(
    const float4* __restrict__ cdata, const uint2* __restrict__ cmeta,
    const float4* __restrict__ leaf, const uint32_t* __restrict__ perm,
    const float* __restrict__ cube, float4* __restrict__ vel, int n, float alpha,
    double theta2, float dmin2, float dmax2, uint32_t step, uint32_t seed, uint32_t* err,
    unsigned long long* stats, uint4* __restrict__ spill, int ngroups, uint32_t* work,
    FlSegs segs, const FlTick* __restrict__ tk) {
  if (tk) alpha = tk->alpha, step = tk->step, seed = tk->seed;
  constexpr int S = 32 / P;  // lanes per point
  constexpr uint32_t kPoints = P == 32 ? FL_FULL : (1u << (P & 31)) - 1u;
  // the stack: kStack entries in shared memory, the rest in this warp slot's region of the spill
  // buffer (at most 32 pushes a round, layers of strictly increasing depth)
  constexpr int kAll = kWalkStackLayers(NDIM) * 32;
  static_assert(kAll - kStack <= kWalkSpillPerWarp, "spill region too small");
  __shared__ WalkShared shw[kWalkWarps];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  WalkShared& sh = shw[warp];
  const int sub = lane / P;
  const uint32_t lanebit = 1u << (lane % P), below_me = (1u << lane) - 1u;
  // (size / 2^k)^2 / theta^2 = T0 * 4^-k, exactly (a power-of-two scaling); the FP64 division
  // once per block
  __shared__ float s_T0;
  if (!BATCH && threadIdx.x == 0) s_T0 = (float)((double)cube[3] * (double)cube[3] / theta2);
  __syncthreads();
  float T0 = BATCH ? 0.f : s_T0;
  uint32_t gfirst = 0, gstep = step, gcount = (uint32_t)n, gcells = 0;
  const uint32_t slot_cap = 2u * (uint32_t)n + 1u;
  unsigned long long st_tests = 0, st_useful = 0, st_open = 0, st_apply = 0, st_rare = 0;
  int maxsp = 0;
  uint4* spl = spill + (size_t)(blockIdx.x * kWalkWarps + warp) * kWalkSpillPerWarp;
  auto sget = [&](int i) { return i < kStack ? sh.stack[i] : spl[i - kStack]; };
  auto sset = [&](int i, uint4 v) {
    if (i < kStack) sh.stack[i] = v;
    else spl[i - kStack] = v;
  };
  // groups are handed out one at a time (the walk's cost varies a lot between groups, so a fixed
  // share per warp would leave some warps working long after the rest)
  int wi = lane == 0 ? (int)atomicAdd(work, 1u) : 0;
  wi = __shfl_sync(FL_FULL, wi, 0);
  while (wi < ngroups) {
    const uint2 range = BATCH ? segs.groups[wi]
                              : make_uint2((uint32_t)wi * P, min((uint32_t)wi * P + P, (uint32_t)n));
    const int base = (int)range.x;
    const int t = base + lane % P;
    const bool live = t < (int)range.y;
    const uint32_t act = __ballot_sync(FL_FULL, live) & kPoints;
    const float4 me = live ? leaf[t] : make_float4(0, 0, 0, 0);
    const uint32_t myid = live ? perm[t] : 0;
    uint4 root = make_uint4(0u, 1u, 0u, act);  // slot 0, one child, top depth 0
    int sp = 1;
    if (BATCH) {
      const uint32_t g = segs.gid_pos[base];
      const FlGraph& gr = segs.g[g];
      T0 = gr.T0, dmin2 = gr.dmin2, dmax2 = gr.dmax2, alpha = gr.alpha;
      gfirst = (uint32_t)gr.first, gstep = step + gr.tick0, gcount = (uint32_t)gr.count;
      root.x = g;
      // the graph's root sits in slot g; its first child slot less one is where the graph's
      // slots are counted from (a lone simulation's root has its children from slot 1)
      if (gr.count > 1) gcells = __ldg(&cmeta[g].x) - 1u;
      if (gr.count < 2 || gr.frozen) sp = 0;  // no tree, or sitting the tick out
    }
    const float dmin_le = below(dmin2);
    // the group's box and coordinate filter
    for (int i = lane; i < 3 * kSeenWords; i += 32) (&sh.seen[0][0])[i] = 0u;
    {
      const float c[3] = {me.x, me.y, me.z};
      float blo[3] = {0.f, 0.f, 0.f}, bhi[3] = {0.f, 0.f, 0.f};
#pragma unroll
      for (int k = 0; k < NDIM; ++k) {
        // a NaN coordinate bounds nothing: its tests all fail, whatever the child's class
        const bool in = live && c[k] == c[k];
        blo[k] = fl::unordered(__reduce_min_sync(FL_FULL, in ? fl::ordered(c[k]) : 0xffffffffu));
        bhi[k] = fl::unordered(__reduce_max_sync(FL_FULL, in ? fl::ordered(c[k]) : 0u));
      }
      if (lane == 0) {
        sh.lo = make_float4(blo[0], blo[1], blo[2], 0.f);
        sh.hi = make_float4(bhi[0], bhi[1], bhi[2], 0.f);
        sset(0, root);
      }
      __syncwarp();
      if (live && sub == 0) {
#pragma unroll
        for (int k = 0; k < NDIM; ++k) {
          const uint32_t h = seen_bit(c[k]);
          atomicOr(&sh.seen[k][h >> 5], 1u << (h & 31u));
        }
      }
    }
    uint64_t AX = 0, AY = 0, AZ = 0;  // force sums, one per child of a pair
    const uint64_t MX = pk2(me.x, me.x), MY = pk2(me.y, me.y), MZ = pk2(me.z, me.z);
    __syncwarp();
    uint32_t guard = 0;
    const uint32_t guard_max = 4u * (uint32_t)n + 64u;
    while (sp > 0) {
      // gather the first 32 children from the top of the stack, in parallel: lane i reads the i-th
      // entry from the top, a prefix sum of the entries' child counts places each entry's
      // children, and a lane's child belongs to the last entry that starts at or before it
      const bool has = lane < sp;
      uint4 e = has ? sget(sp - 1 - lane) : make_uint4(0u, 0u, 0u, 0u);
      if (has && (e.x >= slot_cap || e.y - 1u >= slot_cap - e.x)) {  // a malformed tree: never read past it
        atomicOr(err, FL_ERR_TREE);
        e.x = 0u, e.y = 1u, e.w = 0u;  // a child that no point tests
      }
      const uint32_t inc = inclusive_sum(e.y), exc = inc - e.y;
      const uint32_t avail = __shfl_sync(FL_FULL, inc, 31), total = min(avail, 32u);
      // entries taken whole leave the stack; one taken in part keeps the rest (the new top)
      const uint32_t taken = __ballot_sync(FL_FULL, has && inc <= total);
      if (avail > 32u && has && exc < 32u && inc > 32u)
        sset(sp - 1 - lane, make_uint4(e.x + (32u - exc), inc - 32u, e.z, e.w));
      sp -= __popc(taken);
      const uint32_t starts = __reduce_or_sync(FL_FULL, has && exc < total ? 1u << exc : 0u);
      const int own = __popc(starts & (below_me | (1u << lane))) - 1;
      const uint32_t slot = __shfl_sync(FL_FULL, e.x - exc, own) + (uint32_t)lane;
      const uint32_t my_mask = __shfl_sync(FL_FULL, e.w, own);
      const uint32_t top = __shfl_sync(FL_FULL, e.z, own);
      // the lane's child: what it can need of the points
      const bool ok = (uint32_t)lane < total;
      float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
      uint2 m = make_uint2(0u, kLeafMark);
      if (ok) q = __ldg(cdata + slot), m = __ldg(cmeta + slot);
      const bool lf = m.y == kLeafMark;
      uint32_t mask = ok && q.w != 0.f ? my_mask : 0u;  // d3 skips a zero value and all it holds
      if (lf) mask &= ~bit_at(m.x - (uint32_t)base);    // itself
      // a point is never approximated (its sum is the same either way); a cell is opened when
      // even its deepest depth fails the theta test
      const uint32_t D = (m.y >> 26) & 31u;
      const bool chain = !lf && top < D;
      const float topen = lf ? -INFINITY : T0 * pow4neg(D);
      const float bound = fmaxf(chain ? T0 * pow4neg(top) : topen, dmin_le);
      float va = q.w * alpha;
      if (chain) va *= damp(NDIM, (int)(D - top));
      const float4 blo = sh.lo, bhi = sh.hi;
      const float nx = fmaxf(fmaxf(blo.x - q.x, q.x - bhi.x), 0.f);
      const float ny = NDIM > 1 ? fmaxf(fmaxf(blo.y - q.y, q.y - bhi.y), 0.f) : 0.f;
      const float nz = NDIM > 2 ? fmaxf(fmaxf(blo.z - q.z, q.z - bhi.z), 0.f) : 0.f;
      float near2 = nx * nx;
      if (NDIM > 1) near2 = fmaf(ny, ny, near2);
      if (NDIM > 2) near2 = fmaf(nz, nz, near2);
      bool zero = (nx == 0.f) & maybe_seen(sh.seen[0], q.x);
      if (NDIM > 1) zero |= (ny == 0.f) & maybe_seen(sh.seen[1], q.y);
      if (NDIM > 2) zero |= (nz == 0.f) & maybe_seen(sh.seen[2], q.z);
      const bool far = mask == 0u || (!zero && near2 > bound);
      const bool plain = far || (!zero && near2 > dmin_le && !chain);
      const uint32_t bfar = __ballot_sync(FL_FULL, far), bplain = __ballot_sync(FL_FULL, plain);
      {
        float* pa = reinterpret_cast<float*>(&sh.a[lane >> 1]) + (lane & 1);
        float* pb = reinterpret_cast<float*>(&sh.b[lane >> 1]) + (lane & 1);
        float* pt = reinterpret_cast<float*>(&sh.t[lane >> 1]) + (lane & 1);
        pa[0] = q.x, pa[2] = q.y, pb[0] = q.z, pb[2] = va, pt[0] = topen, pt[2] = bound;
        sh.mask[lane] = mask;
        sh.opens[lane] = 0u;
      }
      __syncwarp();
      // two children per step and lane (per point: S pairs): independent work to overlap. Two steps
      // of far children are taken at once
#define FL_WALK_PAIR(jj)                                             \
  const float4 pa = sh.a[jj], pb = sh.b[jj];                         \
  const uint2 pm = reinterpret_cast<const uint2*>(sh.mask)[jj];      \
  uint64_t DX = sub2(pk2(pa.x, pa.y), MX);                           \
  uint64_t DY = NDIM > 1 ? sub2(pk2(pa.z, pa.w), MY) : 0ull;         \
  uint64_t DZ = NDIM > 2 ? sub2(pk2(pb.x, pb.y), MZ) : 0ull;         \
  uint64_t L = mul2(DX, DX);                                         \
  if (NDIM > 1) L = fma2(DY, DY, L);                                 \
  if (NDIM > 2) L = fma2(DZ, DZ, L);                                 \
  float2 l = up2(L);                                                 \
  const bool m0 = pm.x & lanebit, m1 = pm.y & lanebit;               \
  bool a0 = m0 && (!DMAX || l.x < dmax2), a1 = m1 && (!DMAX || l.y < dmax2)
#define FL_WALK_APPLY(v0, v1)                                                                    \
  do {                                                                                           \
    const float2 w = up2(mul2(pk2(v0, v1), pk2(rcp_approx(l.x), rcp_approx(l.y))));              \
    const uint64_t W = pk2(a0 ? w.x : 0.f, a1 ? w.y : 0.f);                                      \
    AX = fma2(DX, W, AX);                                                                        \
    if (NDIM > 1) AY = fma2(DY, W, AY);                                                          \
    if (NDIM > 2) AZ = fma2(DZ, W, AZ);                                                          \
    if (STATS) st_apply += a0 + a1;                                                              \
  } while (0)
      constexpr uint32_t kStep = S == 1 ? 3u : 15u, kTwo = S == 1 ? 15u : 255u;
      int j = 0;
      while (j < (int)total) {
        const int jj = (j >> 1) + sub;
        if (((bfar >> j) & kTwo) == kTwo) {
          { FL_WALK_PAIR(jj); FL_WALK_APPLY(pb.z, pb.w); }
          { FL_WALK_PAIR(jj + S); FL_WALK_APPLY(pb.z, pb.w); }
          j += 4 * S;
          continue;
        }
        if (((bplain >> j) & kStep) == kStep) {
          FL_WALK_PAIR(jj);
          const float4 pt = sh.t[jj];
          const bool o0 = m0 && pt.x >= l.x, o1 = m1 && pt.y >= l.y;
          a0 = a0 && !o0, a1 = a1 && !o1;
          const uint32_t b0 = __ballot_sync(FL_FULL, o0), b1 = __ballot_sync(FL_FULL, o1);
          reinterpret_cast<uint2*>(sh.opens)[jj] =
              make_uint2(b0 >> (sub * P & 31) & kPoints, b1 >> (sub * P & 31) & kPoints);
          FL_WALK_APPLY(pb.z, pb.w);
          j += 2 * S;
          continue;
        }
        FL_WALK_PAIR(jj);
        const float4 pt = sh.t[jj];
        float v0 = pb.z, v1 = pb.w;
        // the bound covers the theta test too: it is no less than the threshold
        const float2 zp = up2(NDIM == 3 ? mul2(mul2(DX, DY), DZ) : NDIM == 2 ? mul2(DX, DY) : DX);
        const bool c0 = l.x <= pt.z || zp.x == 0.f, c1 = l.y <= pt.w || zp.y == 0.f;
        if (__any_sync(FL_FULL, (m0 && c0) || (m1 && c1))) {
          const bool o0 = m0 && pt.x >= l.x, o1 = m1 && pt.y >= l.y;
          a0 = a0 && !o0, a1 = a1 && !o1;
          const uint32_t b0 = __ballot_sync(FL_FULL, o0), b1 = __ballot_sync(FL_FULL, o1);
          reinterpret_cast<uint2*>(sh.opens)[jj] =
              make_uint2(b0 >> (sub * P & 31) & kPoints, b1 >> (sub * P & 31) & kPoints);
          if (__any_sync(FL_FULL, (a0 && c0) || (a1 && c1))) {
            if (STATS && lane == 0) ++st_rare;
            const uint32_t y0 = __shfl_sync(FL_FULL, m.y, 2 * jj), y1 = __shfl_sync(FL_FULL, m.y, 2 * jj + 1);
            const uint32_t x0 = __shfl_sync(FL_FULL, m.x, 2 * jj), x1 = __shfl_sync(FL_FULL, m.x, 2 * jj + 1);
            const uint32_t p0 = __shfl_sync(FL_FULL, top, 2 * jj), p1 = __shfl_sync(FL_FULL, top, 2 * jj + 1);
            float2 dx = up2(DX), dy = up2(DY), dz = up2(DZ);
            if (a0 && c0)
              rare_case<NDIM>(y0, p0, x0, T0, dmin2, myid, gfirst, gcount, gcells, perm, n, gstep,
                              seed, v0, dx.x, dy.x, dz.x, l.x);
            if (a1 && c1)
              rare_case<NDIM>(y1, p1, x1, T0, dmin2, myid, gfirst, gcount, gcells, perm, n, gstep,
                              seed, v1, dx.y, dy.y, dz.y, l.y);
            DX = pk2(dx.x, dx.y), DY = pk2(dy.x, dy.y), DZ = pk2(dz.x, dz.y);
          }
        }
        FL_WALK_APPLY(v0, v1);
        j += 2 * S;
      }
#undef FL_WALK_PAIR
#undef FL_WALK_APPLY
      __syncwarp();
      // the children some points must open go on the stack, in child order
      const uint32_t opens = sh.opens[lane];
      const uint32_t pushes = __ballot_sync(FL_FULL, opens != 0u);
      if (opens) {
        const int to = sp + __popc(pushes & below_me);
        if (to < kAll) sset(to, make_uint4(m.x, m.y & kCountMask, D + 1u, opens));
      }
      sp += __popc(pushes);
      if (sp > kAll) {  // beyond the bound on the stack's depth: a malformed tree
        if (lane == 0) atomicOr(err, FL_ERR_STACK);
        sp = kAll;
      }
      if (STATS) {
        if (ok) st_tests += P, st_useful += __popc(mask), st_open += __popc(opens);
        if (sp > maxsp) maxsp = sp;
      }
      __syncwarp();
      if (++guard > guard_max) {
        if (lane == 0) atomicOr(err, FL_ERR_STACK);
        break;
      }
    }
    const float2 ax2 = up2(AX), ay2 = up2(AY), az2 = up2(AZ);
    float ax = ax2.x + ax2.y, ay = ay2.x + ay2.y, az = az2.x + az2.y;
#pragma unroll
    for (int o = P; o < 32; o <<= 1) {  // a point's lanes
      ax += __shfl_xor_sync(FL_FULL, ax, o);
      if (NDIM > 1) ay += __shfl_xor_sync(FL_FULL, ay, o);
      if (NDIM > 2) az += __shfl_xor_sync(FL_FULL, az, o);
    }
    if (live && sub == 0) {
      float4 v = vel[myid];
      v.x += ax;
      if (NDIM > 1) v.y += ay;
      if (NDIM > 2) v.z += az;
      vel[myid] = v;
    }
    __syncwarp();
    wi = lane == 0 ? (int)atomicAdd(work, 1u) : 0;
    wi = __shfl_sync(FL_FULL, wi, 0);
  }
  // every warp ends on one claim past the last group; the last of those claims puts the counter
  // back to 0 for the next launch (no other warp touches it after its own last claim)
  if (lane == 0 && wi == ngroups + (int)(gridDim.x * kWalkWarps) - 1) *work = 0u;
  if (STATS) {
    atomicAdd(stats, st_tests);
    atomicAdd(stats + 1, st_useful);
    atomicMax(stats + 2, (unsigned long long)maxsp);
    atomicAdd(stats + 3, st_open);
    atomicAdd(stats + 4, st_apply);
    if (lane == 0) atomicAdd(stats + 5, st_rare);
  }
}

// The walk of one point per warp, for small layouts: where the union walk above has too few
// groups of 32 points to fill the device (a 1,000-node layout is 32 warps, each a long serial
// chain of rounds), each warp walks one point's own d3 traversal and its lanes test up to 32
// children of it at once. The children are gathered from the top of the point's stack as in the
// union walk; a lane tests its child against the point, applies it, takes the uncommon case or
// pushes the child's children. Each lane sums what it applied, and the warp adds the lanes'
// sums in a fixed shuffle tree, so a layout is the same run after run. The stack holds the
// bound on its depth in shared memory, 8 bytes an entry (first child slot; count | top depth
// << 26), so nothing spills and the grid is not limited by spill regions. Bound by instruction issue
// (68 % of the slots): 20,000 points take some 9 rounds of 165 instructions each, 44 us; finding each
// child's entry by marks in shared memory and a running maximum in place of one ballot took 47.
// stats (STATS): [0] children tested, [1] of those, the ones the point's d3 traversal needs
// (not a zero value, not the point itself; the union walk's [1], [3] and [4] count the same
// (point, child) pairs), [2] deepest stack, [3] cells opened, [4] cells or points applied,
// [5] rounds in which a lane took the uncommon case.
template <int NDIM, bool STATS, bool DMAX>
__global__ void __launch_bounds__(kWalkThreads) k_walk_lanes(
    const float4* __restrict__ cdata, const uint2* __restrict__ cmeta,
    const float4* __restrict__ leaf, const uint32_t* __restrict__ perm,
    const float* __restrict__ cube, float4* __restrict__ vel, int n, float alpha,
    double theta2, float dmin2, float dmax2, uint32_t step, uint32_t seed, uint32_t* err,
    unsigned long long* stats, uint32_t* work, const FlTick* __restrict__ tk) {
  if (tk) alpha = tk->alpha, step = tk->step, seed = tk->seed;
  // at most 32 children per round and one push per child: the union walk's bound with G = 32
  constexpr int kAll = kWalkStackLayers(NDIM) * 32;
  __shared__ uint2 s_stack[kWalkWarps][kAll];
  __shared__ float s_T0;
  if (threadIdx.x == 0) s_T0 = (float)((double)cube[3] * (double)cube[3] / theta2);
  __syncthreads();
  const float T0 = s_T0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t below_me = (1u << lane) - 1u;
  const float dmin_le = below(dmin2);
  const uint32_t slot_cap = 2u * (uint32_t)n + 1u;
  unsigned long long st_tests = 0, st_useful = 0, st_open = 0, st_apply = 0, st_rare = 0;
  int maxsp = 0;
  uint2* stk = s_stack[warp];
  int t = lane == 0 ? (int)atomicAdd(work, 1u) : 0;
  t = __shfl_sync(FL_FULL, t, 0);
  while (t < n) {
    const float4 me = leaf[t];  // the same address in every lane: one load
    const uint32_t myid = perm[t];
    float ax = 0.f, ay = 0.f, az = 0.f;
    if (lane == 0) stk[0] = make_uint2(0u, 1u);  // the root: slot 0, one child, top depth 0
    int sp = 1;
    uint32_t guard = 0;
    const uint32_t guard_max = 4u * (uint32_t)n + 64u;
    __syncwarp();
    while (sp > 0) {
      // the gather of the union walk: lane i reads the i-th entry from the top, a prefix sum of the
      // entries' child counts places their children, lane j takes child j of the round
      const bool has = lane < sp;
      const uint2 se = has ? stk[sp - 1 - lane] : make_uint2(0u, 0u);
      uint32_t ex = se.x, ey = se.y & kCountMask;
      if (has && (ex >= slot_cap || ey - 1u >= slot_cap - ex)) {  // a malformed tree: never read past it
        atomicOr(err, FL_ERR_TREE);
        ex = slot_cap - 1u, ey = 1u;  // the last slot: no tree fills it, and its value is 0
      }
      const uint32_t inc = inclusive_sum(ey), exc = inc - ey;
      const uint32_t avail = __shfl_sync(FL_FULL, inc, 31), total = min(avail, 32u);
      // entries taken whole leave the stack; one taken in part keeps the rest (the new top)
      const uint32_t taken = __ballot_sync(FL_FULL, has && inc <= total);
      if (avail > 32u && has && exc < 32u && inc > 32u)
        stk[sp - 1 - lane] = make_uint2(ex + (32u - exc), (inc - 32u) | (se.y & ~kCountMask));
      sp -= __popc(taken);
      const uint32_t starts = __reduce_or_sync(FL_FULL, has && exc < total ? 1u << exc : 0u);
      const int own = __popc(starts & (below_me | (1u << lane))) - 1;
      const uint32_t slot = __shfl_sync(FL_FULL, ex - exc, own) + (uint32_t)lane;
      const uint32_t my_top = __shfl_sync(FL_FULL, se.y >> 26, own);
      bool o = false, a = false, rare = false, need = false;
      uint2 m = make_uint2(0u, 0u);
      uint32_t D = 0;
      if ((uint32_t)lane < total) {
        const float4 q = __ldg(cdata + slot);
        m = __ldg(cmeta + slot);
        const bool lf = m.y == kLeafMark;
        D = (m.y >> 26) & 31u;
        // d3 skips a zero value and all it holds, and the point itself
        const bool mask = q.w != 0.f && !(lf && m.x == (uint32_t)t);
        need = mask;
        const bool chain = !lf && my_top < D;
        const float topen = lf ? -INFINITY : T0 * pow4neg(D);
        const float ttop = chain ? T0 * pow4neg(my_top) : topen;
        float va = chain ? q.w * alpha * damp(NDIM, (int)(D - my_top)) : q.w * alpha;
        float dx = q.x - me.x;
        float dy = NDIM > 1 ? q.y - me.y : 0.f;
        float dz = NDIM > 2 ? q.z - me.z : 0.f;
        float l = dx * dx;
        if (NDIM > 1) l = fmaf(dy, dy, l);
        if (NDIM > 2) l = fmaf(dz, dz, l);
        const float zp = NDIM == 3 ? (dx * dy) * dz : NDIM == 2 ? dx * dy : dx;
        o = mask && topen >= l;
        a = mask && !o && (!DMAX || l < dmax2);
        rare = a && (l <= fmaxf(ttop, dmin_le) || zp == 0.f);
        if (rare)
          rare_case<NDIM>(m.y, my_top, m.x, T0, dmin2, myid, 0u, (uint32_t)n, 0u, perm, n, step,
                          seed, va, dx, dy, dz, l);
        if (a) {
          const float w = va * rcp_approx(l);
          ax = fmaf(dx, w, ax);
          if (NDIM > 1) ay = fmaf(dy, w, ay);
          if (NDIM > 2) az = fmaf(dz, w, az);
        }
      }
      // the children to open go on the stack in child order, the last on top
      const uint32_t opened = __ballot_sync(FL_FULL, o);
      if (o) {
        const int at = sp + __popc(opened & below_me);
        if (at < kAll) stk[at] = make_uint2(m.x, (m.y & kCountMask) | (D + 1u) << 26);
      }
      sp += __popc(opened);
      if (sp > kAll) {  // beyond the bound on the stack's depth: a malformed tree
        if (lane == 0) atomicOr(err, FL_ERR_STACK);
        sp = kAll;
      }
      if (STATS) {
        const uint32_t ap = __ballot_sync(FL_FULL, a), nd = __ballot_sync(FL_FULL, need);
        const bool rr = __any_sync(FL_FULL, rare);
        if (lane == 0) {
          st_tests += total, st_useful += __popc(nd), st_open += __popc(opened);
          st_apply += __popc(ap), st_rare += rr;
          if (sp > maxsp) maxsp = sp;
        }
      }
      __syncwarp();
      if (++guard > guard_max) {
        if (lane == 0) atomicOr(err, FL_ERR_STACK);
        break;
      }
    }
#pragma unroll
    for (int k = 16; k > 0; k >>= 1) {
      ax += __shfl_xor_sync(FL_FULL, ax, k);
      if (NDIM > 1) ay += __shfl_xor_sync(FL_FULL, ay, k);
      if (NDIM > 2) az += __shfl_xor_sync(FL_FULL, az, k);
    }
    if (lane == 0) {
      float4 v = vel[myid];
      v.x += ax;
      if (NDIM > 1) v.y += ay;
      if (NDIM > 2) v.z += az;
      vel[myid] = v;
    }
    __syncwarp();
    t = lane == 0 ? (int)atomicAdd(work, 1u) : 0;
    t = __shfl_sync(FL_FULL, t, 0);
  }
  // as in k_walk: the last claim past the end puts the counter back to 0
  if (lane == 0 && t == n + (int)(gridDim.x * kWalkWarps) - 1) *work = 0u;
  if (STATS && lane == 0) {
    atomicAdd(stats, st_tests);
    atomicAdd(stats + 1, st_useful);
    atomicMax(stats + 2, (unsigned long long)maxsp);
    atomicAdd(stats + 3, st_open);
    atomicAdd(stats + 4, st_apply);
    atomicAdd(stats + 5, st_rare);
  }
}

// Exact all-pairs sum (theta ~ 0; src/gpu/passes/manyBody.js:5-16 semantics). A cluster of up to 8
// blocks sums the forces on 32 Q points: every warp holds the same points, Q per lane, and takes
// every (warps of the cluster)-th tile of 32 sources, which its lanes load and lay out in shared
// memory as pairs for the f32x2 arithmetic. Four sources at a time, for every point of the lane,
// are tested for what is not the common case (the point itself, distanceMin, a zero component)
// by the least of their squared distances and components, with one vote; such a four is summed
// source by source. The common path weighs a source that does not count with 0, so its displacement
// has to be finite: a source without strength is laid out at a place that no point meets, and a tile
// with a source beyond kPairFar (infinite or NaN too), or for a point beyond it, is summed source by
// source. The warps' sums are added in a fixed order, in shared memory and then
// over the cluster's.
//
// Bound by the FP32 pipe and instruction issue (57 % of the slots): a pair of sources and a point take
// 10 packed instructions of 2 cycles each, 22 instructions in all. 20,000 points in 3D: 212 us alone
// (110 is the packed instructions), where one thread per point and sixteenth of the sources, each source
// tested in scalars, took 757; 4,000 points 64 -> 18, 1,000 points 21 -> 9. Blocks of 128 threads: 256 wait longer
// for their slowest warp (249 us).
constexpr int kPairThreads = 128;
constexpr int kPairWarps = kPairThreads / 32;
constexpr int kPairClusterMax = 8;
// More points than this: two per lane. Ticks in 3D with one and with two: 9,000 points 62 and 65 us, 10,000
// 73 and 72, 12,000 98 and 93 (in 2D 8,000 already take 44 and 42).
constexpr int kPairTwoPoints = 10000;
constexpr float kPairFar = 8.5070592e37f;  // 2^126: no difference of coordinates below it overflows
constexpr float kPairNowhere = 1.1529215e18f;  // 2^60: finite squares, and no subnormal distance nearby
// whether a coordinate of p is kPairFar or more, infinite or NaN
template <int NDIM>
__device__ __forceinline__ bool pair_far(float4 p) {
  return !(fabsf(p.x) < kPairFar) || (NDIM > 1 && !(fabsf(p.y) < kPairFar)) || (NDIM > 2 && !(fabsf(p.z) < kPairFar));
}

// One source's force on a point, every case but, without DMAX, that of an infinite distance between
// infinite coordinates, which is left out too (an infinite l of finite ones adds 0).
template <int NDIM, bool DMAX>
__device__ __forceinline__ void pair_term(float4 me, uint32_t i, float4 o, uint32_t other,
                                          float dmin2, float dmax2, uint32_t step, uint32_t seed,
                                          float& ax, float& ay, float& az) {
  if (other == i || o.w == 0.f) return;
  float dx = o.x - me.x, dy = NDIM > 1 ? o.y - me.y : 0.f, dz = NDIM > 2 ? o.z - me.z : 0.f;
  float l = dx * dx;
  if (NDIM > 1) l = fmaf(dy, dy, l);
  if (NDIM > 2) l = fmaf(dz, dz, l);
  if (DMAX && l >= dmax2) return;
  if (dx == 0.f) dx = fl::jiggle(i, other, 0, step, seed), l += dx * dx;
  if (NDIM > 1 && dy == 0.f) dy = fl::jiggle(i, other, 1, step, seed), l += dy * dy;
  if (NDIM > 2 && dz == 0.f) dz = fl::jiggle(i, other, 2, step, seed), l += dz * dz;
  if (l < dmin2) l = sqrtf(dmin2 * l);
  const float w = o.w * rcp_approx(l);
  ax = fmaf(dx, w, ax), ay = fmaf(dy, w, ay), az = fmaf(dz, w, az);
}

template <int NDIM, int Q, bool DMAX>
__global__ void __launch_bounds__(kPairThreads) k_allpairs(
    const float4* __restrict__ pos, const float* __restrict__ strength, float4* __restrict__ vel,
    int n, float alpha, float dmin2, float dmax2, uint32_t step, uint32_t seed,
    const FlTick* __restrict__ tk) {
  if (tk) alpha = tk->alpha, step = tk->step, seed = tk->seed;
  __shared__ float4 s_a[kPairWarps][16], s_b[kPairWarps][16];  // {x, x', y, y'}, {z, z', s, s'}
  __shared__ float s_part[kPairWarps][3][32 * Q];
  __shared__ float s_sum[3][32 * Q];
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int rank = (int)cluster.block_rank(), blocks = (int)cluster.num_blocks();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int first = (int)(blockIdx.x / blocks) * 32 * Q;
  bool far_point = false;
  float4 me[Q];
  uint64_t MX[Q], MY[Q], MZ[Q], AX[Q], AY[Q], AZ[Q];
#pragma unroll
  for (int p = 0; p < Q; ++p) {
    const int i = first + 32 * p + lane;
    me[p] = i < n ? pos[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    MX[p] = pk2(me[p].x, me[p].x), MY[p] = pk2(me[p].y, me[p].y), MZ[p] = pk2(me[p].z, me[p].z);
    AX[p] = AY[p] = AZ[p] = 0;
    far_point |= pair_far<NDIM>(me[p]);
  }
  far_point = __any_sync(FL_FULL, far_point);
  constexpr int K = 2;  // pairs of sources at a time
  const float close = fmaxf(below(dmin2), 0.f);  // l <= close: distanceMin, or no distance at all
  float4* sa = s_a[warp];
  float4* sb = s_b[warp];
  for (int base = 32 * (rank * kPairWarps + warp); base < n; base += 32 * kPairWarps * blocks) {
    const int j = base + lane;
    float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
    if (j < n) o = pos[j], o.w = strength[j];
    if (o.w == 0.f) o.x = o.y = o.z = kPairNowhere;
    o.w *= alpha;
    const bool apart = far_point || __any_sync(FL_FULL, pair_far<NDIM>(o));
    __syncwarp();
    {
      float* pa = reinterpret_cast<float*>(&sa[lane >> 1]) + (lane & 1);
      float* pb = reinterpret_cast<float*>(&sb[lane >> 1]) + (lane & 1);
      pa[0] = o.x, pa[2] = o.y, pb[0] = o.z, pb[2] = o.w;
    }
    __syncwarp();
    // pair k of the tile, source by source
    auto one_by_one = [&](int k, auto dmax) {
      const float4 u = sa[k], v = sb[k];
      const uint32_t at = (uint32_t)(base + 2 * k);
#pragma unroll
      for (int p = 0; p < Q; ++p) {
        float2 ax = up2(AX[p]), ay = up2(AY[p]), az = up2(AZ[p]);
        const uint32_t i = (uint32_t)(first + 32 * p + lane);
        pair_term<NDIM, decltype(dmax)::value>(me[p], i, make_float4(u.x, u.z, v.x, v.z), at, dmin2, dmax2, step, seed, ax.x, ay.x, az.x);
        pair_term<NDIM, decltype(dmax)::value>(me[p], i, make_float4(u.y, u.w, v.y, v.w), at + 1, dmin2, dmax2, step, seed, ax.y, ay.y, az.y);
        AX[p] = pk2(ax.x, ax.y), AY[p] = pk2(ay.x, ay.y), AZ[p] = pk2(az.x, az.y);
      }
    };
    if (apart) {
#pragma unroll 1
      for (int k = 0; k < 16; ++k) one_by_one(k, std::true_type());
      continue;
    }
#pragma unroll 1
    for (int k = 0; k < 16; k += K) {
      float4 a[K], b[K];
      uint64_t DX[Q][K], DY[Q][K], DZ[Q][K];
      float2 l[Q][K];
      float lmin = INFINITY, cmin = INFINITY;
#pragma unroll
      for (int c = 0; c < K; ++c) a[c] = sa[k + c], b[c] = sb[k + c];
#pragma unroll
      for (int p = 0; p < Q; ++p)
#pragma unroll
        for (int c = 0; c < K; ++c) {
          DX[p][c] = sub2(pk2(a[c].x, a[c].y), MX[p]);
          DY[p][c] = NDIM > 1 ? sub2(pk2(a[c].z, a[c].w), MY[p]) : 0ull;
          DZ[p][c] = NDIM > 2 ? sub2(pk2(b[c].x, b[c].y), MZ[p]) : 0ull;
          uint64_t L = mul2(DX[p][c], DX[p][c]);
          if (NDIM > 1) L = fma2(DY[p][c], DY[p][c], L);
          if (NDIM > 2) L = fma2(DZ[p][c], DZ[p][c], L);
          l[p][c] = up2(L);
          const float2 dx = up2(DX[p][c]), dy = up2(DY[p][c]), dz = up2(DZ[p][c]);
          lmin = fminf(fminf(lmin, l[p][c].x), l[p][c].y);
          cmin = fminf(fminf(cmin, fabsf(dx.x)), fabsf(dx.y));
          if (NDIM > 1) cmin = fminf(fminf(cmin, fabsf(dy.x)), fabsf(dy.y));
          if (NDIM > 2) cmin = fminf(fminf(cmin, fabsf(dz.x)), fabsf(dz.y));
        }
      bool odd = lmin <= close || cmin == 0.f;
      // in a small layout mostly the point itself: then as if infinitely far (in a large one it is
      // met too seldom for what the test costs in registers)
      if (Q == 1 && __any_sync(FL_FULL, odd)) {
        odd = false;
#pragma unroll
        for (int c = 0; c < K; ++c) {
          const int self = first + lane - (base + 2 * (k + c));
          const float2 dx = up2(DX[0][c]), dy = up2(DY[0][c]), dz = up2(DZ[0][c]);
          if (self == 0) l[0][c].x = INFINITY;
          else odd |= l[0][c].x <= close || dx.x == 0.f || (NDIM > 1 && dy.x == 0.f) || (NDIM > 2 && dz.x == 0.f);
          if (self == 1) l[0][c].y = INFINITY;
          else odd |= l[0][c].y <= close || dx.y == 0.f || (NDIM > 1 && dy.y == 0.f) || (NDIM > 2 && dz.y == 0.f);
        }
      }
      if (__any_sync(FL_FULL, odd)) {
#pragma unroll 1
        for (int c = 0; c < K; ++c) one_by_one(k + c, std::bool_constant<DMAX>());
        continue;
      }
#pragma unroll
      for (int p = 0; p < Q; ++p)
#pragma unroll
        for (int c = 0; c < K; ++c) {
          uint64_t W = mul2(pk2(b[c].z, b[c].w), pk2(rcp_approx(l[p][c].x), rcp_approx(l[p][c].y)));
          if (DMAX) {
            const float2 w = up2(W);
            W = pk2(l[p][c].x < dmax2 ? w.x : 0.f, l[p][c].y < dmax2 ? w.y : 0.f);
          }
          AX[p] = fma2(DX[p][c], W, AX[p]);
          if (NDIM > 1) AY[p] = fma2(DY[p][c], W, AY[p]);
          if (NDIM > 2) AZ[p] = fma2(DZ[p][c], W, AZ[p]);
        }
    }
  }
#pragma unroll
  for (int p = 0; p < Q; ++p) {
    const float2 ax = up2(AX[p]), ay = up2(AY[p]), az = up2(AZ[p]);
    s_part[warp][0][32 * p + lane] = ax.x + ax.y;
    s_part[warp][1][32 * p + lane] = ay.x + ay.y;
    s_part[warp][2][32 * p + lane] = az.x + az.y;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < 3 * 32 * Q; t += kPairThreads) {
    const int c = t / (32 * Q), x = t % (32 * Q);
    float sum = 0.f;
#pragma unroll
    for (int w = 0; w < kPairWarps; ++w) sum += s_part[w][c][x];
    s_sum[c][x] = sum;
  }
  if (blocks > 1) cluster.sync();
  else __syncthreads();
  const int i = first + (int)threadIdx.x;
  if (rank == 0 && threadIdx.x < 32 * Q && i < n) {
    float4 v = vel[i];
    float a[3] = {0.f, 0.f, 0.f};
    for (int r = 0; r < blocks; ++r)
#pragma unroll
      for (int c = 0; c < NDIM; ++c) a[c] += cluster.map_shared_rank(&s_sum[c][threadIdx.x], r)[0];
    v.x += a[0];
    if (NDIM > 1) v.y += a[1];
    if (NDIM > 2) v.z += a[2];
    vel[i] = v;
  }
  if (blocks > 1) cluster.sync();  // no block leaves while its sums are read
}

}  // namespace

size_t fl_tree_bytes(int64_t n) {
  const size_t m = (size_t)(n > 1 ? n - 1 : 1), N = (size_t)(n > 0 ? n : 1);
  const size_t blocks = (N + kThreads - 1) / kThreads;
  return align256(4 * m) * 3 + align256(4 * N) + align256(8 * m) + align256(m) +
         align256(4 * m) * 3 + align256(16 * m) + align256(16 * N) +
         align256(16 * (2 * N + 1)) +
         align256(8 * (2 * N + 1)) * 2 + align256(4 * blocks) + align256(32 * N) +
         align256(32 * blocks) + align256(4 * m) + align256(4 * (2 * N)) +
         align256((size_t)fl_walk_slots(n) * kWalkSpillPerWarp * 16) + align256(4) + 256;
}

int fl_walk_slots(int64_t n) {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    sms = 1;
  const int64_t warps = (n > 0 ? n : 1) + 31 >> 5;
  const int64_t want = (warps + kWalkWarps - 1) / kWalkWarps * kWalkWarps;
  const int64_t cap = (int64_t)sms * kWalkBlocksPerSm * kWalkWarps;
  return (int)(want < cap ? want : cap);
}

void fl_tree_carve(FlTreeBufs* t, void* base, int64_t n, int ndim) {
  const size_t m = (size_t)(n > 1 ? n - 1 : 1), N = (size_t)(n > 0 ? n : 1);
  const size_t blocks = (N + kThreads - 1) / kThreads;
  char* p = static_cast<char*>(base);
  auto take = [&](size_t bytes) {
    void* r = p;
    p += align256(bytes);
    return r;
  };
  t->n = (int)n, t->ndim = ndim;
  t->levels = ndim == 3 ? 21 : 24;
  t->bits = t->levels * ndim;
  t->left = (uint32_t*)take(4 * m);
  t->right = (uint32_t*)take(4 * m);
  t->parent = (uint32_t*)take(4 * m);
  t->leaf_parent = (uint32_t*)take(4 * N);
  t->range = (uint32_t*)take(8 * m);
  t->depth = (uint8_t*)take(m);
  t->count = (uint32_t*)take(4 * m);
  t->first = (uint32_t*)take(4 * m);
  t->flag = (uint32_t*)take(4 * m);
  t->slot64 = (double*)take(8 * (2 * N + 1));
  t->cell = (float4*)take(16 * m);
  t->leaf = (float4*)take(16 * N);
  t->child_data = (float4*)take(16 * (2 * N + 1));
  t->child_meta = (uint2*)take(8 * (2 * N + 1));
  t->scan_scratch = take(4 * blocks);  // per-block totals of the child counts
  t->wsum = (double*)take(32 * N);
  t->wtiles = (double*)take(32 * blocks);  // per-block totals of the point records
  t->omask = (uint32_t*)take(4 * m);
  t->head_of = (uint32_t*)take(4 * (2 * N));
  t->walk_slots = fl_walk_slots(n);
  t->walk_blocks = 0;
  int dev = 0;
  cudaGetDevice(&dev);
  if (cudaDeviceGetAttribute(&t->sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || t->sms < 1)
    t->sms = 1;
  t->spill = (uint4*)take((size_t)t->walk_slots * kWalkSpillPerWarp * 16);
  t->work = (uint32_t*)take(4);
}

void fl_launch_morton(const float4* pos, int n, int ndim, const FlReduce* red, uint64_t* keys,
                      uint32_t* vals, uint32_t* hist, int lo_bit, float* cube_out,
                      cudaStream_t st) {
  // one full wave of large blocks (2 of 1024 threads per SM, so that enough loads are in
  // flight): each block flushes its digit histograms with up to 1024 global atomics (4
  // passes), so fewer blocks contend less for the same counters (8 blocks of 256 per SM took
  // 9.5 us more per 1M keys; 1 block of 1024, 4 us more)
  int g = (n + kMortonThreads - 1) / kMortonThreads;
  if (g > 2 * fl_sms()) g = 2 * fl_sms();
  if (g < 1) g = 1;
  k_morton<<<g, kMortonThreads, 0, st>>>(pos, n, ndim, red, keys, vals, hist, lo_bit, cube_out);
}

int fl_fixed_exponent(int64_t n, double wmax) {
  if (!(wmax > 0)) return 32;
  const int e = 62 - (int)std::ceil(std::log2((double)(n > 1 ? n : 1) * wmax));
  return e < 0 ? 0 : e > 100 ? 100 : e;
}

void fl_launch_build_points(const FlTreeBufs* t, const uint64_t* skeys, const uint32_t* perm,
                            const float4* pos, const float* strength, bool closed,
                            const float* cube, int fx_exp, cudaStream_t st, int64_t* launches,
                            FlSegs segs) {
  const int n = t->n;
  const int nb = (n + kThreads - 1) / kThreads;
  k_build<1><<<nb, kThreads, 0, st>>>(skeys, perm, pos, strength, n, t->ndim, t->left, t->right,
                                      t->parent, t->leaf_parent, t->range, t->depth, t->omask, t->leaf,
                                      closed ? reinterpret_cast<D4*>(t->wsum) : nullptr,
                                      reinterpret_cast<D4*>(t->wtiles), cube, fx_exp, segs);
  ++*launches;
  if (closed) {
    k_top4<<<1, kTopThreads, 0, st>>>(reinterpret_cast<D4*>(t->wtiles), nb);
    ++*launches;
  }
}

void fl_launch_build_nodes(const FlTreeBufs* t, const uint64_t* skeys, const uint32_t* perm,
                           const float4* pos, const float* strength, const float* cube,
                           int fx_exp, cudaStream_t st, int64_t* launches, FlSegs segs) {
  const int n = t->n;
  const int nb = (n + kThreads - 1) / kThreads;
  k_build<2><<<nb, kThreads, 0, st>>>(skeys, perm, pos, strength, n, t->ndim, t->left, t->right,
                                      t->parent, t->leaf_parent, t->range, t->depth, t->omask, t->leaf,
                                      nullptr, nullptr, cube, fx_exp, segs);
  ++*launches;
}

void fl_launch_build(const FlTreeBufs* t, const uint64_t* skeys, const uint32_t* perm,
                     const float4* pos, const float* strength, bool closed, const float* cube,
                     int fx_exp, cudaStream_t st, int64_t* launches, FlSegs segs) {
  // two kernels: the internal nodes' searches are latency chains that want every warp an SM
  // can hold, which the points' fixed-point records and prefix (more registers) would limit
  fl_launch_build_points(t, skeys, perm, pos, strength, closed, cube, fx_exp, st, launches, segs);
  fl_launch_build_nodes(t, skeys, perm, pos, strength, cube, fx_exp, st, launches, segs);
}

void fl_launch_frontier(const FlTreeBufs* t, const uint64_t* skeys, uint32_t* err,
                        cudaStream_t st, int64_t* launches) {
  const int n = t->n;
  const int g2 = (2 * n - 1 + kThreads - 1) / kThreads;
  k_frontier<<<g2, kThreads, 0, st>>>(n, t->ndim, skeys, t->parent, t->leaf_parent, t->range,
                                      t->depth, t->omask, t->head_of, err);
  ++*launches;
}

// The recursion, once every slot has its meta and the arrivals are zero.
static void launch_cells_up(const FlTreeBufs* t, int fp64_depth, uint32_t* err, cudaStream_t st,
                            int64_t* launches, FlSegs segs) {
  const int n = t->n, owned = kUpWarps * kUpNodes;
  // d3's c = Math.sqrt(4 / 2^dims), correctly rounded as IEEE sqrt is on host and device
  const double c1 = std::sqrt(4.0 / (double)(1 << t->ndim));
  k_cells_up<<<(n - 1 + owned - 1) / owned, kUpThreads, 0, st>>>(
      n, t->ndim, t->head_of, t->omask, t->depth, t->count, t->first,
      static_cast<const uint32_t*>(t->scan_scratch), t->range, t->flag, t->child_data, t->child_meta,
      t->slot64, fp64_depth, c1, err, segs);
  ++*launches;
}

void fl_launch_small_tree(const FlTreeBufs* t, const FlSortBufs* sb, const float4* pos, const float* strength,
                          const FlReduce* red, FlReduce* zero, bool closed, float sign, float* cube, int fx_exp,
                          int fp64_depth, uint32_t* err, cudaStream_t st, int64_t* launches) {
  const int n = t->n;
  SmallTree a;
  a.pos = pos, a.strength = strength, a.red = red, a.zero = zero;
  a.tmp = sb->keys[0], a.keys = sb->keys[1], a.vtmp = sb->vals[0], a.perm = sb->vals[1];
  a.cube = cube, a.err = err, a.t = *t, a.sign = sign, a.fx_exp = fx_exp;
  a.slots64 = !closed && fp64_depth != 0;
  static std::atomic<uint64_t> configured[2];  // zero: static
  // both kernels at the first launch, which is never inside a capture
  fl_raise_shared_limit(configured[0], (const void*)k_small_tree<false>, 13 * kSmallTreeMax);
  fl_raise_shared_limit(configured[1], (const void*)k_small_tree<true>, 13 * kSmallTreeMax);
  const int slice = kSmallRun * ((n + kSmallRun * kSmallBlocks - 1) / (kSmallRun * kSmallBlocks));
  int blocks = 1;
  while (blocks * slice < n) blocks *= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks);
  cfg.blockDim = dim3((unsigned)slice);
  cfg.dynamicSmemBytes = (size_t)(13 * small_align(n) > 12 * slice ? 13 * small_align(n) : 12 * slice);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)blocks, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr, cfg.numAttrs = blocks > 1 ? 1 : 0;
  if (closed) cudaLaunchKernelEx(&cfg, k_small_tree<true>, a);
  else cudaLaunchKernelEx(&cfg, k_small_tree<false>, a);
  ++*launches;
  if (!closed) launch_cells_up(t, fp64_depth, err, st, launches, FlSegs{});
}

void fl_launch_cells(const FlTreeBufs* t, bool closed, float sign, const float* cube, int fx_exp,
                     int fp64_depth, uint32_t* err, cudaStream_t st, int64_t* launches,
                     FlSegs segs) {
  const int n = t->n, m = n - 1;
  const int g = (m + kThreads - 1) / kThreads, g2 = (2 * n - 1 + kThreads - 1) / kThreads;
  uint32_t* ctot = static_cast<uint32_t*>(t->scan_scratch);
  const D4* P = reinterpret_cast<const D4*>(t->wsum);
  const D4* Ptot = reinterpret_cast<const D4*>(t->wtiles);
  if (closed)
    k_heads<true><<<g, kThreads, 0, st>>>(n, t->ndim, t->parent, t->range, t->depth, t->omask,
                                          t->count, t->first, ctot, sign, P, Ptot, t->leaf, cube,
                                          fx_exp, t->cell, t->flag, segs);
  else
    k_heads<false><<<g, kThreads, 0, st>>>(n, t->ndim, t->parent, t->range, t->depth, t->omask,
                                           t->count, t->first, ctot, sign, P, Ptot, t->leaf, cube,
                                           fx_exp, t->cell, t->flag, segs);
  k_top_u32<<<1, kTopThreads, 0, st>>>(ctot, g);
  *launches += 2;
  k_slots<<<g2, kThreads, 0, st>>>(n, t->ndim, t->head_of, t->omask, t->parent, t->range,
                                   t->depth, t->count, t->first, ctot, t->cell, t->leaf,
                                   t->child_data, t->child_meta, err, segs, !closed,
                                   closed || fp64_depth == 0 ? nullptr : t->slot64);
  ++*launches;
  if (!closed) launch_cells_up(t, fp64_depth, err, st, launches, segs);
}

void fl_launch_aggregate(const FlTreeBufs* t, const uint64_t* skeys, bool closed, float sign,
                         const float* cube, int fx_exp, int fp64_depth, uint32_t* err,
                         cudaStream_t st, int64_t* launches, FlSegs segs) {
  fl_launch_frontier(t, skeys, err, st, launches);
  fl_launch_cells(t, closed, sign, cube, fx_exp, fp64_depth, err, st, launches, segs);
}

// Blocks of this walk variant resident on one SM (queried once), at most kWalkBlocksPerSm.
template <int NDIM, int G, bool STATS, bool DMAX, bool BATCH>
int walk_blocks_per_sm() {
  // an atomic: host threads racing on the first query store the same value
  static std::atomic<int> blocks{0};
  int c = blocks.load(std::memory_order_relaxed);
  if (!c) {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_walk<NDIM, G, STATS, DMAX, BATCH>,
                                                      kWalkThreads, 0) != cudaSuccess || b < 1) {
      cudaGetLastError();
      b = 1;
    }
    c = b < kWalkBlocksPerSm ? b : kWalkBlocksPerSm;
    blocks.store(c, std::memory_order_relaxed);
  }
  return c;
}

template <int NDIM, bool STATS, bool DMAX>
int walk_lanes_blocks_per_sm() {
  static std::atomic<int> blocks{0};
  int c = blocks.load(std::memory_order_relaxed);
  if (!c) {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_walk_lanes<NDIM, STATS, DMAX>,
                                                      kWalkThreads, 0) != cudaSuccess || b < 1) {
      cudaGetLastError();
      b = 1;
    }
    c = b < kWalkBlocksPerSm ? b : kWalkBlocksPerSm;
    blocks.store(c, std::memory_order_relaxed);
  }
  return c;
}

int fl_walk_group_for(int n) { return n <= kLaneWalkMaxNodes ? 1 : 32; }

void fl_launch_walk(const FlTreeBufs* t, const uint32_t* perm, const float* cube, float4* vel,
                    float alpha, double theta2, double dmin2, double dmax2, uint32_t step,
                    uint32_t seed, uint32_t* err, unsigned long long* stats, int group,
                    cudaStream_t st, FlSegs segs, const FlTick* tk) {
  const int n = t->n;
  const int points = group == 16 && !segs.graphs ? 16 : 32;
  const int groups = segs.graphs ? segs.ngroups : (n + points - 1) / points;
  // a persistent grid of the blocks that fit on the device at once (and that the spill buffer
  // has regions for), each warp walking every (grid)-th group of 32 points
  const int cap = t->walk_slots / kWalkWarps;
  // the counter is 0 before a launch: zeroed with the scratch, and each launch's last claim puts
  // it back (a batch, whose tree buffers are carved anew as it grows, zeroes it here as well)
  if (segs.graphs) cudaMemsetAsync(t->work, 0, 4, st);
  const float fmax2 = dmax2 > 3e38 ? INFINITY : (float)dmax2;
#define FL_WALK_ONE(D, G, S, M, B)                                                             \
  do {                                                                                         \
    int per = walk_blocks_per_sm<D, G, S, M, B>();                                             \
    if (t->walk_blocks > 0 && t->walk_blocks < per) per = t->walk_blocks;                      \
    int g = t->sms * per;                                                                      \
    if (g > cap) g = cap;                                                                      \
    if (g < 1) g = 1;                                                                          \
    k_walk<D, G, S, M, B><<<g, kWalkThreads, 0, st>>>(                                         \
        t->child_data, t->child_meta, t->leaf, perm, cube, vel, n, alpha, theta2,              \
        (float)dmin2, fmax2, step, seed, err, stats, t->spill, groups, t->work, segs, tk);      \
  } while (0)
#define FL_WALK(D, G)                                                                          \
  do {                                                                                         \
    if (stats) FL_WALK_ONE(D, G, true, true, false);                                           \
    else if (fmax2 < INFINITY) FL_WALK_ONE(D, G, false, true, false);                          \
    else FL_WALK_ONE(D, G, false, false, false);                                               \
  } while (0)
  // a batch: distanceMax per graph (the walk tests it when any graph has a finite one)
#define FL_WALK_BATCH(D)                                                                       \
  do {                                                                                         \
    if (fmax2 < INFINITY) FL_WALK_ONE(D, 32, false, true, true);                               \
    else FL_WALK_ONE(D, 32, false, false, true);                                               \
  } while (0)
  if (!segs.graphs && group == 0) group = fl_walk_group_for(n);
  if (!segs.graphs && group == 1) {
    // one point per warp: no more blocks than the points need (the stacks are in shared
    // memory, so the grid needs no spill regions)
#define FL_LANES_ONE(D, S, M)                                                                  \
  do {                                                                                         \
    int per = walk_lanes_blocks_per_sm<D, S, M>();                                             \
    if (t->walk_blocks > 0 && t->walk_blocks < per) per = t->walk_blocks;                      \
    int g = t->sms * per;                                                                      \
    if (g > (n + kWalkWarps - 1) / kWalkWarps) g = (n + kWalkWarps - 1) / kWalkWarps;          \
    if (g < 1) g = 1;                                                                          \
    k_walk_lanes<D, S, M><<<g, kWalkThreads, 0, st>>>(                                         \
        t->child_data, t->child_meta, t->leaf, perm, cube, vel, n, alpha, theta2,              \
        (float)dmin2, fmax2, step, seed, err, stats, t->work, tk);                             \
  } while (0)
#define FL_LANES(D)                                                                            \
  do {                                                                                         \
    if (stats) FL_LANES_ONE(D, true, true);                                                    \
    else if (fmax2 < INFINITY) FL_LANES_ONE(D, false, true);                                   \
    else FL_LANES_ONE(D, false, false);                                                        \
  } while (0)
    if (t->ndim == 3) FL_LANES(3);
    else if (t->ndim == 2) FL_LANES(2);
    else FL_LANES(1);
#undef FL_LANES
#undef FL_LANES_ONE
  } else if (segs.graphs) {
    if (t->ndim == 3) FL_WALK_BATCH(3);
    else if (t->ndim == 2) FL_WALK_BATCH(2);
    else FL_WALK_BATCH(1);
  } else if (group == 32) {
    if (t->ndim == 3) FL_WALK(3, 32);
    else if (t->ndim == 2) FL_WALK(2, 32);
    else FL_WALK(1, 32);
  } else {
    if (t->ndim == 3) FL_WALK(3, 16);
    else if (t->ndim == 2) FL_WALK(2, 16);
    else FL_WALK(1, 16);
  }
#undef FL_WALK
#undef FL_WALK_BATCH
#undef FL_WALK_ONE
}

void fl_launch_allpairs(const float4* pos, const float* strength, float4* vel, int n, int ndim,
                        float alpha, float dmin2, float dmax2, uint32_t step, uint32_t seed,
                        cudaStream_t st, const FlTick* tk) {
  // two points per lane halve the reads of shared memory, one spreads a small layout over more
  // warps: 8,000 points take 49 us with one and 55 with two, 20,000 268 and 212. Clusters of 8
  // blocks, unless fewer give every SM 16 blocks (4 at 20,000 points: 215 us) or a warp has no tile
  const int q = n > kPairTwoPoints ? 2 : 1;
  const int units = (n + 32 * q - 1) / (32 * q);
  int blocks = kPairClusterMax;
  while (blocks > 1 && ((int64_t)units * blocks / 2 >= (int64_t)16 * fl_sms() || n <= 32 * kPairWarps * (blocks / 2)))
    blocks /= 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(units < 1 ? 1 : units) * (unsigned)blocks);
  cfg.blockDim = dim3(kPairThreads);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)blocks, attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr, cfg.numAttrs = blocks > 1 ? 1 : 0;
#define FL_PAIRS(D, Q, M) \
  cudaLaunchKernelEx(&cfg, k_allpairs<D, Q, M>, pos, strength, vel, n, alpha, dmin2, dmax2, step, seed, tk)
#define FL_PAIRS_DIM(D)                                              \
  do {                                                               \
    if (dmax2 < INFINITY) {                                          \
      if (q == 2) FL_PAIRS(D, 2, true);                              \
      else FL_PAIRS(D, 1, true);                                     \
    } else {                                                         \
      if (q == 2) FL_PAIRS(D, 2, false);                             \
      else FL_PAIRS(D, 1, false);                                    \
    }                                                                \
  } while (0)
  if (ndim == 3) FL_PAIRS_DIM(3);
  else if (ndim == 2) FL_PAIRS_DIM(2);
  else FL_PAIRS_DIM(1);
#undef FL_PAIRS_DIM
#undef FL_PAIRS
}

void fl_launch_bgraph(int graphs, int ndim, const int32_t* off, const FlReduce* red,
                      const FlBatchParams* prm, const double* alpha, FlGraph* gr, cudaStream_t st) {
  // A warp per graph has the shorter chain, while the FP64 pipe (2 lanes a clock) takes the warps of an SM
  // side by side; beyond that its one active lane costs what 32 would. 512 graphs: 7.5 us with a warp each,
  // 8.7 with a thread; 1,024: 10.1 and 8.7; 16,384: 89 and 9.4.
  if (graphs <= 4 * fl_sms())
    k_bgraph<true><<<(graphs + 3) / 4, 128, 0, st>>>(graphs, ndim, off, red, prm, alpha, gr);
  else
    k_bgraph<false><<<(graphs + 31) / 32, 32, 0, st>>>(graphs, ndim, off, red, prm, alpha, gr);
}

void fl_launch_bmorton(const float4* pos, int n, int ndim, const uint32_t* gid, const FlGraph* gr,
                       uint64_t* keys, uint32_t* vals, uint32_t* hist, int lo_bit, cudaStream_t st) {
  int g = (n + kMortonThreads - 1) / kMortonThreads;  // as fl_launch_morton
  if (g > 2 * fl_sms()) g = 2 * fl_sms();
  if (g < 1) g = 1;
  k_bmorton<<<g, kMortonThreads, 0, st>>>(pos, n, ndim, gid, gr, keys, vals, hist, lo_bit);
}

void fl_launch_bgidkey(int n, const uint32_t* mperm, const uint32_t* gid, const int32_t* off,
                       int graphs, int passes, uint64_t* keys, uint32_t* vals, uint32_t* hist,
                       cudaStream_t st) {
  // as fl_launch_morton: few, large blocks (each flushes its histograms with global atomics
  // and loads the graph offsets once)
  int g = (n + kMortonThreads - 1) / kMortonThreads;
  if (g > 2 * fl_sms()) g = 2 * fl_sms();
  if (g < 1) g = 1;
  k_bgidkey<<<g, kMortonThreads, 0, st>>>(n, mperm, gid, off, graphs, passes, keys, vals, hist);
}

void fl_launch_bgather(int n, const uint32_t* order2, const uint64_t* mkeys, const uint32_t* mperm,
                       const uint32_t* gid, uint64_t* skeys, uint32_t* perm, uint32_t* gid_pos,
                       cudaStream_t st) {
  k_bgather<<<(n + kThreads - 1) / kThreads, kThreads, 0, st>>>(n, order2, mkeys, mperm, gid,
                                                                 skeys, perm, gid_pos);
}
