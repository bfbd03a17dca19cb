// forceCollide (src/collide.js:30-95) in the all-at-once form of the reference's GPU pass
// (src/gpu/passes/collide.js:5-17): every node takes its own share of every overlapping pair,
// against one snapshot of p + v (read as p and v_in; v_out is written, so nothing is copied):
//     d = s_i - s_j,  r = r_i + r_j;  |d| < r:  v_i += d (r - |d|) / |d| * strength * r_j^2 / (r_i^2 + r_j^2)
// A zero component of d is replaced by the pair's antisymmetric jiggle.
//
// Small graphs test every pair. Large graphs find the pairs with
// a uniform grid over cell-sorted nodes: cells 2 * max radius wide, so overlapping nodes sit in
// the same or adjacent cells. Each cell maps to a slot of a table of 2^bits >= 2n slots: cells
// are grouped in blocks (4^3, 8^2 or 64 cells) whose cells take consecutive slots in Morton
// order from a hashed block offset, so the sort by slot keeps nearby cells nearby. Two cells
// sharing a slot only cost extra distance tests; the 3^d neighbour cells of a node never share one
// (cells of one place in their blocks are at least a block's side apart). A slot's run of sorted
// nodes, [start, end), is written when it has one and never cleared: its words carry the low bits of
// the tick's step, and a run whose bits match is trusted only if the sorted keys confirm it. (If
// the slot has nodes now, its run was written now.)
#include "kernels.h"

namespace {

constexpr int kThreads = 256;

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// One pair's push on node idi (radius ri), if they overlap. Every rounding is spelt out, so that a
// pair pushes the same bit for bit wherever it is found. (The other node's id, perm[t] - first, or t
// itself without perm, is read only for a jiggle.)
__device__ __forceinline__ void pair_push(float3 me, float ri, float4 o, uint32_t idi,
                                          const uint32_t* __restrict__ perm, uint32_t t,
                                          uint32_t first, int ndim, float strength, uint32_t step,
                                          uint32_t seed, float3& acc) {
  const float rj = o.w, r = ri + rj;
  float dx = me.x - o.x, dy = ndim > 1 ? me.y - o.y : 0.f, dz = ndim > 2 ? me.z - o.z : 0.f;
  float l = __fmaf_rn(dz, dz, __fmaf_rn(dx, dx, __fmul_rn(dy, dy)));
  if (!(l < r * r)) return;
  if (dx == 0.f || (ndim > 1 && dy == 0.f) || (ndim > 2 && dz == 0.f)) {
    const uint32_t idj = perm ? perm[t] - first : t;
    if (dx == 0.f) dx = fl::jiggle(idi, idj, 0, step, seed), l = __fmaf_rn(dx, dx, l);
    if (ndim > 1 && dy == 0.f) dy = fl::jiggle(idi, idj, 1, step, seed), l = __fmaf_rn(dy, dy, l);
    if (ndim > 2 && dz == 0.f) dz = fl::jiggle(idi, idj, 2, step, seed), l = __fmaf_rn(dz, dz, l);
  }
  const float len = sqrtf(l);
  const float k = __fmul_rn(__fdiv_rn(__fsub_rn(r, len), len), strength);
  const float rj2 = __fmul_rn(rj, rj), w = __fdiv_rn(rj2, __fmaf_rn(ri, ri, rj2));
  acc.x = __fmaf_rn(__fmul_rn(dx, k), w, acc.x);
  acc.y = __fmaf_rn(__fmul_rn(dy, k), w, acc.y);
  acc.z = __fmaf_rn(__fmul_rn(dz, k), w, acc.z);
}

// Packed FP32 pairs (the f32x2 arithmetic of sm_100 and later).
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ float2 unpack2(uint64_t x) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
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

// Every pair of a small layout. The nodes j of one residue mod 16 push in order, and the 16 partial
// sums are added in order, so a node's sum does not depend on the launch. A block takes 8 nodes and
// its 128 threads 16 residues each: the block lays a tile of nodes out in shared memory, where nodes j
// and j + 16 lie as a pair for the packed arithmetic, and a thread tests its residue's pairs, two at a
// time (four: 22 us, eight: 26), with the very roundings of pair_push; those with an overlap go to
// pair_push one by one, from the registers of the test (read again from shared memory, half as many per
// load, 8,191 nodes that nearly all overlap took 233 us a tick, 188 so; with one scalar pair_push per
// pair 212). Bound by the reads of shared memory, two 16-byte loads a pair (11 us of them).
// 5,003 nodes in 2D (ncu): 45 us with one scalar pair_push per pair, now 20.
constexpr int kPairNodes = 8, kPairResidues = 16, kPairThreads = kPairNodes * kPairResidues;
constexpr int kPairTile = 512;  // 256 took 20.7 us, 1,024 20.3

template <int NDIM>
__global__ void __launch_bounds__(kPairThreads) k_collide_allpairs(
    const float4* __restrict__ pos, const float4* __restrict__ vel_in, float4* __restrict__ vel_out,
    const float* __restrict__ radius, int n, float strength, uint32_t step, uint32_t seed,
    const FlTick* __restrict__ tk) {
  if (tk) step = tk->step, seed = tk->seed;
  __shared__ float4 s_a[kPairTile / 2], s_b[kPairTile / 2];  // {x, x', y, y'}, {z, z', r, r'}
  __shared__ float3 s_part[kPairResidues][kPairNodes];
  const int residue = threadIdx.x / kPairNodes, x = threadIdx.x % kPairNodes;
  const int i = blockIdx.x * kPairNodes + x;
  const bool live = i < n;
  float4 p = make_float4(0, 0, 0, 0), v = p;
  float ri = 0.f;
  if (live) p = pos[i], v = vel_in[i], ri = radius[i];
  const float3 me = make_float3(p.x + v.x, p.y + v.y, p.z + v.z);
  const uint64_t MX = pack2(me.x, me.x), MY = pack2(me.y, me.y), MZ = pack2(me.z, me.z), R = pack2(ri, ri);
  float3 acc = make_float3(0.f, 0.f, 0.f);
  constexpr int kLoads = kPairTile / kPairThreads;
  float4 q[kLoads];
  auto load = [&](int base) {
#pragma unroll
    for (int k = 0; k < kLoads; ++k) {
      const int j = base + k * kPairThreads + (int)threadIdx.x;
      // past the end: a radius with which nothing overlaps
      q[k] = make_float4(0.f, 0.f, 0.f, __int_as_float(0x7fffffff));
      if (j < n) {
        const float4 a = pos[j], b = vel_in[j];
        q[k] = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, radius[j]);
      }
    }
  };
  load(0);
  for (int base = 0; base < n; base += kPairTile) {
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kLoads; ++k) {
      const int t = k * kPairThreads + (int)threadIdx.x;
      const int pair = (t >> 5) * kPairResidues + (t & 15), half = t >> 4 & 1;
      float* pa = reinterpret_cast<float*>(&s_a[pair]) + half;
      float* pb = reinterpret_cast<float*>(&s_b[pair]) + half;
      pa[0] = q[k].x, pa[2] = q[k].y, pb[0] = q[k].z, pb[2] = q[k].w;
    }
    __syncthreads();
    if (base + kPairTile < n) load(base + kPairTile);  // on its way during the tests
#pragma unroll 2
    for (int g = 0; g < kPairTile / 32; g += 2) {
      bool hit = false;
      float4 ta[2], tb[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const float4 a = ta[k] = s_a[(g + k) * kPairResidues + residue], b = tb[k] = s_b[(g + k) * kPairResidues + residue];
        const uint64_t DX = sub2(MX, pack2(a.x, a.y));
        uint64_t L;
        if (NDIM > 1) {
          const uint64_t DY = sub2(MY, pack2(a.z, a.w));
          L = fma2(DX, DX, mul2(DY, DY));
        } else {
          L = mul2(DX, DX);
        }
        if (NDIM > 2) {
          const uint64_t DZ = sub2(MZ, pack2(b.x, b.y));
          L = fma2(DZ, DZ, L);
        }
        const uint64_t S = add2(R, pack2(b.z, b.w));
        const float2 l = unpack2(L), r2 = unpack2(mul2(S, S));
        hit |= l.x < r2.x || l.y < r2.y;
      }
      if (!hit || !live) continue;
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int j = base + (g + k) * 32 + residue;
        const float4 a = ta[k], b = tb[k];
        if (j < n && j != i)
          pair_push(me, ri, make_float4(a.x, a.z, b.x, b.z), i, nullptr, j, 0u, NDIM, strength, step, seed, acc);
        if (j + 16 < n && j + 16 != i)
          pair_push(me, ri, make_float4(a.y, a.w, b.y, b.w), i, nullptr, j + 16, 0u, NDIM, strength, step, seed, acc);
      }
    }
  }
  s_part[residue][x] = acc;
  __syncthreads();
  if (!live || residue != 0) return;
  for (int r = 1; r < kPairResidues; ++r) {
    const float3 q = s_part[r][x];
    acc.x += q.x, acc.y += q.y, acc.z += q.z;
  }
  v.x += acc.x;
  if (NDIM > 1) v.y += acc.y;
  if (NDIM > 2) v.z += acc.z;
  vel_out[i] = v;
}

__device__ __forceinline__ uint32_t spread3_3(uint32_t x) {  // 2 bits -> bits 0, 3
  return (x & 1u) | ((x & 2u) << 2);
}
__device__ __forceinline__ uint32_t spread2_3(uint32_t x) {  // 3 bits -> bits 0, 2, 4
  return (x & 1u) | ((x & 2u) << 1) | ((x & 4u) << 2);
}

// Table slot of a cell: hashed block offset + the cell's Morton index inside its block.
__device__ __forceinline__ uint32_t cell_slot(int cx, int cy, int cz, int ndim, uint32_t mask) {
  uint32_t bx, by = 0, bz = 0, w;
  if (ndim == 3) {
    bx = (uint32_t)cx >> 2, by = (uint32_t)cy >> 2, bz = (uint32_t)cz >> 2;
    w = spread3_3(cx & 3) | spread3_3(cy & 3) << 1 | spread3_3(cz & 3) << 2;
  } else if (ndim == 2) {
    bx = (uint32_t)cx >> 3, by = (uint32_t)cy >> 3;
    w = spread2_3(cx & 7) | spread2_3(cy & 7) << 1;
  } else {
    bx = (uint32_t)cx >> 6;
    w = cx & 63;
  }
  const uint32_t h = fl::mix32(bx ^ fl::mix32(by ^ fl::mix32(bz + 0x9e3779b9u)));
  return ((h << 6) + w) & mask;
}

// A table entry's two words: the run's start and end (26 bits), tagged with the tick.
constexpr uint32_t kRunMask = (1u << 26) - 1;
__device__ __forceinline__ uint32_t run_word(uint32_t at, uint32_t step) { return at | step << 26; }

// The slots of a node's 3^NDIM neighbour cells, in the order z, y, x: a row of three cells along x
// lies in at most two blocks, so a row hashes at most two.
template <int NDIM>
struct Neighbours {
  int hx, hy, hz;
  uint32_t mask, seed;
  uint32_t hyz;            // the hash of the row's block so far
  uint32_t w;              // the row's place in its block
  template <bool BATCH = false>  // the graph's seed is xored to the block's z, the plain one added
  __device__ __forceinline__ void row(int dy, int dz) {
    const int cy = hy + dy, cz = hz + dz;
    if (NDIM == 3) {
      const uint32_t bz = (uint32_t)cz >> 2;
      hyz = fl::mix32((uint32_t)cy >> 2 ^ fl::mix32(BATCH ? bz ^ seed : bz + seed));
      w = spread3_3(cy & 3) << 1 | spread3_3(cz & 3) << 2;
    } else if (NDIM == 2) {
      hyz = fl::mix32((uint32_t)cy >> 3 ^ fl::mix32(seed));
      w = spread2_3(cy & 7) << 1;
    } else {
      hyz = fl::mix32(fl::mix32(seed));
      w = 0;
    }
  }
  __device__ __forceinline__ uint32_t slot(int dx) const {
    const int cx = hx + dx;
    const uint32_t bx = (uint32_t)cx >> (NDIM == 3 ? 2 : NDIM == 2 ? 3 : 6);
    const uint32_t wx = NDIM == 3 ? spread3_3(cx & 3) : NDIM == 2 ? spread2_3(cx & 7) : (uint32_t)cx & 63u;
    return ((fl::mix32(bx ^ hyz) << 6) + (wx | w)) & mask;
  }
};

// Bound by the latency of the table's and the nodes' loads, which land all over L2: a node looks at
// 27 cells, of which a sparse layout fills one in five. With one entry loaded after the other, a
// check of the keys before and at each start and a list of the slots seen, the query of 100,000
// nodes in 3D took 64 us, of 200,000 in 2D 30 us; now 22 and 21 (ncu).
// Visits the sorted nodes of a node's neighbour cells, in the order of the cells and, in a cell, of the
// sort: push(t, node t's record). KEY_SHIFT: the sorted keys' shift to a slot. The table's words of a
// whole plane of cells are loaded before the first is looked at, and a row's first nodes with the
// keys that confirm them, so that the loads overlap.
template <int NDIM, bool BATCH, typename Push>
__device__ __forceinline__ void visit_cells(Neighbours<NDIM> cells, const uint64_t* __restrict__ skeys,
                                            const uint2* __restrict__ runs,
                                            const float4* __restrict__ sorted, int n, int key_shift,
                                            uint32_t step, Push push) {
  constexpr int ROWS = NDIM > 1 ? 3 : 1, PLANES = NDIM > 2 ? 3 : 1;
  for (int p = 0; p < PLANES; ++p) {
    uint32_t slot[3 * ROWS];
    uint2 run[3 * ROWS];
#pragma unroll
    for (int y = 0; y < ROWS; ++y) {
      cells.template row<BATCH>(ROWS == 3 ? y - 1 : 0, PLANES == 3 ? p - 1 : 0);
#pragma unroll
      for (int k = 0; k < 3; ++k) slot[3 * y + k] = cells.slot(k - 1), run[3 * y + k] = runs[slot[3 * y + k]];
    }
#pragma unroll
    for (int y = 0; y < ROWS; ++y) {
      bool ok[3];
      float4 o[3];
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const uint32_t start = run[3 * y + k].x & kRunMask;
        ok[k] = !((run[3 * y + k].x ^ step << 26) >> 26) && start < (uint32_t)n;
        if (ok[k]) {
          o[k] = sorted[start];
          ok[k] = skeys[start] == (uint64_t)slot[3 * y + k] << key_shift;
        }
      }
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        if (!ok[k]) continue;
        const uint32_t end = min(run[3 * y + k].y & kRunMask, (uint32_t)n);
        uint32_t t = run[3 * y + k].x & kRunMask;
        for (;;) {
          push(t, o[k]);
          if (++t >= end) break;
          o[k] = sorted[t];
        }
      }
    }
  }
}

__device__ __forceinline__ int cell_coord(float s, float inv) {
  return (int)fminf(fmaxf(floorf(s * inv), -1073741824.f), 1073741824.f);
}

constexpr int kKeyThreads = 1024;
// the query's registers: 80 hold a plane's loads; 8 blocks (64) took 25 us for 22, 10 (48) 29
constexpr int kQueryThreads = 128, kQueryBlocks = 6;

__global__ void __launch_bounds__(kKeyThreads) k_grid_keys(const float4* __restrict__ pos,
                                                        const float4* __restrict__ vel, int n,
                                                        int ndim, float inv, int bits,
                                                        uint64_t* __restrict__ keys,
                                                        uint32_t* __restrict__ vals,
                                                        uint32_t* __restrict__ hist, int lo_bit) {
  __shared__ uint32_t sh[8 * 256];
  for (int i = threadIdx.x; i < 8 * 256; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const int passes = (64 - lo_bit + 7) / 8;
  const uint32_t mask = (1u << bits) - 1;
  const int stride = gridDim.x * blockDim.x;
  for (int base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const int i = base + threadIdx.x;
    const bool ok = i < n;
    uint64_t key = 0;
    if (ok) {
      float4 p = pos[i], v = vel[i];
      int cx = cell_coord(p.x + v.x, inv);
      int cy = ndim > 1 ? cell_coord(p.y + v.y, inv) : 0;
      int cz = ndim > 2 ? cell_coord(p.z + v.z, inv) : 0;
      key = (uint64_t)cell_slot(cx, cy, cz, ndim, mask) << (64 - bits);
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

// The slots' runs, and the sorted nodes' snapshot position and radius.
__global__ void __launch_bounds__(kThreads) k_grid_begin(const uint64_t* __restrict__ skeys,
                                                         const uint32_t* __restrict__ perm,
                                                         const float4* __restrict__ pos,
                                                         const float4* __restrict__ vel,
                                                         const float* __restrict__ radius, int n,
                                                         int bits, uint2* __restrict__ runs,
                                                         float4* __restrict__ sorted, uint32_t step,
                                                         const FlTick* __restrict__ tk) {
  if (tk) step = tk->step;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const uint64_t k = skeys[s];
  const uint32_t slot = (uint32_t)(k >> (64 - bits));
  if (s == 0 || skeys[s - 1] != k) runs[slot].x = run_word((uint32_t)s, step);
  if (s == n - 1 || skeys[s + 1] != k) runs[slot].y = run_word((uint32_t)s + 1u, step);
  const uint32_t i = perm[s];
  const float4 p = pos[i], v = vel[i];
  sorted[s] = make_float4(p.x + v.x, p.y + v.y, p.z + v.z, radius[i]);
}

template <int NDIM>
__global__ void __launch_bounds__(kQueryThreads, kQueryBlocks) k_grid_query(
    const uint64_t* __restrict__ skeys, const uint32_t* __restrict__ perm,
    const uint2* __restrict__ runs, const float4* __restrict__ sorted,
    const float4* __restrict__ vel_in, float4* __restrict__ vel_out, int n, int bits, float inv,
    float strength, uint32_t step, uint32_t seed, const FlTick* __restrict__ tk) {
  if (tk) step = tk->step, seed = tk->seed;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const float4 me4 = sorted[s];
  const uint32_t i = perm[s];
  const float3 me = make_float3(me4.x, me4.y, me4.z);
  const float ri = me4.w;
  Neighbours<NDIM> cells;
  cells.hx = cell_coord(me.x, inv), cells.hy = NDIM > 1 ? cell_coord(me.y, inv) : 0;
  cells.hz = NDIM > 2 ? cell_coord(me.z, inv) : 0;
  cells.mask = (1u << bits) - 1, cells.seed = 0x9e3779b9u;
  float3 acc = make_float3(0.f, 0.f, 0.f);
  visit_cells<NDIM, false>(cells, skeys, runs, sorted, n, 64 - bits, step, [&](uint32_t t, float4 o) {
    if (t != (uint32_t)s) pair_push(me, ri, o, i, perm, t, 0u, NDIM, strength, step, seed, acc);
  });
  float4 v = vel_in[i];
  v.x += acc.x;
  if (NDIM > 1) v.y += acc.y;
  if (NDIM > 2) v.z += acc.z;
  vel_out[i] = v;
}

// ---- batches: one grid over all the graphs of a batch, each with its own cell side

// The slot of a graph's cell: as cell_slot, the graph mixed into the hash of the block, so that
// different graphs' cells spread over the table (two sharing a slot only cost tests, and a node
// never pairs with another graph's).
__device__ __forceinline__ uint32_t bcell_slot(int cx, int cy, int cz, int ndim, uint32_t mask,
                                               uint32_t g) {
  uint32_t bx, by = 0, bz = 0, w;
  if (ndim == 3) {
    bx = (uint32_t)cx >> 2, by = (uint32_t)cy >> 2, bz = (uint32_t)cz >> 2;
    w = spread3_3(cx & 3) | spread3_3(cy & 3) << 1 | spread3_3(cz & 3) << 2;
  } else if (ndim == 2) {
    bx = (uint32_t)cx >> 3, by = (uint32_t)cy >> 3;
    w = spread2_3(cx & 7) | spread2_3(cy & 7) << 1;
  } else {
    bx = (uint32_t)cx >> 6;
    w = cx & 63;
  }
  const uint32_t h = fl::mix32(bx ^ fl::mix32(by ^ fl::mix32(bz ^ fl::mix32(g + 0x9e3779b9u))));
  return ((h << 6) + w) & mask;
}

// A node takes part in iteration `iter` when its graph has that many collide iterations and
// does not sit the tick out.
__device__ __forceinline__ bool bcollides(const FlGraph& g, int iter) {
  return g.citer > iter && !g.frozen;
}

__global__ void __launch_bounds__(kKeyThreads) k_bgrid_keys(
    const float4* __restrict__ pos, const float4* __restrict__ vel, int n, int ndim,
    const uint32_t* __restrict__ gid, const FlGraph* __restrict__ gr, int iter, int bits,
    uint64_t* __restrict__ keys, uint32_t* __restrict__ vals, uint32_t* __restrict__ hist,
    int lo_bit) {
  __shared__ uint32_t sh[8 * 256];
  for (int i = threadIdx.x; i < 8 * 256; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const int passes = (64 - lo_bit + 7) / 8;
  const uint32_t mask = (1u << bits) - 1;
  const int stride = gridDim.x * blockDim.x;
  for (int base = blockIdx.x * blockDim.x; base < n; base += stride) {
    const int i = base + threadIdx.x;
    const bool ok = i < n;
    uint64_t key = ~0ull;  // not taking part: after every cell
    if (ok) {
      const uint32_t g = gid[i];
      const FlGraph& G = gr[g];
      if (bcollides(G, iter)) {
        const float4 p = pos[i], v = vel[i];
        const int cx = cell_coord(p.x + v.x, G.cinv);
        const int cy = ndim > 1 ? cell_coord(p.y + v.y, G.cinv) : 0;
        const int cz = ndim > 2 ? cell_coord(p.z + v.z, G.cinv) : 0;
        key = (uint64_t)bcell_slot(cx, cy, cz, ndim, mask, g) << (63 - bits);
      }
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

// The slots' runs, and each sorted node's snapshot position, radius and graph.
__global__ void __launch_bounds__(kThreads) k_bgrid_begin(
    const uint64_t* __restrict__ skeys, const uint32_t* __restrict__ perm,
    const float4* __restrict__ pos, const float4* __restrict__ vel,
    const float* __restrict__ radius, const uint32_t* __restrict__ gid, int n, int bits,
    uint2* __restrict__ runs, float4* __restrict__ sorted, uint32_t* __restrict__ sgid,
    const FlTick* __restrict__ tk) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const uint64_t k = skeys[s];
  if (k == ~0ull) return;  // not taking part (and sorted after every node that does)
  const uint32_t slot = (uint32_t)(k >> (63 - bits));
  if (s == 0 || skeys[s - 1] != k) runs[slot].x = run_word((uint32_t)s, tk->step);
  if (s == n - 1 || skeys[s + 1] != k) runs[slot].y = run_word((uint32_t)s + 1u, tk->step);
  const uint32_t i = perm[s];
  const float4 p = pos[i], v = vel[i];
  sorted[s] = make_float4(p.x + v.x, p.y + v.y, p.z + v.z, radius[i]);
  sgid[s] = gid[i];
}

// Each node's pushes from the overlapping nodes of its own graph in the 3^d cells around its
// own (the jiggle's ids and step are the graph's own: the same alone or in any batch).
template <int NDIM>
__global__ void __launch_bounds__(kQueryThreads, kQueryBlocks) k_bgrid_query(
    const uint64_t* __restrict__ skeys, const uint32_t* __restrict__ perm,
    const uint2* __restrict__ runs, const float4* __restrict__ sorted,
    const uint32_t* __restrict__ sgid, const FlGraph* __restrict__ gr,
    const float4* __restrict__ vel_in, float4* __restrict__ vel_out, int n, int bits,
    const FlTick* __restrict__ tk) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const uint32_t i = perm[s];
  float4 v = vel_in[i];
  const uint64_t mykey = skeys[s];
  if (mykey != ~0ull) {
    const uint32_t g = sgid[s];
    const FlGraph& G = gr[g];
    const uint32_t first = (uint32_t)G.first, step = tk->step + G.tick0, seed = tk->seed;
    const float4 me4 = sorted[s];
    const float3 me = make_float3(me4.x, me4.y, me4.z);
    const float ri = me4.w, cinv = G.cinv, cstr = G.cstr;
    Neighbours<NDIM> cells;
    cells.hx = cell_coord(me.x, cinv), cells.hy = NDIM > 1 ? cell_coord(me.y, cinv) : 0;
    cells.hz = NDIM > 2 ? cell_coord(me.z, cinv) : 0;
    cells.mask = (1u << bits) - 1, cells.seed = fl::mix32(g + 0x9e3779b9u);
    float3 acc = make_float3(0.f, 0.f, 0.f);
    visit_cells<NDIM, true>(cells, skeys, runs, sorted, n, 63 - bits, tk->step, [&](uint32_t t, float4 o) {
      if (t != (uint32_t)s && sgid[t] == g)
        pair_push(me, ri, o, i - first, perm, t, first, NDIM, cstr, step, seed, acc);
    });
    v.x += acc.x;
    if (NDIM > 1) v.y += acc.y;
    if (NDIM > 2) v.z += acc.z;
  }
  vel_out[i] = v;
}

}  // namespace

void fl_launch_bgrid_keys(const float4* pos, const float4* vel, int n, int ndim,
                          const uint32_t* gid, const FlGraph* gr, int iter, int bits,
                          uint64_t* keys, uint32_t* vals, uint32_t* hist, int lo_bit,
                          cudaStream_t st) {
  int g = (n + kKeyThreads - 1) / kKeyThreads;  // as fl_launch_grid_keys
  if (g > 2 * fl_sms()) g = 2 * fl_sms();
  if (g < 1) g = 1;
  k_bgrid_keys<<<g, kKeyThreads, 0, st>>>(pos, vel, n, ndim, gid, gr, iter, bits, keys, vals,
                                          hist, lo_bit);
}

void fl_launch_bgrid_query(const FlGridBufs* g, const uint64_t* skeys, const uint32_t* perm,
                           const float4* pos, const float4* vel_in, float4* vel_out,
                           const float* radius, int ndim, const uint32_t* gid,
                           const FlGraph* gr, uint32_t* sgid, const FlTick* tk, cudaStream_t st,
                           int64_t* launches) {
  const int n = g->n, blocks = (n + kThreads - 1) / kThreads;
  k_bgrid_begin<<<blocks, kThreads, 0, st>>>(skeys, perm, pos, vel_in, radius, gid, n, g->bits,
                                             g->runs, g->sorted, sgid, tk);
  auto* query = ndim == 3 ? k_bgrid_query<3> : ndim == 2 ? k_bgrid_query<2> : k_bgrid_query<1>;
  query<<<(n + kQueryThreads - 1) / kQueryThreads, kQueryThreads, 0, st>>>(skeys, perm, g->runs, g->sorted, sgid, gr, vel_in, vel_out, n,
                                     g->bits, tk);
  *launches += 2;
}

void fl_launch_collide_allpairs(const float4* pos, const float4* vel_in, float4* vel_out,
                                const float* radius, int n, int ndim, float strength,
                                uint32_t step, uint32_t seed, cudaStream_t st, const FlTick* tk) {
  const int g = (n + kPairNodes - 1) / kPairNodes;
  auto* pairs = ndim == 3 ? k_collide_allpairs<3> : ndim == 2 ? k_collide_allpairs<2> : k_collide_allpairs<1>;
  pairs<<<g < 1 ? 1 : g, kPairThreads, 0, st>>>(pos, vel_in, vel_out, radius, n, strength, step, seed, tk);
}

size_t fl_grid_bytes(int64_t n) {
  int bits = 8;
  while ((int64_t(1) << bits) < 2 * n) ++bits;
  return align256(8 * ((size_t)1 << bits)) + align256(16 * (size_t)(n > 0 ? n : 1));
}

void fl_grid_carve(FlGridBufs* g, void* base, int64_t n) {
  int bits = 8;
  while ((int64_t(1) << bits) < 2 * n) ++bits;
  char* p = static_cast<char*>(base);
  g->n = (int)n, g->bits = bits;
  g->runs = (uint2*)p, p += align256(8 * ((size_t)1 << bits));
  g->sorted = (float4*)p;
}

void fl_launch_grid_keys(const float4* pos, const float4* vel, int n, int ndim, float inv_cell,
                         int bits, uint64_t* keys, uint32_t* vals, uint32_t* hist, int lo_bit,
                         cudaStream_t st) {
  // few, large blocks: each flushes its histograms with global atomics
  int g = (n + kKeyThreads - 1) / kKeyThreads;
  if (g > 2 * fl_sms()) g = 2 * fl_sms();
  if (g < 1) g = 1;
  k_grid_keys<<<g, kKeyThreads, 0, st>>>(pos, vel, n, ndim, inv_cell, bits, keys, vals, hist, lo_bit);
}

void fl_launch_grid_query(const FlGridBufs* g, const uint64_t* skeys, const uint32_t* perm,
                          const float4* pos, const float4* vel_in, float4* vel_out,
                          const float* radius, int ndim, float inv_cell, float strength,
                          uint32_t step, uint32_t seed, cudaStream_t st, int64_t* launches,
                          const FlTick* tk) {
  const int n = g->n, blocks = (n + kThreads - 1) / kThreads;
  k_grid_begin<<<blocks, kThreads, 0, st>>>(skeys, perm, pos, vel_in, radius, n, g->bits, g->runs,
                                            g->sorted, step, tk);
  auto* query = ndim == 3 ? k_grid_query<3> : ndim == 2 ? k_grid_query<2> : k_grid_query<1>;
  query<<<(n + kQueryThreads - 1) / kQueryThreads, kQueryThreads, 0, st>>>(skeys, perm, g->runs, g->sorted, vel_in, vel_out, n, g->bits,
                                     inv_cell, strength, step, seed, tk);
  *launches += 2;
}
