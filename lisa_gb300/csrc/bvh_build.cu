// GPU BVH construction for the triangle soup.
//
// Replaces the closed optixAccelBuild call of the reference
// (src/LiSA/src/optix_wrapper.cc:92-145).  Pipeline, all on the device:
//   1. per-triangle AABB and centroid, scene and centroid bounds
//   2. 30-bit Morton code of each centroid
//   3. stable LSD radix sort of (code, triangle) pairs: one histogram of all
//      four digits, then 4 passes of 8 bits that rank a tile in shared memory
//      (warp match-any) and find its place by looking back over the tiles
//      before it (Adinets & Merrill, "Onesweep", 2022); written here without
//      a sort library
//   4. binary radix tree over the sorted codes (Karras, "Maximizing
//      Parallelism in the Construction of BVHs, Octrees, and k-d Trees",
//      HPG 2012), equal codes ordered by index
//   5. bottom-up AABBs with one atomic arrival counter per node
//   6. the least-cost plan of the 8-wide collapse, bottom up (renderers)
//   7. collapse into 8-wide nodes, level by level in one cooperative launch,
//      eight lanes per node: each node adopts up to 8 descendants, by the
//      plan and then, while slots are free, by opening the child of largest
//      surface area (subtrees of <= 3 triangles become leaves, split if
//      slots stay free), and stores its child
//      boxes quantised to 8 bits against a per-axis power-of-two grid,
//      rounded outward (compressed layout in the style of Ylitie, Karras,
//      Laine, "Efficient Incoherent Ray Traversal on GPUs Through Compressed
//      Wide BVHs", HPG 2017).  Leaf triangles are copied into leaf order.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "lisa_device.cuh"
#include "lisa_internal.h"

namespace lisa {
namespace {

constexpr uint32_t LEAF_BIT = 0x80000000u;

// bounds[0..2] = min scene xyz, [3..5] = max scene xyz, [6..8] min centroid,
// [9..11] max centroid, as order-preserving ints.  Blocks of 256.
__global__ void k_prim_bounds(const float* __restrict__ v, uint32_t n, float4* __restrict__ lo,
                              float4* __restrict__ hi, int* bounds) {
  float mn[6], mx[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    mn[k] = __int_as_float(0x7f800000);
    mx[k] = -__int_as_float(0x7f800000);
  }
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float* t = v + 9ull * i;
    float a[3], b[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      a[k] = fminf(fminf(t[k], t[3 + k]), t[6 + k]);
      b[k] = fmaxf(fmaxf(t[k], t[3 + k]), t[6 + k]);
      const float c = 0.5f * (a[k] + b[k]);
      mn[k] = fminf(mn[k], a[k]);
      mx[k] = fmaxf(mx[k], b[k]);
      mn[3 + k] = fminf(mn[3 + k], c);
      mx[3 + k] = fmaxf(mx[3 + k], c);
    }
    lo[i] = make_float4(a[0], a[1], a[2], 0.0f);
    hi[i] = make_float4(b[0], b[1], b[2], 0.0f);
  }
  // one set of atomics per block (per warp, they took longer than the scan:
  // 249 us of 1.31 M triangles, all on the same 12 words)
  __shared__ float red[8][12];
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    for (int o = 16; o > 0; o >>= 1) {
      mn[k] = fminf(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
      mx[k] = fmaxf(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
    }
    if ((threadIdx.x & 31) == 0) {
      red[threadIdx.x >> 5][k] = mn[k];
      red[threadIdx.x >> 5][6 + k] = mx[k];
    }
  }
  __syncthreads();
  if (threadIdx.x < 12) {
    const int k = threadIdx.x;
    float v = red[0][k];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) v = k < 6 ? fminf(v, red[w][k]) : fmaxf(v, red[w][k]);
    // red: min scene, min centroid, max scene, max centroid
    if (k < 6) atomicMin(&bounds[k < 3 ? k : k + 3], f2ord(v));
    else atomicMax(&bounds[k < 9 ? k - 3 : k], f2ord(v));
  }
}

__device__ __forceinline__ uint32_t expand10(uint32_t v) {
  v = (v * 0x00010001u) & 0xFF0000FFu;
  v = (v * 0x00000101u) & 0x0F00F00Fu;
  v = (v * 0x00000011u) & 0xC30C30C3u;
  v = (v * 0x00000005u) & 0x49249249u;
  return v;
}

#ifndef LISA_MORTON_SIZE_BITS
#define LISA_MORTON_SIZE_BITS 2
#endif

// Sort key: the triangle's size class above the 30-bit Morton code of its
// centroid (extended Morton codes, Vinkler, Bittner, Havran, HPG 2017), so
// large triangles -- walls, quads -- separate from the small ones near the
// root instead of overlapping every deep subtree.  Class 0 holds triangles
// whose box diagonal exceeds 1/8 of the scene's, then 1/64, 1/512.
__global__ void k_morton(const float4* __restrict__ lo, const float4* __restrict__ hi, uint32_t n,
                         const int* __restrict__ bounds, uint32_t* __restrict__ keys, uint32_t* __restrict__ vals) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 a = lo[i], b = hi[i];
  const float c[3] = {0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z)};
  uint32_t q[3];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float cmin = ord2f(bounds[6 + k]), cmax = ord2f(bounds[9 + k]);
    const float ext = cmax - cmin;
    float u = ext > 0.0f ? (c[k] - cmin) / ext : 0.5f;
    u = fminf(fmaxf(u, 0.0f), 1.0f);
    q[k] = min((uint32_t)(u * 1024.0f), 1023u);
  }
  uint32_t key = (expand10(q[0]) << 2) | (expand10(q[1]) << 1) | expand10(q[2]);
#if LISA_MORTON_SIZE_BITS > 0
  float s2 = 0.0f, t2 = 0.0f;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float se = ord2f(bounds[3 + k]) - ord2f(bounds[k]);
    s2 += se * se;
  }
  t2 = (b.x - a.x) * (b.x - a.x) + (b.y - a.y) * (b.y - a.y) + (b.z - a.z) * (b.z - a.z);
  // diagonal ratio thresholds 1/8, 1/64, 1/512 on squared lengths
  const uint32_t cls = t2 * 64.0f > s2 ? 0u : (t2 * 4096.0f > s2 ? 1u : (t2 * 262144.0f > s2 ? 2u : 3u));
  key |= cls << 30;
#endif
  keys[i] = key;
  vals[i] = i;
}

// ---- radix sort -----------------------------------------------------------
constexpr uint32_t RS_POLLS = 1u << 22;  // of a look-back wait, then the build fails

// Histograms of the four digits (hist: 4 x 256, zeroed before).
__global__ void __launch_bounds__(RS_THREADS) k_rs_hist(const uint32_t* __restrict__ keys, uint32_t n,
                                                       uint32_t* __restrict__ hist) {
  __shared__ uint32_t h[RS_PASSES][256];
#pragma unroll
  for (int d = 0; d < RS_PASSES; ++d) h[d][threadIdx.x] = 0;
  __syncthreads();
  for (uint32_t i = blockIdx.x * RS_THREADS + threadIdx.x; i < n; i += gridDim.x * RS_THREADS) {
    const uint32_t k = keys[i];
#pragma unroll
    for (int d = 0; d < RS_PASSES; ++d) atomicAdd(&h[d][(k >> (8 * d)) & 255u], 1u);
  }
  __syncthreads();
#pragma unroll
  for (int d = 0; d < RS_PASSES; ++d)
    if (h[d][threadIdx.x]) atomicAdd(&hist[256 * d + threadIdx.x], h[d][threadIdx.x]);
}

__device__ __forceinline__ uint32_t block_exclusive(uint32_t v) {
  __shared__ uint32_t ws[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) ws[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const int nw = blockDim.x >> 5;
    uint32_t s = lane < nw ? ws[lane] : 0u;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < nw) ws[lane] = s;
  }
  __syncthreads();
  return (warp > 0 ? ws[warp - 1] : 0u) + x - v;
}

// One pass over a tile of RS_THREADS x ROUNDS keys.  Tiles are numbered in
// the order their blocks start (a ticket), so a block only waits for blocks
// that run already.  look[tile][digit]: 0 = nothing yet, 1 << 30 | the tile's
// count, 2 << 30 | the count of all tiles up to it.  With five launches for
// the sort instead of twenty, its kernels take 42 us instead of 141 for
// 30,001 keys and 143 instead of 160 for 1.31 M (cold).
template <int ROUNDS>
__global__ void __launch_bounds__(RS_THREADS) k_rs_pass(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin,
                                                       uint32_t* __restrict__ kout, uint32_t* __restrict__ vout,
                                                       uint32_t n, int shift, const uint32_t* __restrict__ hist,
                                                       uint32_t* look, uint32_t* ticket, uint32_t* failed) {
  constexpr int WARPS = RS_THREADS / 32;
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_wc[WARPS][256];  // per warp: its count of each digit, then its first place in the tile
  __shared__ uint32_t s_base[256];       // place of the tile's first key of each digit
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_tile = atomicAdd(ticket, 1u);
#pragma unroll
  for (int w = 0; w < WARPS; ++w) s_wc[w][tid] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  const uint64_t base = (uint64_t)tile * (RS_THREADS * ROUNDS) + (uint32_t)(warp * 32 * ROUNDS + lane);
  const uint32_t lt = (1u << lane) - 1u;
  uint32_t key[ROUNDS], rank[ROUNDS];
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) key[r] = base + 32 * r < n ? kin[base + 32 * r] : 0u;
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    const bool valid = base + 32 * r < n;
    const uint32_t d = valid ? ((key[r] >> shift) & 255u) : 256u;
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    const uint32_t before = valid ? s_wc[warp][d] : 0u;
    __syncwarp();
    if (valid && (peers & lt) == 0u) s_wc[warp][d] = before + __popc(peers);
    __syncwarp();
    rank[r] = before + __popc(peers & lt);
  }
  __syncthreads();
  uint32_t count = 0;
#pragma unroll
  for (int w = 0; w < WARPS; ++w) {
    const uint32_t c = s_wc[w][tid];
    s_wc[w][tid] = count;
    count += c;
  }
  // the digit's keys in the tiles before this one
  uint32_t prefix = 0;
  volatile uint32_t* mine = look + (uint64_t)tile * 256 + tid;
  if (tile == 0) {
    *mine = (2u << 30) | count;
  } else {
    *mine = (1u << 30) | count;
    uint32_t polls = 0;
    for (int64_t t = (int64_t)tile - 1; t >= 0;) {
      const uint32_t v = *(volatile uint32_t*)(look + (uint64_t)t * 256 + tid);
      if ((v >> 30) == 0u) {
        if (++polls < RS_POLLS) continue;
        *failed = 1u;
        break;
      }
      prefix += v & 0x3fffffffu;
      if ((v >> 30) == 2u) break;
      --t;
    }
    *mine = (2u << 30) | (prefix + count);
  }
  const uint32_t first = block_exclusive(hist[tid]);
  s_base[tid] = first + prefix;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < ROUNDS; ++r) {
    if (base + 32 * r >= n) continue;
    const uint32_t d = (key[r] >> shift) & 255u;
    const uint32_t pos = s_base[d] + s_wc[warp][d] + rank[r];
    if (pos >= n) continue;  // (only after a failed wait)
    kout[pos] = key[r];
    vout[pos] = vin[base + 32 * r];
  }
}

// A sort whose wait ran out leaves places of its output unwritten and keys
// out of order, so the kernels behind it, which take indices from there,
// do nothing: the build then ends with its status alone.  (They look at the
// mark beside their first loads; waiting for it before those would add its
// latency to each.)

// ---- Karras radix tree ------------------------------------------------------
__device__ __forceinline__ int kdelta(const uint32_t* keys, int64_t n, int64_t i, int64_t j) {
  if (j < 0 || j >= n) return -1;
  const uint32_t a = keys[i], b = keys[j];
  if (a == b) return 32 + __clz((uint32_t)(i ^ j));
  return __clz(a ^ b);
}

__global__ void k_karras(const uint32_t* __restrict__ keys, uint32_t n, uint32_t* __restrict__ left,
                         uint32_t* __restrict__ right, uint32_t* __restrict__ first, uint32_t* __restrict__ last,
                         uint32_t* __restrict__ parent_int, uint32_t* __restrict__ parent_leaf,
                         const uint32_t* __restrict__ failed) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)n - 1) return;
  const uint32_t bad = *failed;
  const int64_t N = n;  // (keys in any order: every index below stays inside)
  const int d = (kdelta(keys, N, i, i + 1) - kdelta(keys, N, i, i - 1)) >= 0 ? 1 : -1;
  const int dmin = kdelta(keys, N, i, i - d);
  int64_t lmax = 2;
  while (kdelta(keys, N, i, i + lmax * d) > dmin) lmax <<= 1;
  int64_t l = 0;
  for (int64_t t = lmax >> 1; t >= 1; t >>= 1)
    if (kdelta(keys, N, i, i + (l + t) * d) > dmin) l += t;
  const int64_t j = i + l * d;
  const int dnode = kdelta(keys, N, i, j);
  int64_t s = 0, t = l;
  do {
    t = (t + 1) >> 1;
    if (kdelta(keys, N, i, i + (s + t) * d) > dnode) s += t;
  } while (t > 1);
  const int64_t gamma = i + s * d + (d < 0 ? -1 : 0);
  const int64_t lo = i < j ? i : j, hi = i < j ? j : i;
  const uint32_t lc = (lo == gamma) ? (LEAF_BIT | (uint32_t)gamma) : (uint32_t)gamma;
  const uint32_t rc = (hi == gamma + 1) ? (LEAF_BIT | (uint32_t)(gamma + 1)) : (uint32_t)(gamma + 1);
  if (bad != 0u) return;
  left[i] = lc;
  right[i] = rc;
  first[i] = (uint32_t)lo;
  last[i] = (uint32_t)hi;
  if (lc & LEAF_BIT) parent_leaf[lc & ~LEAF_BIT] = (uint32_t)i; else parent_int[lc] = (uint32_t)i;
  if (rc & LEAF_BIT) parent_leaf[rc & ~LEAF_BIT] = (uint32_t)i; else parent_int[rc] = (uint32_t)i;
  if (i == 0) parent_int[0] = 0xffffffffu;
}

__device__ __forceinline__ void node_box(uint32_t c, const uint32_t* vals, const float4* plo, const float4* phi,
                                         const float4* ilo, const float4* ihi, float4& lo, float4& hi) {
  if (c & LEAF_BIT) {
    const uint32_t p = vals[c & ~LEAF_BIT];
    lo = plo[p];
    hi = phi[p];
  } else {
    lo = __ldcg(ilo + c);
    hi = __ldcg(ihi + c);
  }
}

// ---- SAH refinement: treelet restructuring -----------------------------------
//
// One bottom-up pass over the binary LBVH (Karras & Aila, "Fast Parallel
// Construction of High-Quality Bounding Volume Hierarchies", HPG 2013): the
// thread that completes a node computes its box, primitive count and SAH
// cost, then takes the treelet of up to 7 leaves under it (grown by opening
// the treelet leaf of largest area) and rebuilds the treelet's internal
// nodes in the topology of least SAH cost, found by dynamic programming over
// the leaf subsets.  The treelet's leaves and everything below them stay as
// they are; every node keeps a box equal to the union of its children's.
// Node counts and costs overwrite the Karras ranges (first -> count,
// last -> cost bits), which the collapse no longer needs.

constexpr float SAH_CI = 1.2f;  // cost of a node visit relative to a triangle test
constexpr float SAH_CT = 1.0f;
constexpr int TL = 7;           // treelet leaves
// Subtrees of fewer primitives keep their LBVH topology: the planned 8-wide
// collapse makes nearly as much of it.  Against 64, 256 takes 26.3 visits a
// ray for 25.9 in the 4.48 M-triangle sphere soup (its frame 0.4 % longer),
// 4.81 for 4.79 in the 1.31 M-triangle icosphere box, and builds that in
// 0.10 ms less, 30,001 triangles in 0.05 ms (a tenth of a query of them).
constexpr uint32_t TREELET_MIN_PRIMS = 256;

__device__ __forceinline__ float4 box_min(float4 a, float4 b) {
  return make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), 0.0f);
}
__device__ __forceinline__ float4 box_max(float4 a, float4 b) {
  return make_float4(fmaxf(a.x, b.x), fmaxf(a.y, b.y), fmaxf(a.z, b.z), 0.0f);
}
__device__ __forceinline__ float box_half_area(float4 lo, float4 hi) {
  const float x = hi.x - lo.x, y = hi.y - lo.y, z = hi.z - lo.z;
  return x * y + y * z + z * x;
}

struct SahTree {
  uint32_t n;
  const uint32_t* vals;
  const float4* plo;
  const float4* phi;
  uint32_t* parent_leaf;
  uint32_t* parent_int;
  uint32_t* left;
  uint32_t* right;
  float4* ilo;
  float4* ihi;
  uint32_t* count;  // per internal node: primitives below
  float* cost;      // per internal node: SAH cost of its subtree
  uint32_t* flags;
  const uint32_t* failed;  // the sort's
};

// box, count and cost of a child (leaf or internal node, already complete)
__device__ __forceinline__ void sah_child(const SahTree& t, uint32_t c, float4& lo, float4& hi, uint32_t& cnt,
                                          float& cost) {
  if (c & LEAF_BIT) {
    const uint32_t q = t.vals[c & ~LEAF_BIT];
    lo = t.plo[q];
    hi = t.phi[q];
    cnt = 1;
    cost = SAH_CT * box_half_area(lo, hi);
  } else {
    lo = __ldcg(t.ilo + c);
    hi = __ldcg(t.ihi + c);
    cnt = __ldcg(t.count + c);
    cost = __ldcg(t.cost + c);
  }
}

// Per-warp shared state of one treelet's restructuring.
struct TreeletSmem {
  float opt[1 << TL];        // best SAH cost of each subset of the treelet's leaves
  uint8_t split[1 << TL];    // its best partition (one side)
  float4 llo[TL], lhi[TL];   // leaf boxes
  uint32_t lcnt[TL];
  uint32_t leaf[TL], inner[TL];
  uint32_t node[TL], set[TL];  // rebuilt nodes and the leaf subsets below them
  uint32_t child[TL][2];
};

// Subsets of up to 7 leaves by size: 21 pairs, 35 triples, 35 of four, 21 of
// five, 7 of six.
__constant__ uint8_t c_subset[119] = {
    3,   5,   6,   9,   10,  12,  17,  18,  20,  24,  33,  34,  36,  40,  48,  65,  66,  68,  72,  80,  96,
    7,   11,  13,  14,  19,  21,  22,  25,  26,  28,  35,  37,  38,  41,  42,  44,  49,  50,  52,  56,  67,  69,
    70,  73,  74,  76,  81,  82,  84,  88,  97,  98,  100, 104, 112,
    15,  23,  27,  29,  30,  39,  43,  45,  46,  51,  53,  54,  57,  58,  60,  71,  75,  77,  78,  83,  85,  86,
    89,  90,  92,  99,  101, 102, 105, 106, 108, 113, 114, 116, 120,
    31,  47,  55,  59,  61,  62,  79,  87,  91,  93,  94,  103, 107, 109, 110, 115, 117, 118, 121, 122, 124,
    63,  95,  111, 119, 123, 125, 126};

// Treelet restructuring (Karras and Aila, HPG 2013) of the subtree at
// `root`, by one warp.  Lane k holds the treelet's leaf k while it grows (the
// leaf of largest area is opened until there are TL), with its children's
// indices loaded ahead, so a step costs one memory latency.  The lanes then
// share the dynamic programme over the subsets of the leaves: all boxes
// first, then the subsets by size, several lanes for the partitions of the
// largest; and each rebuilds one node when the best topology is cheaper.
// What bounds the kernel is the chain of treelets from a leaf to the root:
// with the growth, the boxes and the rebuilding on one lane it took 351 us
// for 30,001 triangles and 2.4 ms for 1.31 M; so 180 us and 0.51 ms, and from
// 256 triangles on 125 us and 0.39 ms.  All 32 lanes call it with the same
// root.
__device__ void treelet_optimize_warp(const SahTree& t, uint32_t root, TreeletSmem& s) {
  const int lane = threadIdx.x & 31;
  __syncwarp();  // the root's box, count and cost, just written by its lane, are visible
  uint32_t id = LEAF_BIT, cnt = 0, lc = 0, rc = 0, inner = 0;
  float4 lo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), hi = lo;
  float cost = 0.0f;
  auto load = [&](uint32_t c) {
    id = c;
    if (!(c & LEAF_BIT)) {
      lc = __ldcg(t.left + c);
      rc = __ldcg(t.right + c);
    }
    sah_child(t, c, lo, hi, cnt, cost);
  };
  if (lane < 2) load(__ldcg((lane ? t.right : t.left) + root));
  int nl = 2;
  for (; nl < TL; ++nl) {
    // (areas are not negative, so their bits order as the floats)
    const bool open = lane < nl && !(id & LEAF_BIT);
    const uint32_t a = open ? __float_as_uint(box_half_area(lo, hi)) + 1u : 0u;
    const uint32_t best = __reduce_max_sync(0xffffffffu, a);
    if (best == 0u) break;
    const int owner = __ffs(__ballot_sync(0xffffffffu, a == best)) - 1;
    const uint32_t c = __shfl_sync(0xffffffffu, id, owner);
    const uint32_t l = __shfl_sync(0xffffffffu, lc, owner), r = __shfl_sync(0xffffffffu, rc, owner);
    if (lane == nl - 2) inner = c;
    if (lane == owner) load(l);
    else if (lane == nl) load(r);
  }
  if (nl < 3) return;  // two leaves have one topology
  const uint32_t full = (1u << nl) - 1u;
  if (lane < nl) {
    s.llo[lane] = lo;
    s.lhi[lane] = hi;
    s.lcnt[lane] = cnt;
    s.leaf[lane] = id;
    s.inner[lane] = inner;
    s.opt[1u << lane] = cost;
  }
  __syncwarp();
  // boxes of the subsets lane, lane + 32, + 64, + 96: the lane's bits choose
  // among the first five leaves
  {
    const float4 elo = make_float4(3.4e38f, 3.4e38f, 3.4e38f, 0.0f), ehi = make_float4(-3.4e38f, -3.4e38f, -3.4e38f, 0.0f);
    float4 blo = elo, bhi = ehi;
    for (int k = 0; k < 5 && k < nl; ++k)
      if (lane & (1 << k)) {
        blo = box_min(blo, s.llo[k]);
        bhi = box_max(bhi, s.lhi[k]);
      }
    for (uint32_t j = 0; j < 4; ++j) {
      const uint32_t sset = (uint32_t)lane + 32u * j;
      if (sset > full || (sset & (sset - 1u)) == 0u) continue;
      float4 ulo = blo, uhi = bhi;
      if (j & 1u) {
        ulo = box_min(ulo, s.llo[5]);
        uhi = box_max(uhi, s.lhi[5]);
      }
      if (j & 2u) {
        ulo = box_min(ulo, s.llo[6]);
        uhi = box_max(uhi, s.lhi[6]);
      }
      s.opt[sset] = SAH_CI * box_half_area(ulo, uhi);  // + the best partition's cost, below
    }
  }
  __syncwarp();
  // Best partition (P, S \ P) of a subset with its lowest member in P, each
  // once: P = low + fixed + a subset of `rest`; P = S is skipped.  The first
  // is taken whatever it costs: costs that overflow (thousands of triangles
  // that overlap, 1e17 across) must still leave a partition, or a subset
  // would be split into nothing and itself.
  auto best_partition = [&](uint32_t sset, uint32_t fixed, uint32_t rest, float& best, uint32_t& bp) {
    uint32_t q = rest;
    best = INFINITY;
    bp = 0;
    while (true) {
      const uint32_t pset = q | fixed;
      if (pset != sset) {
        const float c = s.opt[pset] + s.opt[sset ^ pset];
        if (bp == 0u || c < best) {
          best = c;
          bp = pset;
        }
      }
      if (q == 0u) break;
      q = (q - 1u) & rest;
    }
  };
  constexpr int FIRST[6] = {0, 0, 0, 21, 56, 91};  // of c_subset, by size
  constexpr int NUM[6] = {0, 0, 21, 35, 35, 21};
  for (int size = 2; size <= 5 && size <= nl; ++size) {
    for (int i = lane; i < NUM[size]; i += 32) {
      const uint32_t sset = c_subset[FIRST[size] + i];
      if (sset > full) continue;
      const uint32_t low = sset & (0u - sset);
      float best;
      uint32_t bp;
      best_partition(sset, low, sset ^ low, best, bp);
      s.opt[sset] += best;
      s.split[sset] = (uint8_t)bp;
    }
    __syncwarp();
  }
  if (nl >= 6) {
    // subsets of six: four lanes each, which fix the membership of the two
    // highest members
    const int i = lane >> 2;
    const uint32_t sset = i < 7 ? c_subset[112 + i] : 0xffu;
    float best = INFINITY;
    uint32_t bp = 0;
    if (sset <= full) {
      const uint32_t low = sset & (0u - sset);
      uint32_t rest = sset ^ low;
      const uint32_t h1 = 0x80000000u >> __clz(rest);
      rest ^= h1;
      const uint32_t h2 = 0x80000000u >> __clz(rest);
      rest ^= h2;
      best_partition(sset, low | ((lane & 1) ? h1 : 0u) | ((lane & 2) ? h2 : 0u), rest, best, bp);
    }
#pragma unroll
    for (int m = 1; m <= 2; m <<= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, m);
      const uint32_t op = __shfl_xor_sync(0xffffffffu, bp, m);
      if (ob < best || (ob == best && op < bp)) {
        best = ob;
        bp = op;
      }
    }
    if (sset <= full && (lane & 3) == 0) {
      s.opt[sset] += best;
      s.split[sset] = (uint8_t)bp;
    }
    __syncwarp();
  }
  if (nl == 7) {
    // the full set: the lane's bits are the membership of leaves 1..5
    float best;
    uint32_t bp;
    best_partition(full, 1u | ((uint32_t)lane << 1), 64u, best, bp);
#pragma unroll
    for (int m = 1; m <= 16; m <<= 1) {
      const float ob = __shfl_xor_sync(0xffffffffu, best, m);
      const uint32_t op = __shfl_xor_sync(0xffffffffu, bp, m);
      if (ob < best || (ob == best && op < bp)) {
        best = ob;
        bp = op;
      }
    }
    if (lane == 0) {
      s.opt[full] += best;
      s.split[full] = (uint8_t)bp;
    }
    __syncwarp();
  }
  if (!(s.opt[full] < __ldcg(t.cost + root) * (1.0f - 1e-6f))) {
    __syncwarp();
    return;
  }
  // rebuild: the root keeps its id, the other internal subsets reuse inner[]
  if (lane == 0) {
    int built = 1, next = 0;
    s.set[0] = full;
    s.node[0] = root;
    for (int i = 0; i < built; ++i) {
      const uint32_t sset = s.set[i];
      const uint32_t part[2] = {s.split[sset], sset ^ (uint32_t)s.split[sset]};
      for (int h = 0; h < 2; ++h) {
        if ((part[h] & (part[h] - 1u)) == 0u) {
          s.child[i][h] = s.leaf[__ffs(part[h]) - 1];
        } else {
          s.child[i][h] = s.node[built] = s.inner[next++];
          s.set[built++] = part[h];
        }
      }
    }
  }
  __syncwarp();
  if (lane < nl - 1) {  // a binary tree over nl leaves has nl - 1 nodes
    const uint32_t node = s.node[lane], sset = s.set[lane];
    for (int h = 0; h < 2; ++h) {
      const uint32_t c = s.child[lane][h];
      if (c & LEAF_BIT) __stcg(t.parent_leaf + (c & ~LEAF_BIT), node);
      else __stcg(t.parent_int + c, node);
    }
    __stcg(t.left + node, s.child[lane][0]);
    __stcg(t.right + node, s.child[lane][1]);
    float4 blo = make_float4(3.4e38f, 3.4e38f, 3.4e38f, 0.0f), bhi = make_float4(-3.4e38f, -3.4e38f, -3.4e38f, 0.0f);
    uint32_t n = 0;
    for (int k = 0; k < nl; ++k)
      if (sset & (1u << k)) {
        blo = box_min(blo, s.llo[k]);
        bhi = box_max(bhi, s.lhi[k]);
        n += s.lcnt[k];
      }
    __stcg(t.ilo + node, blo);
    __stcg(t.ihi + node, bhi);
    __stcg(t.count + node, n);
    __stcg(t.cost + node, s.opt[sset]);
  }
  __syncwarp();
}

// Bottom-up pass: boxes, primitive counts and SAH costs of the internal
// nodes, one leaf per lane climbing to the root; the second lane to reach a
// node finishes it (the first stops there).  Nodes with enough primitives
// below are restructured by the whole warp, one lane's node at a time, so
// the restructuring's dynamic programme runs on 32 lanes.
constexpr int SAH_THREADS = 256;

__global__ void __launch_bounds__(SAH_THREADS) k_bottom_up_sah(SahTree t, int refine) {
  __shared__ TreeletSmem tls[SAH_THREADS / 32];
  TreeletSmem& tl = tls[threadIdx.x >> 5];
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t p = (i < t.n && t.n >= 2) ? t.parent_leaf[i] : 0xffffffffu;
  bool active = p != 0xffffffffu && *t.failed == 0u;
  while (__any_sync(0xffffffffu, active)) {
    bool want = false;
    if (active) {
      __threadfence();
      if (atomicAdd(&t.flags[p], 1u) == 0u) {
        active = false;
      } else {
        __threadfence();
        float4 a0, a1, b0, b1;
        uint32_t ca, cb;
        float sa, sb;
        sah_child(t, __ldcg(t.left + p), a0, a1, ca, sa);
        sah_child(t, __ldcg(t.right + p), b0, b1, cb, sb);
        const float4 lo = box_min(a0, b0), hi = box_max(a1, b1);
        __stcg(t.ilo + p, lo);
        __stcg(t.ihi + p, hi);
        __stcg(t.count + p, ca + cb);
        __stcg(t.cost + p, SAH_CI * box_half_area(lo, hi) + sa + sb);
        want = refine && ca + cb >= TREELET_MIN_PRIMS;
      }
    }
    uint32_t m = __ballot_sync(0xffffffffu, want);
    while (m) {
      const int owner = __ffs(m) - 1;
      m &= m - 1;
      treelet_optimize_warp(t, __shfl_sync(0xffffffffu, p, owner), tl);
    }
    if (active) {
      p = __ldcg(t.parent_int + p);
      active = p != 0xffffffffu;
    }
  }
}

// ---- plan of the 8-wide collapse ------------------------------------------------
//
// The least cost of a subtree in m slots of an 8-wide node (m = 1..7) follows
// from its children's (the optimal collapse of Ylitie, Karras, Laine, HPG
// 2017): in one slot it is a leaf, or a node of its own whose eight slots its
// children share; in m slots it is that or its children share the m.  Costs
// count a node visit 1 and a triangle test PLAN_CT, by area.  Opening the
// largest child first instead takes 2.45 visits a ray in the Cornell box for
// 2.07, 26.9 for 26.3 in the 4.48 M-triangle soup and 4.90 for 4.81 in the
// icosphere box (frames 5, 3 and 2 % longer).  A third of a visit is what a
// test costs the traversal; 0.15 and 0.6 differ by under 1 %.
constexpr float PLAN_CT = 0.3f;

// Costs o[1..7] of a node over children of costs a, b; returns its splits:
// four bits for each m = 2..8, the slots of the left child, or 0 if m - 1
// slots cost no more.
__device__ __forceinline__ uint32_t plan_node(const float* a, const float* b, float area, uint32_t cnt, float* o) {
  uint32_t d = 0;
  float s8 = 0.0f;
#pragma unroll
  for (int m = 8; m >= 2; --m) {
    float best = 3.4e38f;
    uint32_t bk = 1;
#pragma unroll
    for (int k = 1; k < 8; ++k)
      if (k < m && m - k < 8) {
        const float v = a[k] + b[m - k];
        if (v < best) {
          best = v;
          bk = (uint32_t)k;
        }
      }
    d |= bk << (4 * (m - 2));
    if (m == 8) s8 = best;
    else o[m] = best;
  }
  o[1] = cnt <= 3u ? PLAN_CT * area * (float)cnt : area + s8;
#pragma unroll
  for (int m = 2; m < 8; ++m)
    if (!(o[m] < o[m - 1])) {
      o[m] = o[m - 1];
      d &= ~(15u << (4 * (m - 2)));
    }
  return d;
}

// One thread for each internal node over two leaves climbs from there: past a
// sibling that is a leaf at once, past an internal one if it comes second
// (the arrival flags stand at 2 after the bottom-up pass).  wide: two float4
// a node, its costs in 1..7 slots; plan: its splits.
//
// Bound by the latency of the climb, a dozen loads and an atomic a level, and
// of the low nodes' scattered loads: 165 us for 1.31 M triangles (cold), as
// much as it saves the first frame of 3.8 M rays.  On the way up in
// k_bottom_up_sah it took 200 us or more: that kernel lives on 64 warps an
// SM of 32 registers.  A build for a single query of some 10^5 rays (0.45 ms
// with the query) goes without.
__global__ void __launch_bounds__(256) k_wide_plan(SahTree t, float4* wide, uint32_t* plan) {
  uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p + 1 >= t.n) return;
  uint32_t l = t.left[p], r = t.right[p];
  if (!(l & r & LEAF_BIT) || *t.failed != 0u) return;
  while (true) {
    float c[2][8], o[8];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const uint32_t ch = h ? r : l;
      if (ch & LEAF_BIT) {
        const uint32_t q = t.vals[ch & ~LEAF_BIT];
        const float a = PLAN_CT * box_half_area(t.plo[q], t.phi[q]);
#pragma unroll
        for (int k = 1; k < 8; ++k) c[h][k] = a;
      } else {
        const float4 a = __ldcg(wide + 2ull * ch), b = __ldcg(wide + 2ull * ch + 1);
        c[h][1] = a.x;
        c[h][2] = a.y;
        c[h][3] = a.z;
        c[h][4] = a.w;
        c[h][5] = b.x;
        c[h][6] = b.y;
        c[h][7] = b.z;
      }
    }
    const uint32_t up = t.parent_int[p];
    plan[p] = plan_node(c[0], c[1], box_half_area(t.ilo[p], t.ihi[p]), t.count[p], o);
    __stcg(wide + 2ull * p, make_float4(o[1], o[2], o[3], o[4]));
    __stcg(wide + 2ull * p + 1, make_float4(o[5], o[6], o[7], 0.0f));
    if (up == 0xffffffffu) return;
    l = t.left[up];
    r = t.right[up];
    if (!((l | r) & LEAF_BIT)) {
      uint32_t seen;
      asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(seen) : "l"(t.flags + up) : "memory");
      if (seen == 2u) return;
    }
    p = up;
  }
}

// ---- collapse to 8-wide compressed nodes -------------------------------------

struct CollapseArgs {
  uint32_t n;
  const uint32_t* vals;
  const float4* plo;
  const float4* phi;
  const float4* ilo;
  const float4* ihi;
  const uint32_t* left;
  const uint32_t* right;
  const uint32_t* count;  // primitives below each internal node
  const uint32_t* plan;   // planned splits (plan_node), or null
  const float* verts;
  const int32_t* mats;  // material per triangle, or null
  uint4* nodes;
  float4* tris;
  uint32_t* source;     // binary node of each 8-wide node, in node order
  BvhDeviceInfo* info;
};

// Smallest e (within [-126, 127]) with 255 * 2^e >= ext.
__device__ __forceinline__ int grid_exponent(float ext) {
  if (!(ext > 0.0f)) return -126;
  const uint32_t q = __float_as_uint(__fdiv_ru(ext, 255.0f));  // 2^e >= q
  const int e = (int)(q >> 23) - 127 + ((q & 0x7fffffu) ? 1 : 0);
  return max(-126, min(127, e));
}

constexpr int COLLAPSE_THREADS = 128;

__device__ __forceinline__ uint64_t gpu_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// All blocks of the cooperative grid meet; false once a wait (bounded) has
// run out in some block.  Memory written before is visible after it to loads
// that bypass L1.
__device__ __forceinline__ bool collapse_barrier(BvhDeviceInfo* info, uint32_t k) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(&info->barrier, 1u);
    const uint32_t target = (k + 1) * gridDim.x;
    bool ok = false;
    for (uint32_t it = 0; it < (1u << 22); ++it) {
      uint32_t v;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&info->barrier) : "memory");
      if (v >= target) {
        ok = true;
        break;
      }
      __nanosleep(32);
    }
    if (!ok) atomicExch(&info->failed, 1u);
    s_ok = ok && *(volatile uint32_t*)&info->failed == 0u;
  }
  __syncthreads();
  return s_ok != 0;
}

// The node numbers are the work list: level l is the range of nodes that
// level l - 1 took, and source[node] says which binary node each stands for.
// Eight lanes collapse one node: lane k holds candidate k, its children's
// indices loaded ahead (a step of the growth costs one memory latency), and
// then quantises and writes child k.  Bound by those latencies, level after
// level: 70 us for 30,001 triangles and 269 for 1.31 M (295 with a plan to
// look up), where 24 launches with a thread per node and the grid in FP64
// took 589 and 1,200 (cold).
__global__ void __launch_bounds__(COLLAPSE_THREADS) k_collapse(CollapseArgs a) {
  const uint32_t FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, k = lane & 7, g0 = lane & 24;  // candidate, first lane of the group
  const uint32_t gmask = 0xffu << g0, glt = ((1u << lane) - 1u) & gmask;
  const uint32_t groups = gridDim.x * (COLLAPSE_THREADS / 8);
  const uint32_t group = (blockIdx.x * COLLAPSE_THREADS + threadIdx.x) >> 3;
  // (nothing to do after a failed sort: the first barrier then says so)
  uint32_t begin = 0, end = *(volatile uint32_t*)&a.info->failed ? 0u : 1u;
  for (uint32_t level = 0;; ++level) {
    // (whole warps run each round: the groups of a warp are consecutive)
    for (uint32_t w0 = begin + (group & ~3u); w0 < end; w0 += groups) {
      const uint32_t dst = w0 + (group & 3u);
      const bool active = dst < end;
      // candidates
      uint32_t id = LEAF_BIT, cnt = 0, lc = 0, rc = 0;
      float4 lo = make_float4(INFINITY, INFINITY, INFINITY, 0.0f), hi = make_float4(-INFINITY, -INFINITY, -INFINITY, 0.0f);
      auto load = [&](uint32_t c) {
        id = c;
        if (c & LEAF_BIT) {
          cnt = 1u;
        } else {
          cnt = a.count[c];
          lc = a.left[c];
          rc = a.right[c];
        }
        node_box(c, a.vals, a.plo, a.phi, a.ilo, a.ihi, lo, hi);
      };
      int nc = 0;
      uint32_t slots = 1;  // what the plan gives the candidate
      if (active) {
        const uint32_t src = __ldcg(a.source + dst);
        nc = !(src & LEAF_BIT) && a.count[src] > 3u ? 2 : 1;
        if (k < nc) load(nc == 1 ? src : (k ? a.right[src] : a.left[src]));
        if (nc == 2 && a.plan) {
          const uint32_t left = a.plan[src] >> 24;
          slots = k ? 8u - left : left;
        }
      }
      // the planned splits, all candidates at once: the right child of the
      // j-th that splits goes to lane nc + j
      while (a.plan) {
        uint32_t left = 0;
        if (k < nc && slots > 1u && !(id & LEAF_BIT)) {
          const uint32_t d = a.plan[id];
          while (slots > 1u && !(left = (d >> (4u * (slots - 2u))) & 15u)) --slots;
        }
        if (!__any_sync(FULL, left != 0u)) break;
        const uint32_t split = __ballot_sync(FULL, left != 0u) & gmask;
        const int j = k - nc, num = __popc(split);
        const bool take = j >= 0 && j < num;
        const int owner = take ? (int)__fns(split, 0u, j + 1) : lane;
        const uint32_t l = lc, r = __shfl_sync(FULL, rc, owner), rest = __shfl_sync(FULL, slots - left, owner);
        if (left) {
          load(l);
          slots = left;
        } else if (take) {
          load(r);
          slots = rest;
        }
        nc += num;
      }
      while (true) {
        // the openable candidate of largest area (its bits order as the
        // float), the first of equals: those that would become nodes, then,
        // while slots are free, leaves of two or three triangles (a slot
        // costs a ray nothing, a triangle test less: 3.7 -> 3.1 tests a ray
        // in the icosphere box, 2 % of a frame)
        const bool open = k < nc && nc < 8 && !(id & LEAF_BIT);
        uint32_t best = open ? ((__float_as_uint(box_half_area(lo, hi)) >> 1) | (cnt > 3u ? 0x40000000u : 0u)) + 1u : 0u;
        const uint32_t mine = best;
#pragma unroll
        for (int m = 1; m <= 4; m <<= 1) best = max(best, __shfl_xor_sync(FULL, best, m));
        const bool go = best != 0u;
        if (!__any_sync(FULL, go)) break;
        const uint32_t at = __ballot_sync(FULL, go && mine == best) & gmask;
        const int owner = at ? __ffs((int)at) - 1 : lane;
        const uint32_t l = __shfl_sync(FULL, lc, owner), r = __shfl_sync(FULL, rc, owner);
        if (go) {
          if (lane == owner) load(l);
          else if (k == nc) load(r);
          ++nc;
        }
      }
      // slots: internal children first, then leaves, in candidate order
      const bool is_int = k < nc && cnt > 3u, is_leaf = k < nc && !is_int;
      const uint32_t imask = __ballot_sync(FULL, is_int) & gmask, lmask = __ballot_sync(FULL, is_leaf) & gmask;
      const uint32_t num_int = __popc(imask);
      const uint32_t slot = is_int ? __popc(imask & glt) : is_leaf ? num_int + __popc(lmask & glt) : (uint32_t)k;
      uint32_t toff = is_leaf ? cnt : 0u;
#pragma unroll
      for (int m = 1; m <= 4; m <<= 1) {
        const uint32_t v = __shfl_up_sync(FULL, toff, m, 8);
        if (k >= m) toff += v;
      }
      const uint32_t num_tri = __shfl_sync(FULL, toff, 7, 8);
      toff -= is_leaf ? cnt : 0u;
      // node and triangle numbers, one atomic each per warp
      uint32_t child_base = num_int, tri_base = num_tri;
#pragma unroll
      for (int m = 8; m <= 16; m <<= 1) {
        const uint32_t u = __shfl_up_sync(FULL, child_base, m), v = __shfl_up_sync(FULL, tri_base, m);
        if (lane >= m) {
          child_base += u;
          tri_base += v;
        }
      }
      uint32_t b0 = 0, b1 = 0;
      if (lane == 31) {
        if (child_base) b0 = atomicAdd(&a.info->level[level % 3u], child_base);
        if (tri_base) b1 = atomicAdd(&a.info->tris, tri_base);
      }
      child_base += end + __shfl_sync(FULL, b0, 31) - num_int;
      tri_base += __shfl_sync(FULL, b1, 31) - num_tri;
      // node frame and grid
      float p[3] = {lo.x, lo.y, lo.z}, q[3] = {hi.x, hi.y, hi.z};
#pragma unroll
      for (int ax = 0; ax < 3; ++ax)
#pragma unroll
        for (int m = 1; m <= 4; m <<= 1) {
          p[ax] = fminf(p[ax], __shfl_xor_sync(FULL, p[ax], m));
          q[ax] = fmaxf(q[ax], __shfl_xor_sync(FULL, q[ax], m));
        }
      uint32_t leaves = is_leaf ? ((1u << cnt) - 1u) << (3u * slot) : 0u;
#pragma unroll
      for (int m = 1; m <= 4; m <<= 1) leaves |= __shfl_xor_sync(FULL, leaves, m);
      if (!active) continue;
      int e[3];
      uint8_t* bytes = (uint8_t*)a.nodes + (size_t)NODE_BYTES * dst + 32 + slot;
      const float clo[3] = {lo.x, lo.y, lo.z}, chi[3] = {hi.x, hi.y, hi.z};
#pragma unroll
      for (int ax = 0; ax < 3; ++ax) {
        e[ax] = grid_exponent(__fsub_ru(q[ax], p[ax]));
        // rounded outward: p + 2^e * ql <= lo and p + 2^e * qh >= hi exactly.
        // (Every whole number of steps up to 255 is a float, so a difference
        // rounded down has the floor of the exact one, and rounded up its
        // ceiling; likewise 255 * 2^e for the exponent.  FP64 would find no
        // tighter box.)
        uint32_t ql = 0, qh = 0;
        if (k < nc) {
          ql = (uint32_t)fminf(fmaxf(floorf(ldexpf(__fsub_rd(clo[ax], p[ax]), -e[ax])), 0.0f), 255.0f);
          qh = (uint32_t)fminf(fmaxf(ceilf(ldexpf(__fsub_ru(chi[ax], p[ax]), -e[ax])), 0.0f), 255.0f);
        }
        bytes[8 * ax] = (uint8_t)ql;
        bytes[8 * (3 + ax)] = (uint8_t)qh;
      }
      uint4* np = a.nodes + (size_t)(NODE_BYTES / 16) * dst;
      if (k == 0)
        np[0] = make_uint4(__float_as_uint(p[0]), __float_as_uint(p[1]), __float_as_uint(p[2]), (uint32_t)(e[0] + 127) << 23);
      if (k == 1)
        np[1] = make_uint4((uint32_t)(e[1] + 127) << 23, (uint32_t)(e[2] + 127) << 23, child_base, tri_base);
      if (k == 2) np[5] = make_uint4(leaves | (((1u << num_int) - 1u) << 24), 0u, 0u, 0u);
      if (is_int) a.source[child_base + slot] = id;
      if (is_leaf) {
        // the (at most 3) primitives below, left to right
        uint32_t leaf[3] = {id, 0u, 0u};
        if (cnt == 2u) {
          leaf[0] = lc;
          leaf[1] = rc;
        } else if (cnt == 3u) {
          const bool in_left = !(lc & LEAF_BIT);
          const uint32_t c = in_left ? lc : rc;
          const uint32_t x = a.left[c], y = a.right[c];
          leaf[0] = in_left ? x : lc;
          leaf[1] = in_left ? y : x;
          leaf[2] = in_left ? rc : y;
        }
#pragma unroll
        for (uint32_t j = 0; j < 3; ++j) {
          if (j >= cnt) break;
          const uint32_t prim = a.vals[leaf[j] & ~LEAF_BIT];
          const float* t = a.verts + 9ull * prim;
          float4* o = a.tris + (size_t)(TRI_BYTES / 16) * (tri_base + toff + j);
          const float id = __int_as_float((int)prim);
          o[0] = make_float4(t[0], t[3], t[6], id);
          o[1] = make_float4(t[1], t[4], t[7], id);
          o[2] = make_float4(t[2], t[5], t[8], id);
          o[3] = make_float4(__int_as_float(a.mats ? a.mats[prim] : 0), 0.0f, 0.0f, 0.0f);
        }
      }
    }
    // The nodes a level took are counted in one of three words, so that the
    // count stands still once the level is over: block 0 clears the next
    // level's, which all blocks read two barriers ago.
    if (blockIdx.x == 0 && threadIdx.x == 0) a.info->level[(level + 1u) % 3u] = 0u;
    if (!collapse_barrier(a.info, level)) return;
    begin = end;
    end += __ldcg(&a.info->level[level % 3u]);
    if (begin == end) {
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        a.info->nodes = end;
        a.info->depth = level + 1u;
        a.info->end_ns = gpu_ns();
      }
      return;
    }
  }
}

// Start values of a build: the tables that count up, the bounds, node 0 (the
// root).
__global__ void k_build_init(uint32_t* zero, uint64_t words, BvhDeviceInfo* info, uint32_t* source, uint32_t root,
                             uint32_t failed) {
  for (uint64_t i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += (uint64_t)gridDim.x * blockDim.x) zero[i] = 0u;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    BvhDeviceInfo b;
    b.nodes = b.tris = b.depth = b.barrier = 0u;
    b.failed = failed;
    b.begin_ns = gpu_ns();
    b.end_ns = 0u;
    for (int k = 0; k < 3; ++k) b.level[k] = 0u;
    for (int k = 0; k < 12; ++k) b.bounds[k] = (k / 3) & 1 ? (int)0x80000000 : 0x7fffffff;  // max, min
    for (int k = 0; k < RS_PASSES; ++k) b.ticket[k] = 0u;
    *info = b;
    source[0] = root;
  }
}

inline uint32_t cdiv(uint64_t a, uint64_t b) { return (uint32_t)((a + b - 1) / b); }

}  // namespace

namespace {
template <class T>
Status take(ScratchSource& src, T** p, uint64_t count, const char* what) {
  void* q = nullptr;
  LISA_TRY(src.get(&q, std::max<uint64_t>(count * sizeof(T), 16), what));
  *p = (T*)q;
  return Status();
}
}  // namespace

// what the kernels after the sort write
static const char *const BVH_TREE = "bvh tree", *const BVH_NODES = "bvh nodes", *const BVH_TRIS = "bvh triangles";

Status enqueue_bvh(const float* d_verts, uint32_t n, cudaStream_t s, ScratchSource& tmp, ScratchSource& out,
                   uint4** d_nodes, float4** d_tris, BvhDeviceInfo** d_info, const int32_t* d_mat, bool refine,
                   bool plan, bool sort_failed) {
  float4 *plo, *phi, *ilo, *ihi;
  uint32_t *keys, *vals, *keys2, *vals2;
  uint32_t *left, *right, *first, *last, *par_int, *par_leaf, *counted, *source;
  BvhDeviceInfo* info;
  const char *w = "bvh build scratch", *wt = BVH_TREE;
  LISA_TRY(take(tmp, &plo, n, w));
  LISA_TRY(take(tmp, &phi, n, w));
  LISA_TRY(take(tmp, &ilo, n, wt));
  LISA_TRY(take(tmp, &ihi, n, wt));
  LISA_TRY(take(tmp, &keys, n, w));
  LISA_TRY(take(tmp, &vals, n, w));
  LISA_TRY(take(tmp, &keys2, n, w));
  LISA_TRY(take(tmp, &vals2, n, w));
  LISA_TRY(take(tmp, &left, n, wt));
  LISA_TRY(take(tmp, &right, n, wt));
  LISA_TRY(take(tmp, &first, n, wt));
  LISA_TRY(take(tmp, &last, n, wt));
  LISA_TRY(take(tmp, &par_int, n, wt));
  LISA_TRY(take(tmp, &par_leaf, n, wt));
  LISA_TRY(take(tmp, &counted, counted_words(n), w));
  LISA_TRY(take(tmp, &source, max_nodes(n), w));
  LISA_TRY(take(tmp, &info, 1, w));
  float4* wide = nullptr;
  uint32_t* splits = nullptr;
  if (plan) {
    LISA_TRY(take(tmp, &wide, 2ull * n, wt));
    LISA_TRY(take(tmp, &splits, n, wt));
  }
  uint4* nodes = nullptr;
  float4* tris = nullptr;
  LISA_TRY(take(out, &nodes, (uint64_t)(NODE_BYTES / 16) * max_nodes(n), BVH_NODES));
  LISA_TRY(take(out, &tris, (uint64_t)(TRI_BYTES / 16) * n, BVH_TRIS));
  int dev = 0, sms = 0;
  LISA_CUDA(cudaGetDevice(&dev));
  LISA_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));

  const uint32_t root = n > 1 ? 0u : LEAF_BIT;
  k_build_init<<<std::min<uint32_t>(cdiv(counted_words(n), 1024), (uint32_t)sms * 8u), 256, 0, s>>>(
      counted, counted_words(n), info, source, root, sort_failed ? 1u : 0u);
  k_prim_bounds<<<std::min<uint32_t>(cdiv(n, 256), (uint32_t)sms * 8u), 256, 0, s>>>(d_verts, n, plo, phi, info->bounds);
  k_morton<<<cdiv(n, 256), 256, 0, s>>>(plo, phi, n, info->bounds, keys, vals);
  const uint32_t tiles = sort_tiles(n);
  uint32_t* hist = counted + (uint64_t)RS_PASSES * 256 * tiles;
  uint32_t* flags = hist + RS_PASSES * 256;
  k_rs_hist<<<std::min<uint32_t>(cdiv(n, RS_THREADS), (uint32_t)sms * 4u), RS_THREADS, 0, s>>>(keys, n, hist);
  for (int p = 0; p < RS_PASSES; ++p) {
    const uint32_t *ki = p & 1 ? keys2 : keys, *vi = p & 1 ? vals2 : vals;
    uint32_t *ko = p & 1 ? keys : keys2, *vo = p & 1 ? vals : vals2;
    uint32_t* look = counted + (uint64_t)p * 256 * tiles;
    if (rs_rounds(n) == 4)
      k_rs_pass<4><<<tiles, RS_THREADS, 0, s>>>(ki, vi, ko, vo, n, 8 * p, hist + 256 * p, look, &info->ticket[p],
                                                &info->failed);
    else
      k_rs_pass<16><<<tiles, RS_THREADS, 0, s>>>(ki, vi, ko, vo, n, 8 * p, hist + 256 * p, look, &info->ticket[p],
                                                 &info->failed);
  }
  LISA_CUDA(cudaGetLastError());
  if (n > 1) {
    k_karras<<<cdiv(n - 1, 256), 256, 0, s>>>(keys, n, left, right, first, last, par_int, par_leaf,
                                             &info->failed);
    // boxes, counts and SAH costs bottom up, with treelet restructuring
    // unless refine is off; first/last become count/cost
    const SahTree st{n, vals, plo, phi, par_leaf, par_int, left, right, ilo, ihi, first, (float*)last, flags,
                     &info->failed};
    k_bottom_up_sah<<<cdiv(n, SAH_THREADS), SAH_THREADS, 0, s>>>(st, refine ? 1 : 0);
    if (plan) k_wide_plan<<<cdiv(n - 1, 256), 256, 0, s>>>(st, wide, splits);
    LISA_CUDA(cudaGetLastError());
  }
  int occ = 0;
  LISA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_collapse, COLLAPSE_THREADS, 0));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(std::min<uint32_t>(cdiv(n, 256), (uint32_t)(sms * std::max(occ, 1))));
  cfg.blockDim = dim3(COLLAPSE_THREADS);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const CollapseArgs a{n, vals, plo, phi, ilo, ihi, left, right, first, splits, d_verts, d_mat, nodes, tris, source, info};
  LISA_CUDA(cudaLaunchKernelEx(&cfg, k_collapse, a));
  *d_nodes = nodes;
  *d_tris = tris;
  *d_info = info;
  return Status();
}

Status bvh_result(const BvhDeviceInfo& h, uint32_t n, BvhBuildResult* info) {
  if (h.failed) return Status(LISA_ERR_DEVICE, "bvh build: a device-side wait ran out");
  if (h.tris != n) return Status(LISA_ERR_DEVICE, "bvh build: leaf triangle count mismatch");
  info->num_nodes = h.nodes;
  info->num_tri_slots = h.tris;
  info->depth = h.depth;
  info->build_ms = 1e-6 * (double)(h.end_ns - h.begin_ns);
  for (int k = 0; k < 3; ++k) {
    info->bmin[k] = ord2f(h.bounds[k]);
    info->bmax[k] = ord2f(h.bounds[3 + k]);
  }
  return Status();
}

// A build whose sort is marked as failed from the start: its status, and how
// many words the kernels after the sort wrote.
Status selftest_bvh_failed(uint32_t n, uint32_t* written) {
  struct Spy : TempDeviceBufs {
    std::vector<std::pair<void*, size_t>> watched;
    Status get(void** p, size_t bytes, const char* what) override {
      bytes = (bytes + 3) & ~(size_t)3;
      LISA_TRY(TempDeviceBufs::get(p, bytes, what));
      LISA_CUDA(cudaMemset(*p, 0xa5, bytes));
      if (what == BVH_TREE || what == BVH_NODES || what == BVH_TRIS) watched.push_back({*p, bytes});
      return Status();
    }
  } spy;
  float* d_verts = nullptr;
  LISA_TRY(spy.get((void**)&d_verts, sizeof(float) * 9ull * n, "vertices"));
  LISA_CUDA(cudaMemset(d_verts, 0, sizeof(float) * 9ull * n));
  uint4* nodes = nullptr;
  float4* tris = nullptr;
  BvhDeviceInfo *d_info = nullptr, h;
  LISA_TRY(enqueue_bvh(d_verts, n, nullptr, spy, spy, &nodes, &tris, &d_info, nullptr, true, true, true));
  LISA_CUDA(cudaMemcpy(&h, d_info, sizeof(h), cudaMemcpyDeviceToHost));
  *written = h.nodes + h.tris + h.depth;
  for (const auto& b : spy.watched) {
    std::vector<uint32_t> words(b.second / 4);
    LISA_CUDA(cudaMemcpy(words.data(), b.first, b.second, cudaMemcpyDeviceToHost));
    for (uint32_t x : words) *written += x != 0xa5a5a5a5u;
  }
  BvhBuildResult info;
  return bvh_result(h, n, &info);
}

Status build_bvh(const float* d_verts, uint32_t n, cudaStream_t s, ScratchSource& tmp, ScratchSource& out,
                 uint4** d_nodes, float4** d_tris, BvhBuildResult* info, const int32_t* d_mat, bool refine) {
  *d_nodes = nullptr;
  *d_tris = nullptr;
  if (n == 0) {
    info->num_nodes = 0;
    info->num_tri_slots = 0;
    info->depth = 0;
    for (int k = 0; k < 3; ++k) info->bmin[k] = info->bmax[k] = 0.0f;
    return Status();
  }
  uint4* nodes = nullptr;
  float4* tris = nullptr;
  BvhDeviceInfo *d_info = nullptr, h;
  LISA_TRY(enqueue_bvh(d_verts, n, s, tmp, out, &nodes, &tris, &d_info, d_mat, refine, true));
  LISA_CUDA(cudaMemcpyAsync(&h, d_info, sizeof(h), cudaMemcpyDeviceToHost, s));
  LISA_CUDA(cudaStreamSynchronize(s));
  LISA_TRY(bvh_result(h, n, info));
  *d_nodes = nodes;
  *d_tris = tris;
  return Status();
}

}  // namespace lisa
