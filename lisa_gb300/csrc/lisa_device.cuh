// Device-side data layout and the closest-hit traversal.
//
// HBM layout of one scene (all arrays 16-byte aligned, read with 128-bit
// loads):
//   nodes  : 8-wide compressed BVH nodes, 96 B each, three 32-byte loads
//              0: origin x, y, z | scale x | scale y, z | child_base | tri_base
//              1: qlo.x[8] qlo.y[8] qlo.z[8] qhi.x[8] (bytes)
//              2: qhi.y[8] qhi.z[8] | leaf triangles (24 bits), imask (8 bits) | 0 0 0
//            child box = origin + scale * q (per axis; the scales are powers
//            of two).  Internal children come first: imask = 2^k - 1 for k of
//            them, at nodes child_base + slot.  Bit 3 c + q of the leaf
//            triangles says that leaf child c has a q-th triangle (at most
//            3); the node's triangles lie one after another from tri_base.
//            An empty slot has none of these bits.
//   tris   : 4 x float4 per leaf triangle slot, in leaf order: the three
//            vertices' x, y and z, each with the original triangle id as int
//            bits, and (material if that is an emitter, else -1; 0 0 0).  One
//            float4 per axis, so the triangle test loads the ray's shear axes
//            by address and selects nothing
//   prims  : 5 x float4 per original triangle (shading record):
//            (v0, n0.x) (v1, n0.y) (v2, n0.z) (n1, n2.x) (n2.y, n2.z, mat, 0)
//   mats   : DevMaterial, 48 B each
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "bvh_sizes.h"
#include "device_math.cuh"

namespace lisa {

enum : int { MAT_OPAQUE = 0, MAT_DIELECTRIC = 1, MAT_EMIT = 2 };

struct DevMaterial {
  float albedo[3];
  float roughness;
  float emission[3];
  float ior;
  int cls;
  float alpha;
  float light_pdf;  // physically based estimator: area pdf (luminance / total) of its emitters
  int pad;
};
static_assert(sizeof(DevMaterial) == 48, "DevMaterial layout");

constexpr float RAY_TMIN = 1e-4f;  // shader.cu:114,202
constexpr float RAY_TMAX = 1e16f;  // shader.cu:115,202
constexpr int NEE_TRIES = 30;      // shader.cu:199
// emissive triangles from which the emitter search uses their own BVH (with
// fewer, the bounds test of the emitter search is as selective)
constexpr uint32_t EMIT_BVH_MIN_TRIS = 32;
// Entries of a ray's traversal stack.  A node pushes up to seven of its
// children, so a tree of depth d takes at most 7 (d - 1): none of up to 33
// levels overflows it (a deeper one may, which sets ST_STACK_OVERFLOW).  The
// scenes here have 6 to 12 levels and use up to 20 entries; soups of six
// million triangles of sizes that span 2^120, or that all overlap, 17 to 29
// levels and up to 110, where 64 entries failed.  Its unused part costs no
// time, only local memory that the driver reserves (1.75 KB a resident thread).
constexpr int TRAV_STACK = 224;

enum StatusBits : uint32_t {
  ST_STACK_OVERFLOW = 1u,
  ST_QUEUE_OVERFLOW = 2u,
  ST_BAD_WAVE = 4u,
  ST_GUIDE_NONFINITE = 8u,
  // 16: a bounded tensor-core wait ran out (LISA_STATUS_WAIT_TIMEOUT)
  ST_BOUNDS = 32u,  // bounds-checked builds: a BVH or triangle index out of range
  ST_BVH_BUILD = 64u,  // a BVH built and traced without the host in between failed to build
};

// Bounds-checked builds (-DLISA_BOUNDS, a stand-in for a memory checker):
// node and triangle indices read from the BVH and the queue slots that
// appends reserve are checked before use; a bad one sets a status bit and
// the access is skipped.  Queue sizes are bounded by construction (one entry
// per path and depth), so in ordinary builds the checks compile away.

struct SceneDev {
  const uint4* nodes;
  const float4* tris;
  const float4* prims;
  const DevMaterial* mats;
  uint32_t num_prims;
  uint32_t num_nodes;
  uint32_t num_mats;
  float extent;  // bounding-box diagonal
  uint32_t width, height;
  uint32_t num_bounces;
  uint32_t pad0;
  float eye[3], U[3], V[3], W[3];
  float lens_radius;  // 0 = pinhole
  float focal_distance;
  float unitU[3], unitV[3], unitW[3];
  float bmin[3], bmax[3];  // scene bounds (guide encoding)
  // accumulation, one entry per pixel
  float4* acc_sum;   // Kahan sum (xyz)
  float4* acc_comp;  // Kahan compensation (xyz)
  double* acc_sq;    // 3 doubles: sum of squares
  double* acc_sum64; // 3 doubles: FP64 sum (accum_fp64 only, else null)
  uint32_t* pix_rng; // reference per-pixel stream state (LISA_RNG_PER_PIXEL)
  int32_t guide;     // guide slot of this scene (-1 = none)
  int32_t pad1;
  // physically based estimator: emitters, 4 float4 each --
  // (v0.xyz, area pdf) (e1 = v1-v0, material bits) (e2 = v2-v0, 0) (unit normal, 0)
  // -- and the CDF over area x luminance that picks them
  const float4* emit;
  const float* emit_cdf;
  uint32_t num_emit;
  uint32_t has_emit_box;     // the scene has emissive triangles, all inside emit_lo..emit_hi
  float emit_lo[3], emit_hi[3];
  // BVH over the emissive triangles alone (0 nodes = none): the emitter
  // search asks it first whether a ray meets an emitter at all
  const uint4* enodes;
  const float4* etris;
  uint32_t num_enodes;
  uint32_t num_etris;
};

// One group of a wave: `nplanes` consecutive sample planes of pixels
// [pix0, pix0+npix) of one scene.  slot = slot0 + m*npix + (p - pix0).
struct WaveGroup {
  uint32_t scene;
  uint32_t pix0, npix;
  uint32_t sample0, nplanes;
  uint32_t slot0;
  uint32_t acc0;  // prefix of npix over the wave's groups (accumulate index)
  uint32_t pad;
};
constexpr int MAX_GROUPS = 128;
struct WaveDesc {
  uint32_t num_groups;
  uint32_t paths;
  uint32_t acc_items;  // sum of npix
  uint32_t rng_mode;
  uint32_t seed;
  uint32_t pad[3];
  WaveGroup groups[MAX_GROUPS];
};

enum { HEAD_TRACE = 0, HEAD_NEE = 2 };
struct WaveCtrl {
  uint32_t qcount[2];
  uint32_t nee_count;
  uint32_t train_count;
  uint32_t head[4];
  uint32_t status;
  uint32_t guided_count;  // guided vertices of the current wave
  uint32_t rec_count;     // training records kept in the current wave
  float drop_prob;        // probability of not keeping a guided vertex's record (0 = keep all)
  unsigned long long rays_primary;
  unsigned long long rays_bounce;
  unsigned long long rays_shadow;
  unsigned long long node_visits[2];  // [0] closest-hit stage, [1] emitter search
  unsigned long long tri_tests[2];
  unsigned long long nee_total;
  unsigned long long shadow_walked;   // emitter-search rays that walked the BVH
  unsigned long long infer_rows;      // emitter-queue entries the guide's inference ran on
  unsigned long long train_samples;   // samples of the guide's training steps
};

// ---------------------------------------------------------------------------
// Watertight ray/triangle test (Woop, Benthin, Wald, "Watertight
// Ray/Triangle Intersection", JCGT 2013), evaluated with one rounding per
// operation and no FMA so the host oracle reproduces every hit bit for bit.

struct RayPre {
  float ox, oy, oz;
  float ix, iy, iz;  // 1/d per axis
  float slack;       // absolute slack on the best distance, in t units
};
// The shear of the triangle test, along the axis kz of the largest |d|, and
// the origin on the shear's axes kx = kz + 1, ky = kz + 2 (mod 3), kz.
struct RayShear {
  float Sx, Sy, Sz;
  int kz;
  V3 o;
};

// Components of a vector on the shear's axes.  The published test swaps kx
// and ky for a negative d[kz] to keep the winding; that negates U, V, W, det
// and T exactly (each is a difference or a sum of products) and leaves t as
// it is, so here they stay.
__device__ __forceinline__ V3 on_shear_axes(V3 v, int kz) {
  return v3(kz == 0 ? v.y : (kz == 1 ? v.z : v.x), kz == 0 ? v.z : (kz == 1 ? v.x : v.y),
            kz == 0 ? v.x : (kz == 1 ? v.y : v.z));
}

__device__ __forceinline__ void ray_prepare(V3 o, V3 d, float extent, RayPre& r, RayShear& h) {
  r.ox = o.x;
  r.oy = o.y;
  r.oz = o.z;
  const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
  const int kz = (ax > ay) ? ((ax > az) ? 0 : 2) : ((ay > az) ? 1 : 2);
  const V3 dk = on_shear_axes(d, kz);
  h.kz = kz;
  h.o = on_shear_axes(o, kz);
  h.Sx = fdiv(dk.x, dk.z);
  h.Sy = fdiv(dk.y, dk.z);
  // __frcp_rn is the correctly rounded 1/x, the same value as 1.0f/x: the
  // shear's 1/dz, and the node-culling reciprocal of that (dominant) axis
  h.Sz = __frcp_rn(dk.z);
  // The other two axes' reciprocals serve node culling only; __fdividef is
  // within 2 ulp there, which the slab padding covers (see trav_node).  A
  // zero or vanishing component's is limited to 1e20 of the dominant one's:
  // the node test then keeps that axis's slab (the ray's constant coordinate
  // against the padded box) instead of turning it into NaN and dropping it,
  // which made such rays visit most of the tree.
  const float most = 1e20f * fabsf(h.Sz);
  const float qx = copysignf(fminf(fabsf(__fdividef(1.0f, d.x)), most), d.x);
  const float qy = copysignf(fminf(fabsf(__fdividef(1.0f, d.y)), most), d.y);
  const float qz = copysignf(fminf(fabsf(__fdividef(1.0f, d.z)), most), d.z);
  r.ix = kz == 0 ? h.Sz : qx;
  r.iy = kz == 1 ? h.Sz : qy;
  r.iz = kz == 2 ? h.Sz : qz;
  // 2^-18 * extent / |d|max; a margin, so an approximate quotient will do
  r.slack = __fdividef(3.814697265625e-6f * extent, fmaxf(ax, fmaxf(ay, az)));
}

// Returns t of the hit (or +inf) of the triangle whose vertices are a, b, c
// on the shear's axes.  prim_t < tbest test is the caller's.
__device__ __forceinline__ float intersect_tri(const RayShear& h, V3 va, V3 vb, V3 vc, float tmin) {
  // translate to the ray origin
  const V3 a = va - h.o, b = vb - h.o, c = vc - h.o;
  // shear
  const float Axs = fsub(a.x, fmul(h.Sx, a.z)), Ays = fsub(a.y, fmul(h.Sy, a.z));
  const float Bxs = fsub(b.x, fmul(h.Sx, b.z)), Bys = fsub(b.y, fmul(h.Sy, b.z));
  const float Cxs = fsub(c.x, fmul(h.Sx, c.z)), Cys = fsub(c.y, fmul(h.Sy, c.z));
  // scaled barycentrics (edge functions)
  const float U = fsub(fmul(Cxs, Bys), fmul(Cys, Bxs));
  const float V = fsub(fmul(Axs, Cys), fmul(Ays, Cxs));
  const float W = fsub(fmul(Bxs, Ays), fmul(Bys, Axs));
  if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return __int_as_float(0x7f800000);
  const float det = fadd(fadd(U, V), W);
  if (det == 0.0f) return __int_as_float(0x7f800000);
  const float Az = fmul(h.Sz, a.z), Bz = fmul(h.Sz, b.z), Cz = fmul(h.Sz, c.z);
  const float T = fadd(fadd(fmul(U, Az), fmul(V, Bz)), fmul(W, Cz));
  const float t = fdiv(T, det);
  if (!(t > tmin)) return __int_as_float(0x7f800000);
  return t;
}

// ---------------------------------------------------------------------------
// Closest-hit traversal of the 8-wide compressed BVH, one node per step.
//
// Box tests are made conservative by padding each slab distance by
// 2^-20 (|c| + 512 |s|) with s = 2^e/d and c = (p-o)/d.  A slab is
// f s + (c - 1024 s -+ pad), f = 1024 + q, the half-precision number whose
// bits are 0x6400 | q: two roundings of 2^-24 (|c| + 1024 |s|) in the
// constant; 1/d within 2 ulp, p-o, the products and the padding's own
// subtraction are about 9 * 2^-24 (|c| + 255 |s|).  Together that is
// 2^-24 (11 |c| + 4343 |s|) against 2^-24 (16 |c| + 8192 |s|) -- so the
// traversal never culls a box the exact ray enters.  (An overflow makes the
// axis NaN, which the minima and maxima drop: the box is kept.)  Candidates
// are culled against best_t + 2^-16 |best_t| + slack.  (A negative entry
// distance, of a ray with tmin < 0, is rounded towards zero by up to 2^-20 of
// it, which this margin covers; it orders the children last, not wrongly.)
// Together with the lowest-index tie rule the result equals a brute-force
// scan with the same triangle test.
//
// The traversal is resumable: trav_step_warp() processes one node -- its
// eight child boxes, then the triangles of the leaf children it hit -- and
// moves to the nearest internal child, the others pushed sorted by entry
// distance.  Kernels call it once per loop trip, so a lane whose ray finished
// can start another ray while the rest of its warp is still traversing.
//
// What bounds it: issue slots, the ALU pipe above all (selects, byte
// extraction, min/max), and the wavefronts of scattered loads through L1.
// So a node is three 32-byte loads instead of five of 16, the boxes are
// tested two at a time with packed FP32 operations, the hit children are
// ordered in registers by their distance bits (the nearest never goes
// through the stack), the leaf triangles follow from the hit mask by a bit
// spread, and their test reads the vertices' axes in the ray's order.

struct TraceScene {
  const uint4* nodes;
  const float4* tris;
  uint32_t num_nodes;
  float extent;
#ifdef LISA_BOUNDS
  uint32_t num_tris;
#endif
};

__device__ __forceinline__ TraceScene trace_scene(const SceneDev& sc) {
  TraceScene t;
  t.nodes = sc.nodes;
  t.tris = sc.tris;
  t.num_nodes = sc.num_nodes;
  t.extent = sc.extent;
#ifdef LISA_BOUNDS
  t.num_tris = sc.num_prims;
#endif
  return t;
}

// The emissive triangles' own BVH, with the scene's extent (the ray set-up
// and so every triangle test are those of the scene's BVH).
__device__ __forceinline__ TraceScene trace_scene_emit(const SceneDev& sc) {
  TraceScene t;
  t.nodes = sc.enodes;
  t.tris = sc.etris;
  t.num_nodes = sc.num_enodes;
  t.extent = sc.extent;
#ifdef LISA_BOUNDS
  t.num_tris = sc.num_etris;
#endif
  return t;
}

// 32 bytes of read-only global memory, 32-byte aligned, in one load.
struct Words8 {
  uint32_t v[8];
};
__device__ __forceinline__ Words8 load32(const void* p) {
  Words8 w;
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(w.v[0]), "=r"(w.v[1]), "=r"(w.v[2]), "=r"(w.v[3]), "=r"(w.v[4]), "=r"(w.v[5]), "=r"(w.v[6]), "=r"(w.v[7])
      : "l"(p));
  return w;
}

// Per-warp scratch of the traversal (shared memory): what a lane needs to
// test another lane's triangle, and the exchange of the triangle passes.
struct TriPass {
  float4 ray0[32];             // origin on the shear's axes, tmin
  float4 ray1[32];             // shear Sx, Sy, Sz; byte offsets of the axes in a triangle (kx, ky << 8, kz << 16)
  unsigned long long key[32];  // (t bits << 32 | triangle id) of each lane's best hit
  unsigned long long list[32]; // address of the pass's j-th triangle | lane that asks for it
  int mat[32];
};

struct TravState {
  RayPre r;
  float tmin;
  // (best_t and best_prim start defined: a lane without a ray still joins
  // its warp's triangle pass, which reads them)
  float best_t = 0.0f;
  float cull;  // best_t * (1+2^-16) + slack
  int best_prim = -1;
  int best_mat;  // emitter material of the best hit, -1 if not an emitter (from the leaf triangle)
  uint32_t node;
  int sp;
  bool any;  // stop at the first non-emitter hit found (see trav_pop)
};

// Starts a ray; returns false when there is nothing to traverse (empty
// scene or zero direction), in which case the ray is a miss.  With `any`
// the traversal ends at the first hit it finds: best_prim then says only
// whether the segment (tmin, tmax) is blocked.
__device__ __forceinline__ bool trav_begin(TravState& s, const TraceScene& sc, V3 o, V3 d, float tmin, float tmax,
                                           TriPass& tp, bool any = false) {
  s.any = any;
  s.best_t = tmax;
  s.cull = tmax;
  s.best_prim = -1;
  s.tmin = tmin;
  s.sp = 0;
  s.node = 0;
  if (sc.num_nodes == 0 || is_zero(d)) return false;
  RayShear h;
  ray_prepare(o, d, sc.extent, s.r, h);
  const int lane = threadIdx.x & 31;
  tp.ray0[lane] = make_float4(h.o.x, h.o.y, h.o.z, tmin);
  tp.ray1[lane] = make_float4(h.Sx, h.Sy, h.Sz,
                              __int_as_float(h.kz == 0 ? 0x002010 : (h.kz == 1 ? 0x100020 : 0x201000)));
  return true;
}

// One node of the traversal, in three parts.  trav_node tests the node's
// eight child boxes, finds the nearest internal child it hits, pushes the
// others and returns the triangles of the leaf children it hits.  The
// triangles are then tested by the warp (trav_tris_warp), and trav_pop moves
// to the next node.
struct NodeWork {
  uint32_t tmask;     // the node's leaf triangles still to test, as bits 3 c + q
  uint32_t leaves;    // all of the node's leaf triangles
  uint32_t tri_base;
  uint32_t next;      // the nearest internal child hit
  float next_t;       // its entry distance (rounded down; NaN when there is none)
};

// Distances of two children's planes on one axis: bytes k and k + 1 of w as
// halves (one permute), widened and multiplied on the FMA pipe (C is the
// constant of the slab, see above).
__device__ __forceinline__ float2 slab2(uint32_t w, int k, float s, float C) {
  const uint32_t h = __byte_perm(w, 0x64646464u, 0x4040u | (uint32_t)k | ((uint32_t)(k + 1) << 8));
  const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&h));
  return __ffma2_rn(f, make_float2(s, s), make_float2(C, C));
}

// a - b on the FMA pipe (an integer multiply-add; `one` is 1, which the
// compiler does not know), to spare the ALU pipe.
__device__ __forceinline__ uint32_t sub_fma_pipe(uint32_t a, uint32_t one, uint32_t neg_b) {
  uint32_t d;
  asm("mad.lo.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(one), "r"(neg_b));
  return d;
}

template <bool COUNT>
__device__ __forceinline__ NodeWork trav_node(TravState& s, const TraceScene& sc, uint2* stack, uint32_t& visits,
                                              uint32_t* status) {
  const RayPre& r = s.r;
#ifdef LISA_BOUNDS
  if (s.node >= sc.num_nodes) {  // end the ray
    if (status) atomicOr(status, ST_BOUNDS);
    s.sp = 0;
    return NodeWork{0u, 0u, 0u, 0u, __int_as_float(0x7fffffff)};
  }
#endif
  if (COUNT) ++visits;
  const char* np = (const char*)sc.nodes + (size_t)NODE_BYTES * s.node;
  const Words8 A = load32(np), B = load32(np + 32), C = load32(np + 64);
  const float sx = __uint_as_float(A.v[3]) * r.ix, sy = __uint_as_float(A.v[4]) * r.iy,
              sz = __uint_as_float(A.v[5]) * r.iz;
  const float cx = (__uint_as_float(A.v[0]) - r.ox) * r.ix;
  const float cy = (__uint_as_float(A.v[1]) - r.oy) * r.iy;
  const float cz = (__uint_as_float(A.v[2]) - r.oz) * r.iz;
  const float gx = fmaf(512.0f, fabsf(sx), fabsf(cx));
  const float gy = fmaf(512.0f, fabsf(sy), fabsf(cy));
  const float gz = fmaf(512.0f, fabsf(sz), fabsf(cz));
  constexpr float PAD = 9.5367431640625e-7f;
  const float mx = fmaf(-1024.0f, sx, cx), my = fmaf(-1024.0f, sy, cy), mz = fmaf(-1024.0f, sz, cz);
  const float cnx = fmaf(-PAD, gx, mx), cfx = fmaf(PAD, gx, mx);
  const float cny = fmaf(-PAD, gy, my), cfy = fmaf(PAD, gy, my);
  const float cnz = fmaf(-PAD, gz, mz), cfz = fmaf(PAD, gz, mz);
  const bool negx = r.ix < 0.0f, negy = r.iy < 0.0f, negz = r.iz < 0.0f;
  const uint32_t nx[2] = {negx ? B.v[6] : B.v[0], negx ? B.v[7] : B.v[1]};
  const uint32_t fx[2] = {negx ? B.v[0] : B.v[6], negx ? B.v[1] : B.v[7]};
  const uint32_t ny[2] = {negy ? C.v[0] : B.v[2], negy ? C.v[1] : B.v[3]};
  const uint32_t fy[2] = {negy ? B.v[2] : C.v[0], negy ? B.v[3] : C.v[1]};
  const uint32_t nz[2] = {negz ? C.v[2] : B.v[4], negz ? C.v[3] : B.v[5]};
  const uint32_t fz[2] = {negz ? B.v[4] : C.v[2], negz ? B.v[5] : C.v[3]};
  const uint32_t imask = C.v[4] >> 24;
  // hit mask, and a sort key per internal child that is hit: its entry
  // distance (positive, so the bits order as the float) with the slot in the
  // low three bits, which rounds the distance down
  uint32_t hit = 0, key[8];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int w = p >> 1, k = 2 * (p & 1);
    const float2 a0 = slab2(nx[w], k, sx, cnx), a1 = slab2(ny[w], k, sy, cny), a2 = slab2(nz[w], k, sz, cnz);
    const float2 f0 = slab2(fx[w], k, sx, cfx), f1 = slab2(fy[w], k, sy, cfy), f2 = slab2(fz[w], k, sz, cfz);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int c = 2 * p + j;
      const float tn = fmaxf(fmaxf(fmaxf(j ? a0.y : a0.x, j ? a1.y : a1.x), j ? a2.y : a2.x), s.tmin);
      const float tf = fminf(fminf(fminf(j ? f0.y : f0.x, j ? f1.y : f1.x), j ? f2.y : f2.x), s.cull);
      const bool h = tn <= tf;
      if (h) hit |= 1u << c;
      key[c] = (h && ((imask >> c) & 1u)) ? ((__float_as_uint(tn) & ~7u) | (uint32_t)c) : 0xffffffffu;
    }
  }
  uint32_t k = min(min(min(key[0], key[1]), min(key[2], key[3])), min(min(key[4], key[5]), min(key[6], key[7])));
  const uint32_t child_base = A.v[6];
  NodeWork w;
  w.next = child_base + (k & 7u);
  w.next_t = __uint_as_float(k & ~7u);
  const int n = __popc(imask & hit);
  if (n > 1) {
    // the others, farthest first: the next larger key is the smallest of
    // key - (k + 1) in unsigned arithmetic
    const int sp0 = s.sp;
    uint32_t one = 1;
    asm volatile("" : "+r"(one));
    int at = sp0 + n - 2;
    s.sp = at + 1;
    if (s.sp > TRAV_STACK) {
      if (status) atomicOr(status, ST_STACK_OVERFLOW);
      s.sp = TRAV_STACK;
    }
#pragma unroll 1
    for (; at >= sp0; --at) {
      const uint32_t o = ~k;  // -(k + 1)
      uint32_t m[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) m[c] = sub_fma_pipe(key[c], one, o);
      k = min(min(min(m[0], m[1]), min(m[2], m[3])), min(min(m[4], m[5]), min(m[6], m[7]))) - o;
      if (at < TRAV_STACK) stack[at] = make_uint2(child_base + (k & 7u), k & ~7u);
    }
  }
  // bit c of the hit mask to bits 3 c .. 3 c + 2
  uint32_t m = (hit | (hit << 8)) & 0x00f00fu;
  m = (m | (m << 4)) & 0x0c30c3u;
  m = (m | (m << 2)) & 0x249249u;
  w.leaves = C.v[4] & 0xffffffu;
  w.tmask = (m * 7u) & w.leaves;
  w.tri_base = A.v[7];
#ifdef LISA_BOUNDS
  if (w.tmask && w.tri_base + (uint32_t)__popc(w.leaves) > sc.num_tris) {
    if (status) atomicOr(status, ST_BOUNDS);
    w.tmask = 0;
  }
#endif
  return w;
}

// Address of the leaf triangle at the lowest bit of w.tmask.
__device__ __forceinline__ const char* first_tri(const TraceScene& sc, const NodeWork& w) {
  const uint32_t low = w.tmask & (0u - w.tmask);
  return (const char*)sc.tris + (size_t)TRI_BYTES * (w.tri_base + (uint32_t)__popc(w.leaves & (low - 1u)));
}

// Tests the triangle at p with the ray (r0, r1) of TriPass.
__device__ __forceinline__ float test_tri(const char* p, float4 r0, float4 r1, int& prim) {
  const uint32_t at = __float_as_uint(r1.w);
  const float4 x = __ldg((const float4*)(p + (at & 0xffu))), y = __ldg((const float4*)(p + ((at >> 8) & 0xffu))),
               z = __ldg((const float4*)(p + (at >> 16)));
  prim = __float_as_int(x.w);
  const RayShear h{r1.x, r1.y, r1.z, 0, ld3(r0)};
  return intersect_tri(h, v3(x.x, y.x, z.x), v3(x.y, y.y, z.y), v3(x.z, y.z, z.z), r0.w);
}

// A distance as an integer in the same order, and back.  The path tracer's are
// positive, so their bits will do; given rays (SIGNED) may start behind their
// origin (tmin < 0), where -0 and +0 are one distance.
template <bool SIGNED>
__device__ __forceinline__ uint32_t dist_key(float t) {
  if (!SIGNED) return __float_as_uint(t);
  const int i = __float_as_int(fadd(t, 0.0f));
  return (uint32_t)(i ^ ((i >> 31) & 0x7fffffff)) ^ 0x80000000u;
}
template <bool SIGNED>
__device__ __forceinline__ float key_dist(uint32_t k) {
  if (!SIGNED) return __uint_as_float(k);
  const int i = (int)(k ^ 0x80000000u);
  return __int_as_float(i ^ ((i >> 31) & 0x7fffffff));
}

// Tests the triangles of all lanes of the warp, up to 32 at a time.  Either
// each lane its own, one per pass (when that takes no more passes), or the
// lanes' triangles laid end to end (a prefix sum of their counts): each lane
// writes the addresses of its own into the pass's list, and lane j takes the
// j-th with the asking lane's ray.  A lane's best hit is the minimum of the
// 64-bit keys (t, triangle id), which is the brute-force tie rule.  Called by all 32 lanes; lanes
// without a ray pass w.tmask = 0.  MAT: the hit's emitter material is wanted
// too.
template <bool COUNT, bool MAT, bool SIGNED>
__device__ __forceinline__ void trav_tris_warp(TravState& s, const TraceScene& sc, NodeWork w, uint32_t& tests,
                                               TriPass& tp) {
  const int lane = threadIdx.x & 31;
  const uint32_t cnt = __popc(w.tmask);
  const uint32_t most = __reduce_max_sync(0xffffffffu, cnt);
  if (most == 0) return;
  uint32_t incl = cnt, total = 0;
  if (most > 1) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    total = __shfl_sync(0xffffffffu, incl, 31);
  }
  const bool own = most <= 1 || most <= ((total + 31u) >> 5);
  uint32_t pos = incl - cnt;
  const unsigned long long key0 =
      ((unsigned long long)dist_key<SIGNED>(s.best_t) << 32) | (uint32_t)s.best_prim;
  tp.key[lane] = key0;
  const uint32_t passes = own ? most : (total + 31u) >> 5;
#pragma unroll 1
  for (uint32_t k = 0; k < passes; ++k) {
    unsigned long long e = 0;
    bool test;
    if (own) {
      test = w.tmask != 0u;
      e = (unsigned long long)first_tri(sc, w) | (uint32_t)lane;
      w.tmask &= w.tmask - 1u;
    } else {
#pragma unroll 1
      while (w.tmask && pos < 32u * k + 32u) {
        tp.list[pos - 32u * k] = (unsigned long long)first_tri(sc, w) | (uint32_t)lane;
        w.tmask &= w.tmask - 1u;
        ++pos;
      }
      __syncwarp();
      test = 32u * k + (uint32_t)lane < total;
      if (test) e = tp.list[lane];
    }
    bool better = false;
    unsigned long long key = 0;
    const int o = (int)(e & 31u);
    if (test) {
      int prim;
      const float t = test_tri((const char*)(e & ~31ull), tp.ray0[o], tp.ray1[o], prim);
      if (COUNT) ++tests;
      const unsigned long long okey = *(volatile unsigned long long*)&tp.key[o];
      const float bt = key_dist<SIGNED>((uint32_t)(okey >> 32));
      if (t < bt || (t == bt && prim < (int)(uint32_t)okey)) {
        better = true;
        key = ((unsigned long long)dist_key<SIGNED>(t) << 32) | (uint32_t)prim;
        atomicMin(&tp.key[o], key);
      }
    }
    __syncwarp();
    if (MAT) {
      if (better && tp.key[o] == key) tp.mat[o] = __ldg((const int*)((e & ~31ull) + 48));
      __syncwarp();
    }
  }
  const unsigned long long best = tp.key[lane];
  if (best != key0) {
    s.best_t = key_dist<SIGNED>((uint32_t)(best >> 32));
    s.best_prim = (int)(uint32_t)best;
    if (MAT) s.best_mat = tp.mat[lane];
    s.cull = fmaf(SIGNED ? fabsf(s.best_t) : s.best_t, 1.52587890625e-5f, s.best_t) + s.r.slack;
  }
  __syncwarp();
}

// Whether the ray may meet the box [lo, hi] inside (tmin, tmax): slab
// distances from the node-culling reciprocals, each widened by 2^-20 of
// their magnitude, which covers their roundings (conservative: a ray that
// meets the box is never rejected).
__device__ __forceinline__ bool box_may_hit(const RayPre& r, const float* lo, const float* hi, float tmin,
                                            float tmax) {
  const float ax = (lo[0] - r.ox) * r.ix, bx = (hi[0] - r.ox) * r.ix;
  const float ay = (lo[1] - r.oy) * r.iy, by = (hi[1] - r.oy) * r.iy;
  const float az = (lo[2] - r.oz) * r.iz, bz = (hi[2] - r.oz) * r.iz;
  const float gx = 9.5367431640625e-7f * (fabsf(ax) + fabsf(bx));
  const float gy = 9.5367431640625e-7f * (fabsf(ay) + fabsf(by));
  const float gz = 9.5367431640625e-7f * (fabsf(az) + fabsf(bz));
  const float tn = fmaxf(fmaxf(fminf(ax, bx) - gx, fminf(ay, by) - gy), fmaxf(fminf(az, bz) - gz, tmin));
  const float tf = fminf(fminf(fmaxf(ax, bx) + gx, fmaxf(ay, by) + gy), fminf(fmaxf(az, bz) + gz, tmax));
  return tn <= tf;
}

// Whether a ray from o along d may meet the scene's emissive triangles
// inside (RAY_TMIN, RAY_TMAX): box_may_hit against their padded bounds with
// the node-culling reciprocals (__fdividef, within 2 ulp; a huge finite
// value for a vanishing component), without the rest of a ray set-up.
// Conservative: false only when no emitter can be hit.
__device__ __forceinline__ bool emit_may_hit(const SceneDev& sc, V3 o, V3 d) {
  if (!sc.has_emit_box) return false;
  RayPre r;
  r.ox = o.x;
  r.oy = o.y;
  r.oz = o.z;
  r.ix = fabsf(d.x) > 1e-30f ? __fdividef(1.0f, d.x) : copysignf(1e30f, d.x);
  r.iy = fabsf(d.y) > 1e-30f ? __fdividef(1.0f, d.y) : copysignf(1e30f, d.y);
  r.iz = fabsf(d.z) > 1e-30f ? __fdividef(1.0f, d.z) : copysignf(1e30f, d.z);
  return box_may_hit(r, sc.emit_lo, sc.emit_hi, RAY_TMIN, RAY_TMAX);
}

// Bounds of the scene's emissive triangles relative to a vertex: centre c,
// half extent h, grown by 2^-19 of |c| + |h|.
struct EmitBounds {
  V3 c, h;
};
__device__ __forceinline__ EmitBounds emit_bounds(const SceneDev& sc, V3 o) {
  const float lx = sc.emit_lo[0] - o.x, ly = sc.emit_lo[1] - o.y, lz = sc.emit_lo[2] - o.z;
  const float ux = sc.emit_hi[0] - o.x, uy = sc.emit_hi[1] - o.y, uz = sc.emit_hi[2] - o.z;
  EmitBounds e;
  e.c = v3(0.5f * (lx + ux), 0.5f * (ly + uy), 0.5f * (lz + uz));
  const float hx = 0.5f * (ux - lx), hy = 0.5f * (uy - ly), hz = 0.5f * (uz - lz);
  const float pad = 1.9073486328125e-6f * (((fabsf(e.c.x) + fabsf(e.c.y)) + fabsf(e.c.z)) + ((hx + hy) + hz));
  e.h = v3(hx + pad, hy + pad, hz + pad);
  return e;
}

// Whether the next try of a vertex's emitter search may reach an emitter
// (`seed` is the stream's state before it, advanced past it).  The try is the
// hemisphere draw q = (x, y, z) of shoot_ray_hemisphere, not normalised: the
// exact direction is a positive multiple of q, flipped by the sign of
// dot(N, q), each component with one more rounding.  A try is left out when
// its line misses the padded bounds of the emissive triangles (one of the
// three cross-product axes separates them; the axes do not depend on the
// flip) or when all of the bounds lie behind the ray; where dot(N, q) is too
// near zero for its sign to be certain, only the line is tested.  The
// bounds' padding is four times the roundings of c, h, the products and the
// direction.  Every comparison rejects on a definite answer, so a NaN leaves
// the try in.
//
// Divisions would cost more than the rest of the test (three reciprocals and
// their guards a try); the separating axes need none: about 40 instructions.
__device__ __forceinline__ bool emit_candidate(const EmitBounds& e, V3 N, uint32_t& seed) {
  const float x = fmaf((float)lcg(seed), 1.1920928955078125e-7f, -1.0f);
  const float y = fmaf((float)lcg(seed), 1.1920928955078125e-7f, -1.0f);
  const float z = fmaf((float)lcg(seed), 1.1920928955078125e-7f, -1.0f);
  const float ax = fabsf(x), ay = fabsf(y), az = fabsf(z);
  const bool off = fabsf(fmaf(y, e.c.z, -(z * e.c.y))) > fmaf(e.h.y, az, e.h.z * ay) ||
                   fabsf(fmaf(z, e.c.x, -(x * e.c.z))) > fmaf(e.h.z, ax, e.h.x * az) ||
                   fabsf(fmaf(x, e.c.y, -(y * e.c.x))) > fmaf(e.h.x, ay, e.h.y * ax);
  const float s = fmaf(N.x, x, fmaf(N.y, y, N.z * z));
  const float f = fmaf(e.c.x, x, fmaf(e.c.y, y, e.c.z * z));
  const bool behind = fabsf(s) > 1e-5f * ((ax + ay) + az) &&
                      copysignf(1.0f, s) * f < -fmaf(e.h.x, ax, fmaf(e.h.y, ay, e.h.z * az));
  return !off && !behind;
}

// All tries of a vertex, as a bit mask (bit j = try j; `seed` is the state
// before try 0).  The last try always stays: the search ends there.
__device__ __forceinline__ uint32_t emit_candidates(const SceneDev& sc, V3 o, V3 N, uint32_t seed) {
  uint32_t mask = 1u << (NEE_TRIES - 1);
  if (!sc.has_emit_box) return mask;
  const EmitBounds e = emit_bounds(sc, o);
#pragma unroll 2
  for (int j = 0; j < NEE_TRIES - 1; ++j)
    if (emit_candidate(e, N, seed)) mask |= 1u << j;
  return mask;
}

// Whether the ray (o, d) may meet the box [lo, hi] inside (tmin, tmax),
// every step a single IEEE rounding so the host oracle takes the same
// decision bit for bit: slab distances with the correctly rounded 1/d (a
// huge finite value of d's sign for a zero component), each widened by
// 2^-20 of their magnitude.  Used where a ray is traced only for the
// emission it may reach: one that misses the emissive triangles' padded
// bounds would gather nothing, so it is not traced at all.
__device__ __forceinline__ bool box_may_hit_exact(V3 o, V3 d, const float* lo, const float* hi, float tmin,
                                                  float tmax) {
  const float dd[3] = {d.x, d.y, d.z}, oo[3] = {o.x, o.y, o.z};
  float tn = tmin, tf = tmax;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const float inv = dd[k] != 0.0f ? __frcp_rn(dd[k]) : copysignf(1e30f, dd[k]);
    const float a = fmul(fsub(lo[k], oo[k]), inv), b = fmul(fsub(hi[k], oo[k]), inv);
    const float g = fmul(9.5367431640625e-7f, fadd(fabsf(a), fabsf(b)));
    tn = fmaxf(tn, fsub(fminf(a, b), g));
    tf = fminf(tf, fadd(fmaxf(a, b), g));
  }
  return tn <= tf;
}

// Moves to the nearest child not culled: the node's own, else the stack's
// top.  Returns true when the traversal is finished.
__device__ __forceinline__ bool trav_pop(TravState& s, uint2* stack, const NodeWork& w) {
  // an any-hit traversal ends at its first hit that is not an emitter's (a
  // ray that cannot reach an emitter only finds such hits; the emitter
  // search's scene pass starts from an emitter hit and looks for a nearer
  // triangle, which cannot be an emitter's)
  if (s.any && s.best_prim >= 0 && s.best_mat < 0) return true;
  if (w.next_t <= s.cull) {
    s.node = w.next;
    return false;
  }
#pragma unroll 1
  while (s.sp > 0) {
    const uint2 e = stack[--s.sp];
    if (__uint_as_float(e.y) <= s.cull) {
      s.node = e.x;
      return false;
    }
  }
  return true;
}

// Processes one node for each active lane of a warp (all 32 lanes call it).
// Returns true for an active lane whose traversal is finished (s.best_prim /
// s.best_t hold the result, best_prim -1 on a miss); inactive lanes get
// false.
template <bool COUNT, bool MAT, bool SIGNED = false>
__device__ __forceinline__ bool trav_step_warp(bool active, TravState& s, const TraceScene& sc, uint2* stack,
                                               uint32_t& visits, uint32_t& tests, uint32_t* status, TriPass& tp) {
  NodeWork w{0u, 0u, 0u, 0u, 0.0f};
  if (active) w = trav_node<COUNT>(s, sc, stack, visits, status);
  trav_tris_warp<COUNT, MAT, SIGNED>(s, sc, w, tests, tp);
  return active && trav_pop(s, stack, w);
}

// Brute-force scan in original triangle order with the same test and tie
// rule (lowest index wins on equal t).
__device__ __forceinline__ void brute_hit(const SceneDev& sc, V3 o, V3 d, float tmin, float tmax, int& out_prim,
                                          float& out_t) {
  out_prim = -1;
  out_t = __int_as_float(0x7f800000);
  if (is_zero(d)) return;
  RayPre r;
  RayShear h;
  ray_prepare(o, d, sc.extent, r, h);
  float best_t = tmax;
  int best = -1;
  for (uint32_t p = 0; p < sc.num_prims; ++p) {
    const float4* pr = sc.prims + 5ull * p;
    const float4 a = __ldg(pr + 0), b = __ldg(pr + 1), c = __ldg(pr + 2);
    const float t = intersect_tri(h, on_shear_axes(ld3(a), h.kz), on_shear_axes(ld3(b), h.kz),
                                  on_shear_axes(ld3(c), h.kz), tmin);
    if (t < best_t) {
      best_t = t;
      best = (int)p;
    }
  }
  if (best >= 0) {
    out_prim = best;
    out_t = fadd(best_t, 0.0f);  // (+0 for -0, as dist_key has it)
  }
}

}  // namespace lisa
