// Wavefront path tracer: the reference estimator (src/LiSA/src/shader.cu)
// re-organised as stages over SoA queues instead of one OptiX thread per
// pixel.
//
//   raygen      one path per (scene, pixel, sample) slot          shader.cu:126-155
//   trace       closest hit of every queued ray (persistent warps) shader.cu:77-98
//   nee         shades 32 hits at a time, by material class:      shader.cu:211-255
//                 miss / emitter -> path ends (emitter adds Le*att)
//                 dielectric     -> Fresnel reflect / refract, next ray
//                 opaque         -> up to 30 hemisphere rays until one
//                   returns the (stale) emitter, att *= albedo, then
//                   the bounce                                      shader.cu:196-209,248-253
//   accumulate  per pixel, Kahan FP32 sum + FP64 sum of squares     shader.cu:156-166
//
// Small plain waves run whole paths in one kernel instead (k_paths).
//
// The persistent kernels take work with warp-aggregated atomics (one atomic
// per warp per refill); queue appends are warp-aggregated the same way.
// Counters that a stage consumes are reset by a stage that does not run
// concurrently with it (see the comments at each reset).
#include <algorithm>
#include <cstring>
#include <vector>

#include "guide.cuh"
#include "guide_mix.cuh"
#include "lisa_device.cuh"
#include "lisa_internal.h"
#include "refill.h"
#include "wavefront.cuh"

#ifndef LISA_BSDF_HEADER
#define LISA_BSDF_HEADER "bsdfs/lambertian.cuh"
#endif
#include LISA_BSDF_HEADER
#include "guide_infer.cuh"
#include "physical.cuh"

namespace lisa {

constexpr uint32_t FULL = 0xffffffffu;

// Residency: blocks of 128 threads per SM that the compiler must fit.
// Measured: the closest-hit kernel at 8 (64 registers, no spills) is 4 %
// faster than at 7; the emitter-search kernels at 6 (80 registers) are best of
// 5..8 -- more blocks leave less L1 for the BVH beside their shared memory
// (soup frame: 105, 103, 109, 110 ms).
#ifndef LISA_TRACE_MIN_BLOCKS
#define LISA_TRACE_MIN_BLOCKS 8
#endif
#ifndef LISA_NEE_MIN_BLOCKS
#define LISA_NEE_MIN_BLOCKS 6
#endif
#ifndef LISA_NEE_PB_MIN_BLOCKS
#define LISA_NEE_PB_MIN_BLOCKS 6
#endif
#ifndef LISA_PATHS_MIN_BLOCKS
#define LISA_PATHS_MIN_BLOCKS 5  // whole paths: 96 registers, best of 4..6
#endif

__device__ __forceinline__ uint32_t lanemask_lt() {
  uint32_t m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

// Warp-aggregated reservation of `want ? 1 : 0` entries in *counter.  All 32
// lanes must call it.  Returns the lane's index (undefined if !want).
__device__ __forceinline__ uint32_t warp_reserve(uint32_t* counter, bool want) {
  const uint32_t mask = __ballot_sync(FULL, want);
  if (!mask) return 0;
  const int leader = __ffs(mask) - 1;
  const int lane = threadIdx.x & 31;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(mask));
  base = __shfl_sync(FULL, base, leader);
  return base + __popc(mask & lanemask_lt());
}

__device__ __forceinline__ void warp_add64(unsigned long long* c, uint32_t v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(c, (unsigned long long)v);
}

// Whether queue slot i, reserved by an append, lies inside the queue: always,
// by construction (one entry per path and depth); checked in bounds-checked
// builds, where a bad slot sets ST_QUEUE_OVERFLOW and the write is skipped.
__device__ __forceinline__ bool queue_fits(const WaveBufs& b, uint32_t i) {
#ifdef LISA_BOUNDS
  if (i < b.capacity) return true;
  atomicOr(&b.ctrl->status, ST_QUEUE_OVERFLOW);
  return false;
#else
  (void)b;
  (void)i;
  return true;
#endif
}

// The ray leaving a path's last vertex (physically based estimator) only
// gathers emission: it is traced only if it may meet the scene's emitters.
__device__ __forceinline__ bool final_ray_wanted(const SceneDev& sc, V3 p, V3 d) {
  return sc.has_emit_box && box_may_hit_exact(p, d, sc.emit_lo, sc.emit_hi, RAY_TMIN, RAY_TMAX);
}

__device__ __forceinline__ void warp_add32(uint32_t* c, uint32_t v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(c, v);
}

__device__ __forceinline__ V3 barycentric_normal(V3 p, const float4* pr) {
  // src/LiSA/src/maths.cu:33-56 (barycentrics re-derived from the hit point)
  const float4 r0 = __ldg(pr + 0), r1 = __ldg(pr + 1), r2 = __ldg(pr + 2), r3 = __ldg(pr + 3), r4 = __ldg(pr + 4);
  const V3 v1 = ld3(r0), v2 = ld3(r1), v3_ = ld3(r2);
  const V3 n1 = v3(r0.w, r1.w, r2.w);
  const V3 n2 = v3(r3.x, r3.y, r3.z);
  const V3 n3 = v3(r3.w, r4.x, r4.y);
  const V3 e1 = v2 - v1, e2 = v3_ - v1, i = p - v1;
  const float d00 = dot(e1, e1), d01 = dot(e1, e2), d11 = dot(e2, e2);
  const float d20 = dot(i, e1), d21 = dot(i, e2);
  const float denom = fsub(fmul(d00, d11), fmul(d01, d01));
  const float w = fdiv(fsub(fmul(d00, d21), fmul(d01, d20)), denom);
  const float v = fdiv(fsub(fmul(d11, d20), fmul(d01, d21)), denom);
  const float u = fsub(fsub(1.0f, v), w);
  return normalize((u * n1 + v * n2) + w * n3);
}

__device__ __forceinline__ int prim_material(const SceneDev& sc, int prim) {
  return __float_as_int(__ldg(sc.prims + 5ull * prim + 4).z);
}

__device__ __forceinline__ int find_group(const WaveDesc& w, uint32_t key, bool by_acc) {
  int lo = 0, hi = (int)w.num_groups - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    const uint32_t b = by_acc ? w.groups[mid].acc0 : w.groups[mid].slot0;
    if (b <= key) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// ---------------------------------------------------------------------------
// raygen (shader.cu:126-152)

// Scene, pixel, stream state and camera ray of the wave's path `slot`
// (shader.cu:126-152).  With one stream per pixel, a path that is not of its
// group's first plane goes on with the state in `seed`, its predecessor's.
__device__ __forceinline__ void camera_ray(const WaveBufs& b, const WaveDesc& w, uint32_t slot, uint32_t& scene,
                                           uint32_t& pix, uint32_t& seed, V3& org, V3& dir) {
  const WaveGroup& g = w.groups[find_group(w, slot, false)];
  const SceneDev& sc = b.scenes[g.scene];
  const uint32_t off = slot - g.slot0;
  const uint32_t m = off / g.npix;
  scene = g.scene;
  pix = g.pix0 + (off - m * g.npix);
  const uint32_t sample = g.sample0 + m;
  const uint32_t x = pix % sc.width, y = pix / sc.width;
  if (w.rng_mode == LISA_RNG_PER_PIXEL) {
    if (m == 0) seed = sc.pix_rng[pix];
  } else {
    seed = tea<16>(pix, tea<4>(sample, w.seed));
  }
  const float jx = rng11(seed);
  const float jy = rng11(seed);
  const float dx = fsub(fdiv(fadd(fmul(2.0f, (float)x), jx), (float)sc.width), 1.0f);
  const float dy = fsub(fdiv(fadd(fmul(2.0f, (float)y), jy), (float)sc.height), 1.0f);
  const V3 U = v3(sc.U[0], sc.U[1], sc.U[2]), V = v3(sc.V[0], sc.V[1], sc.V[2]), W = v3(sc.W[0], sc.W[1], sc.W[2]);
  dir = normalize((dx * U + dy * V) + W);
  org = v3(sc.eye[0], sc.eye[1], sc.eye[2]);
  if (sc.lens_radius > 0.0f) {
    // Thin lens (not in the reference, whose camera is a pinhole): the
    // pinhole ray meets the focal plane at distance focal_distance along
    // the view axis; the origin moves to a uniform point of the lens disk,
    // drawn by rejection from the square (trig-free, so the oracle draws
    // the same point bit for bit).
    const V3 wu = v3(sc.unitW[0], sc.unitW[1], sc.unitW[2]);
    const float tf = fdiv(sc.focal_distance, dot(dir, wu));
    const V3 focus = org + tf * dir;
    float lu, lv;
    do {
      lu = rng11(seed);
      lv = rng11(seed);
    } while (fadd(fmul(lu, lu), fmul(lv, lv)) > 1.0f);
    org = org + fmul(sc.lens_radius, lu) * v3(sc.unitU[0], sc.unitU[1], sc.unitU[2]) +
          fmul(sc.lens_radius, lv) * v3(sc.unitV[0], sc.unitV[1], sc.unitV[2]);
    dir = normalize(focus - org);
  }
}

// One path per slot; also resets the counters of depth 0.
__global__ void k_raygen(WaveBufs b, const WaveDesc* __restrict__ wave) {
  const WaveDesc& w = *wave;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    // nothing else runs during raygen
    b.ctrl->qcount[0] = w.paths;
    b.ctrl->qcount[1] = 0;
    b.ctrl->nee_count = 0;
    b.ctrl->head[HEAD_TRACE] = 0;
    b.ctrl->head[HEAD_NEE] = 0;
    b.ctrl->guided_count = 0;
    b.ctrl->rec_count = 0;
    b.ctrl->train_count = 0;
    b.ctrl->rays_primary += w.paths;
  }
  for (uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x; slot < w.paths; slot += gridDim.x * blockDim.x) {
    uint32_t scene, pix, seed;
    V3 org, dir;
    camera_ray(b, w, slot, scene, pix, seed, org, dir);
    b.ro[0][slot] = make_float4(org.x, org.y, org.z, __uint_as_float(slot));
    b.rd[0][slot] = make_float4(dir.x, dir.y, dir.z, __uint_as_float(scene));
    // w: the stale emitter flag (compat, -1 = none) or the pdf of the last
    // diffuse bounce (physically based, 0 = camera or specular)
    b.ps_att[slot] = make_float4(1.0f, 1.0f, 1.0f, b.physical ? 0.0f : __int_as_float(-1));
    b.ps_col[slot] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float((scene << 24) | pix));
    b.ps_rng[slot] = seed;
  }
}

// ---------------------------------------------------------------------------
// closest hit of the queued rays: each lane traverses one node per loop trip
// and takes the next ray as soon as its own is done (warp-aggregated fetch).

template <bool COUNT>
__global__ void __launch_bounds__(128, LISA_TRACE_MIN_BLOCKS) k_trace(WaveBufs b, int depth) {
  const int q = depth & 1;
  const uint32_t count = *(volatile uint32_t*)&b.ctrl->qcount[q];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    // the emitter search of this depth has not started; the previous depth's
    // consumers of these counters have finished
    b.ctrl->qcount[q ^ 1] = 0;
    b.ctrl->nee_count = 0;
    b.ctrl->head[HEAD_NEE] = 0;
    if (depth > 0) b.ctrl->rays_bounce += count;
  }
  const int lane = threadIdx.x & 31;
  const uint32_t lt = lanemask_lt();
  uint2 stack[TRAV_STACK];
  TravState s;
  TraceScene ts;
  uint32_t ray = 0, visits = 0, tests = 0;
  bool active = false, exhausted = false;
  __shared__ TriPass tri_pass[4];
  TriPass& tp = tri_pass[threadIdx.x >> 5];
  while (true) {
    // take new rays only once enough lanes are idle (see k_nee)
    if (__popc(__ballot_sync(FULL, active)) <= (int)b.refill_busy_max) {
      const bool need = !active && !exhausted;
      const uint32_t nmask = __ballot_sync(FULL, need);
      if (nmask) {
        const int leader = __ffs(nmask) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(&b.ctrl->head[HEAD_TRACE], (uint32_t)__popc(nmask));
        base = __shfl_sync(FULL, base, leader);
        if (need) {
          ray = base + __popc(nmask & lt);
          if (ray < count) {
            const float4 o = b.ro[q][ray], d = b.rd[q][ray];
            ts = trace_scene(b.scenes[__float_as_uint(d.w)]);
            active = trav_begin(s, ts, ld3(o), ld3(d), RAY_TMIN, RAY_TMAX, tp);
            if (!active) b.hit[ray] = make_int2(-1, 0x7f800000);
          } else {
            exhausted = true;
          }
        }
      }
      if (!__any_sync(FULL, active || !exhausted)) break;
    }
    if (trav_step_warp<COUNT, false>(active, s, ts, stack, visits, tests, &b.ctrl->status, tp)) {
      b.hit[ray] = make_int2(s.best_prim, s.best_prim >= 0 ? __float_as_int(s.best_t) : 0x7f800000);
      active = false;
    }
  }
  if (COUNT) {
    warp_add64(&b.ctrl->node_visits[0], visits);
    warp_add64(&b.ctrl->tri_tests[0], tests);
  }
}

// ---------------------------------------------------------------------------
// shade: emitter / miss / dielectric / opaque (shader.cu:189-194,211-255)

// What an emitter hit adds to a path: Le * throughput (shader.cu:216-218),
// weighted in the physically based estimator when a diffuse bounce of density
// att.w reached it (power heuristic against the emitter sampler's density
// for this direction).
template <bool PHYS>
__device__ __forceinline__ V3 emitter_hit(const SceneDev& sc, const DevMaterial& m, int prim, float t, V3 d,
                                          float4 att) {
  V3 le = v3(m.emission[0], m.emission[1], m.emission[2]) * ld3(att);
  if (PHYS && att.w > 0.0f) {
    const float prev = att.w;
    const float4* pr = sc.prims + 5ull * prim;
    const V3 v0 = ld3(pr[0]);
    const V3 cr = cross3(ld3(pr[1]) - v0, ld3(pr[2]) - v0);
    const V3 n = cr * fdiv(1.0f, fsqrt(dot(cr, cr)));
    const float cos_y = fabsf(dot(n, d));
    float w = 0.0f;
    if (cos_y > 0.0f) {
      const float pl = fdiv(fmul(m.light_pdf, fmul(t, t)), cos_y);
      w = fdiv(fmul(prev, prev), fadd(fmul(prev, prev), fmul(pl, pl)));
    }
    le = le * w;
  }
  return le;
}

// Continuation at a dielectric hit with shading normal N (shader.cu:226-247):
// the direction (zero on total internal reflection in the reference
// estimator, a miss), the throughput a and the stream updated.
template <bool PHYS>
__device__ __forceinline__ V3 dielectric_bounce(const DevMaterial& m, V3 d, V3 N, V3& a, uint32_t& seed) {
  float cosI = dot(d, N);
  float eta;
  V3 nrm;
  if (cosI < 0.0f) {
    cosI = -cosI;
    eta = fdiv(1.0f, m.ior);
    nrm = N;
  } else {
    a = a * v3(m.albedo[0], m.albedo[1], m.albedo[2]);
    eta = m.ior;
    nrm = -N;
  }
  if (eta == 1.0f) return d;
  if (PHYS) {
    // total internal reflection reflects; Schlick's term takes the cosine on
    // the less dense side (the transmitted one on exit)
    const float cost2 = fsub(1.0f, fmul(fmul(eta, eta), fsub(1.0f, fmul(cosI, cosI))));
    if (cost2 <= 0.0f) return reflect(d, nrm);
    if (rnd(seed) <= bsdf::BTDF(eta > 1.0f ? fsqrt(cost2) : cosI, eta)) return reflect(d, nrm);
    return bsdf::refract(cosI, d, nrm, eta);
  }
  if (rnd(seed) <= bsdf::BTDF(cosI, eta)) return reflect(d, nrm);
  return bsdf::refract(cosI, d, nrm, eta);
}

// An opaque hit: a vertex for the emitter search.  The path's throughput is
// still the one before the vertex (its albedo is applied when the vertex is
// left).
struct Vertex {
  V3 p, N;
  uint32_t slot, scene;
  int mat;
  float4 att;
};

// Shades entry i of the depth's ray queue (valid: there is one): misses and
// emitters end their path, a dielectric's ray goes to the next queue, an
// opaque hit is returned as a vertex.  Called by all 32 lanes, on consecutive
// entries, so that the queue reads coalesce.
template <bool PHYS>
__device__ __forceinline__ bool shade_ray(const WaveBufs& b, int depth, uint32_t i, bool valid, Vertex& v) {
  const int q = depth & 1;
  bool want_ray = false, vertex = false;
  V3 nd = v3(0.0f);
  if (valid) {
    const int2 h = b.hit[i];
    const float4 o4 = b.ro[q][i];
    const float4 d4 = b.rd[q][i];
    v.slot = __float_as_uint(o4.w);
    v.scene = __float_as_uint(d4.w);
    if (h.x >= 0) {  // a miss adds the background, 0 (optix_wrapper.cc:354-356), and ends the path
      const SceneDev& sc = b.scenes[v.scene];
      v.mat = prim_material(sc, h.x);
      v.att = b.ps_att[v.slot];
      const DevMaterial& m = sc.mats[v.mat];
      const float t = __int_as_float(h.y);
      if (m.cls == MAT_EMIT) {
        const float4 col = b.ps_col[v.slot];
        const V3 c = ld3(col) + emitter_hit<PHYS>(sc, m, h.x, t, ld3(d4), v.att);
        b.ps_col[v.slot] = make_float4(c.x, c.y, c.z, col.w);
      } else if (!PHYS || depth < (int)sc.num_bounces) {
        // (physically based: the ray leaving the last vertex only gathers
        // the emission it reaches, so any other hit ends the path)
        const V3 d = ld3(d4);
        v.p = ld3(o4) + t * d;
        v.N = barycentric_normal(v.p, sc.prims + 5ull * h.x);
        if (m.cls == MAT_DIELECTRIC) {
          // the reference estimator traces num_bounces rays; the physically
          // based one also the ray leaving its last vertex
          V3 a = ld3(v.att);
          uint32_t seed = b.ps_rng[v.slot];
          nd = dielectric_bounce<PHYS>(m, d, v.N, a, seed);
          b.ps_rng[v.slot] = seed;
          b.ps_att[v.slot] = make_float4(a.x, a.y, a.z, PHYS ? 0.0f : v.att.w);
          want_ray = (PHYS || depth + 1 < (int)sc.num_bounces) && !is_zero(nd);
          if (PHYS && want_ray && depth + 1 == (int)sc.num_bounces) want_ray = final_ray_wanted(sc, v.p, nd);
        } else {
          vertex = true;
        }
      }
    }
  }
  const uint32_t ri = warp_reserve(&b.ctrl->qcount[q ^ 1], want_ray);
  if (want_ray && queue_fits(b, ri)) {
    b.ro[q ^ 1][ri] = make_float4(v.p.x, v.p.y, v.p.z, __uint_as_float(v.slot));
    b.rd[q ^ 1][ri] = make_float4(nd.x, nd.y, nd.z, __uint_as_float(v.scene));
  }
  return vertex;
}

// Throughput after the vertex's material (shader.cu:248).
__device__ __forceinline__ V3 vertex_throughput(float4 att, const DevMaterial& m) {
  return ld3(att) * v3(m.albedo[0], m.albedo[1], m.albedo[2]);
}

// Guided mode: the vertex's entry of the queue that the guide's inference
// reads.  Called by all 32 lanes; returns the entry.
__device__ __forceinline__ uint32_t queue_vertex(const WaveBufs& b, bool vertex, const Vertex& v, V3 d) {
  const uint32_t ni = warp_reserve(&b.ctrl->nee_count, vertex);
  if (vertex && queue_fits(b, ni)) {
    b.nee_a[ni] = make_float4(v.p.x, v.p.y, v.p.z, __uint_as_float(v.slot));
    b.nee_b[ni] = make_float4(v.N.x, v.N.y, v.N.z, __int_as_float(v.mat));
    b.nee_c[ni] = make_float4(d.x, d.y, d.z, __uint_as_float(v.scene));
  }
  return ni;
}

// ---------------------------------------------------------------------------
// emitter search + bounce (shader.cu:196-209, 248-253; lambertian.cu:7-22)
//
// Each lane owns one opaque vertex at a time and runs a small state machine:
// start a shadow ray (hemisphere draw), traverse one BVH node per loop trip,
// and when the ray ends apply the reference's occlusion programs; after an
// emitter is seen (or 30 rays) it draws the bounce, writes the path state,
// appends the continuation ray and takes the next vertex.  Lanes advance
// independently, so a warp stays full while its vertices need between 1 and
// 30 rays of different lengths.
//
// Bound by issue: most tries are decided without a traversal, so the kernel
// is the arithmetic around the queue.  A warp therefore shades 32 rays at a
// time, each lane then testing all tries of its own vertex, and keeps the
// answers as a bit mask; shading, bound by memory latency in a kernel of its
// own, overlaps the other warps' traversals here, and its vertices never go
// through memory.  On the 1.31 M-triangle icosphere step (86 M rays, 59 M
// vertices) shading and search take 12.1 ms: 5.8 + 13.3 with a shading
// kernel and one warp-wide search per vertex and traversal, 5.7 + 8.9 with a
// shading kernel and prepared vertices.

// Guided bounce at an opaque vertex with roughness 1, where the reference
// draws hemi(N) (lambertian.cu:7-13): one-sample MIS between that sampler
// (probability c) and the guide's vMF mixture.  The path continues with
// weight p_hemi(w) / (c p_hemi(w) + (1-c) q_guide(w)), so the estimator's
// expectation is unchanged; directions below the surface get weight 0.
//
// Without NET, c = 1: the mixture is neither sampled nor weighed (its
// density times 0 adds nothing), so o is not read.
template <bool NET>
__device__ __forceinline__ V3 guided_bounce(const float* o, V3 N, uint32_t& seed, float c, float& weight) {
  guide::Lobe L[guide::LOBES];
  if (NET) guide::decode(o, L);
  V3 w;
  if (rnd(seed) < c || !NET) {
    w = bsdf::shoot_ray_hemisphere(N, seed);
  } else {
    const float u0 = rnd(seed), u1 = rnd(seed), u2 = rnd(seed);
    guide::mix_sample(L, u0, u1, u2, w.x, w.y, w.z);
  }
  const float ph = guide::hemi_pdf(N.x, N.y, N.z, w.x, w.y, w.z);
  const float q = NET ? c * ph + (1.0f - c) * guide::mix_pdf(L, w.x, w.y, w.z) : ph;
  weight = (ph > 0.0f && q > 0.0f && isfinite(q)) ? ph / q : 0.0f;
  return w;
}

// A warp of k_nee's vertices in shared memory: those it has prepared and not
// yet started, and each lane's own, which only the bookkeeping rounds touch
// (in registers it would cost the traversal a quarter of its occupancy).
struct NeeVertices {
  float4 p[32];      // position, slot
  float4 n[32];      // normal, material
  uint4 s[32];       // stream state, emitter flag, candidate tries, scene
  uint32_t ray[32];  // ray queue entry (its direction is the incoming one)
};
struct NeeLanes {
  float4 n[32];      // normal, material
  float4 d[32];      // shadow ray's direction, slot
  uint4 s[32];       // stream state, emitter flag, candidate tries, tries made
  uint2 r[32];       // ray queue entry, scene
};

// The whole warp shades 32 consecutive rays and prepares the opaque hits'
// emitter searches, whose tries are tested (emit_candidates) on all lanes.
// Returns the number of vertices.  A function of its own: inlined, its
// registers would be spilled inside the traversal.
template <bool GUIDED>
__device__ __noinline__ uint32_t fill_vertices(const WaveBufs& b, int depth, uint32_t base, uint32_t count,
                                               NeeVertices& vb) {
  const int lane = threadIdx.x & 31;
  const uint32_t i = base + (uint32_t)lane;
  Vertex v;
  const bool vertex = shade_ray<false>(b, depth, i, i < count, v);
  if (GUIDED) queue_vertex(b, vertex, v, vertex ? ld3(b.rd[depth & 1][i]) : v3(0.0f));
  const uint32_t vmask = __ballot_sync(FULL, vertex);
  if (vertex) {
    const uint32_t k = __popc(vmask & lanemask_lt()), vseed = b.ps_rng[v.slot];
    vb.p[k] = make_float4(v.p.x, v.p.y, v.p.z, __uint_as_float(v.slot));
    vb.n[k] = make_float4(v.N.x, v.N.y, v.N.z, __int_as_float(v.mat));
    vb.s[k] = make_uint4(vseed, __float_as_uint(v.att.w), emit_candidates(b.scenes[v.scene], v.p, v.N, vseed), v.scene);
    vb.ray[k] = i;
  }
  return __popc(vmask);
}

template <bool COUNT, bool GUIDED = false>
__global__ void __launch_bounds__(128, LISA_NEE_MIN_BLOCKS) k_nee(const __grid_constant__ WaveBufs b, int depth) {
  const int q = depth & 1;
  const uint32_t count = *(volatile uint32_t*)&b.ctrl->qcount[q];
  const int lane = threadIdx.x & 31;
  const uint32_t lt = lanemask_lt();
  uint2 stack[TRAV_STACK];
  TravState s;
  TraceScene ts;
  bool have = false, exhausted = false, ray_active = false;
  // the vertex position lives in the shadow ray's origin (s.r.o*)
  s.r.ox = s.r.oy = s.r.oz = 0.0f;
  uint32_t shadow = 0, walked = 0, visits = 0, tests = 0, vertices = 0;
  bool pending = false;  // a finished shadow ray not yet evaluated
  bool emit_pass = false;  // the traversal is of the emitters' own BVH
  __shared__ NeeLanes lane_buf[4];
  NeeLanes& vl = lane_buf[threadIdx.x >> 5];
  __shared__ NeeVertices vertex_buf[4];
  NeeVertices& vb = vertex_buf[threadIdx.x >> 5];
  uint32_t vb_next = 0, vb_count = 0;  // (the same in every lane)
  bool queue_empty = false;
  // LCG jumps over j tries (3 draws each), j = 0..31
  __shared__ uint2 s_jump[32];
  if (threadIdx.x < 32) {
    const LcgJump j = lcg_jump(3u * threadIdx.x);
    s_jump[threadIdx.x] = make_uint2(j.a, j.c);
  }
  __syncthreads();
  __shared__ TriPass tri_pass[4];
  TriPass& tp = tri_pass[threadIdx.x >> 5];
  while (true) {
    // Bookkeeping (evaluate finished rays, finish and fetch vertices, start
    // rays) runs only once enough lanes are idle, so its divergent code is
    // shared by many lanes; otherwise the warp keeps traversing.
    const uint32_t busy = __ballot_sync(FULL, ray_active);
    if (__popc(busy) <= (int)b.refill_busy_max) {
      bool want_ray = false, start = false, nearer = false;
      V3 nd = v3(0.0f);
      if (pending && emit_pass && s.best_prim >= 0) {
        // A try with the flag unset matters only if its closest hit is an
        // emitter.  The emitters' BVH gave the nearest emitter on the ray
        // (if none, the try is inconsequential: evaluated as a miss); the
        // scene's BVH, started from that hit as the best so far, keeps it
        // unless a triangle is nearer (or as near with a lower index) --
        // the same closest hit as one traversal of the whole scene.  Such a
        // triangle is not an emitter's, so that pass ends at the first one.
        nearer = start = true;
        pending = false;
      }
      emit_pass = emit_pass && !pending && !nearer;
      if (pending) {
        pending = false;
        uint4 s4 = vl.s[lane];
        int stale = (int)s4.y;
        if (s.best_prim >= 0) {
          // the occlusion hit program marks a hit only on an emitter and
          // otherwise leaves the flag as it was (shader.cu:177-184)
          if (s.best_mat >= 0) stale = s.best_mat;
        } else {
          stale = -1;  // miss (shader.cu:172-175)
        }
        const bool lit = stale >= 0;
        if (lit || ++s4.w == (uint32_t)NEE_TRIES) {
          const float4 n4 = vl.n[lane], d4 = vl.d[lane];
          const uint2 r2 = vl.r[lane];
          const V3 N = ld3(n4);
          const uint32_t slot = __float_as_uint(d4.w);
          uint32_t seed = s4.x;
          const SceneDev& sc = b.scenes[r2.y];
          const DevMaterial& m = sc.mats[__float_as_int(n4.w)];
          const V3 att = vertex_throughput(b.ps_att[slot], m);
          if (lit) {
            const DevMaterial& em = sc.mats[stale];
            const float brdf = bsdf::BRDF(N, ld3(d4), m);
            const float4 c = b.ps_col[slot];
            const V3 col = ld3(c) + (v3(em.emission[0], em.emission[1], em.emission[2]) * brdf) * att;
            b.ps_col[slot] = make_float4(col.x, col.y, col.z, c.w);
          }
          if (GUIDED && m.roughness == 1.0f) {
            // the bounce of a guided vertex is drawn by k_guided_infer,
            // after the guide has seen the emitter flag this search left
            want_ray = false;
          } else {
            const V3 D = ld3(b.rd[q][r2.x]);
            // the bounce is drawn at every vertex, the last one included, so
            // the per-pixel stream advances exactly as in the reference
            nd = bsdf::bounce(D, N, seed, m);
            want_ray = depth + 1 < (int)sc.num_bounces && !is_zero(nd);
          }
          b.ps_rng[slot] = seed;
          b.ps_att[slot] = make_float4(att.x, att.y, att.z, __int_as_float(stale));
          have = false;
        }
        vl.s[lane] = make_uint4(s4.x, (uint32_t)stale, s4.z, s4.w);
      }
      const uint32_t ri = warp_reserve(&b.ctrl->qcount[q ^ 1], want_ray);
      if (want_ray && queue_fits(b, ri)) {
        b.ro[q ^ 1][ri] = make_float4(s.r.ox, s.r.oy, s.r.oz, vl.d[lane].w);
        b.rd[q ^ 1][ri] = make_float4(nd.x, nd.y, nd.z, __uint_as_float(vl.r[lane].y));
      }
      // Idle lanes take their next vertices from the warp's buffer.  An empty
      // buffer is filled by the whole warp: it shades 32 consecutive rays, and
      // the opaque hits' tries are tested (emit_candidates) on all lanes.
      while (__any_sync(FULL, !have && !exhausted)) {
        if (vb_next == vb_count) {
          uint32_t base = 0;
          if (!queue_empty) {
            if (lane == 0) base = atomicAdd(&b.ctrl->head[HEAD_NEE], 32u);
            base = __shfl_sync(FULL, base, 0);
          }
          if (queue_empty || base >= count) {
            queue_empty = true;
            if (!have) exhausted = true;
            break;
          }
          vb_next = 0;
          vb_count = fill_vertices<GUIDED>(b, depth, base, count, vb);
          vertices += vb_count;
          __syncwarp();
        }
        const bool need = !have && !exhausted;
        const uint32_t nmask = __ballot_sync(FULL, need);
        const uint32_t k = vb_next + __popc(nmask & lt);
        vb_next = min(vb_next + (uint32_t)__popc(nmask), vb_count);
        if (need && k < vb_count) {
          const float4 a4 = vb.p[k];
          const uint4 v4 = vb.s[k];
          s.r.ox = a4.x;
          s.r.oy = a4.y;
          s.r.oz = a4.z;
          vl.n[lane] = vb.n[k];
          vl.d[lane] = make_float4(0.0f, 0.0f, 0.0f, a4.w);
          vl.s[lane] = make_uint4(v4.x, v4.y, v4.z, 0u);
          vl.r[lane] = make_uint2(vb.ray[k], v4.w);
          have = true;
        }
        __syncwarp();
      }
      if (!__any_sync(FULL, have)) break;
      // The next try of a vertex.  A ray that cannot reach an emitter can
      // only miss (the flag is cleared) or hit something else (the flag is
      // kept): with the flag unset, neither lights the vertex nor changes
      // the flag, so such a try is counted and its traversal skipped -- the
      // search's outcome, the flag it leaves and the seed after it are those
      // of tracing every try.  With the flag set, a ray that cannot reach an
      // emitter is traced to its first hit only (a hit lights the vertex
      // with the flag's emitter, a miss clears it); a ray that may reach one
      // is traced to its closest hit.
      //
      // The next try of a vertex whose flag is unset is its next candidate:
      // the LCG jumps over the tries before it.
      const V3 p = v3(s.r.ox, s.r.oy, s.r.oz);
      const float4 d4 = vl.d[lane];
      const SceneDev& sc = b.scenes[have ? vl.r[lane].y : 0u];
      V3 dir = ld3(d4);
      bool any = nearer;
      if (have && !ray_active && !start) {
        uint4 s4 = vl.s[lane];
        if ((int)s4.y < 0) {
          const uint32_t skipped = (uint32_t)__ffs((int)(s4.z >> s4.w)) - 1u;  // (the last try is always a candidate)
          const uint2 j = s_jump[skipped];
          s4.x = j.x * s4.x + j.y;
          s4.w += skipped;
          shadow += skipped;
        }
        ++shadow;
        const float hx = rng11(s4.x);
        const float hy = rng11(s4.x);
        const float hz = rng11(s4.x);
        dir = bsdf::hemisphere_direction(ld3(vl.n[lane]), hx, hy, hz);
        vl.s[lane] = s4;
        vl.d[lane] = make_float4(dir.x, dir.y, dir.z, d4.w);
        const bool capable = emit_may_hit(sc, p, dir);
        if (!capable && (int)s4.y < 0) {
          s.best_prim = -1;  // an inconsequential try: evaluated as a miss
          pending = true;
        } else {
          // with the flag unset, a ray that may reach an emitter first asks
          // the emitters' own BVH (scenes with more than a few emitter
          // triangles; with a few, the bounds test above is as selective)
          emit_pass = (int)s4.y < 0 && sc.num_etris >= EMIT_BVH_MIN_TRIS;
          any = !capable;
          start = true;
        }
      }
      if (start) {
        const float te = s.best_t;
        const int pe = s.best_prim, me = s.best_mat;
        ts = emit_pass ? trace_scene_emit(sc) : trace_scene(sc);
        ray_active = trav_begin(s, ts, p, dir, RAY_TMIN, RAY_TMAX, tp, any);
        if (nearer) {
          s.best_t = te;
          s.best_prim = pe;
          s.best_mat = me;
          s.cull = fmaf(te, 1.52587890625e-5f, te) + s.r.slack;
        }
        if (ray_active) ++walked;
        else emit_pass = false;
        pending = !ray_active;  // nothing to traverse: a miss
      }
      // while few lanes have a ray and some have a try to evaluate, the
      // bookkeeping goes on: most vertices need no traversal at all
      if (__popc(__ballot_sync(FULL, ray_active)) <= (int)b.refill_busy_max && __any_sync(FULL, pending)) continue;
    }
    if (trav_step_warp<COUNT, true>(ray_active, s, ts, stack, visits, tests, &b.ctrl->status, tp)) {
      ray_active = false;
      pending = true;
    }
  }
  warp_add64(&b.ctrl->rays_shadow, shadow);
  warp_add64(&b.ctrl->shadow_walked, walked);
  if (lane == 0 && vertices) atomicAdd(&b.ctrl->nee_total, (unsigned long long)vertices);
  if (COUNT) {
    warp_add64(&b.ctrl->node_visits[1], visits);
    warp_add64(&b.ctrl->tri_tests[1], tests);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) b.ctrl->head[HEAD_TRACE] = 0;  // trace of this depth is done
}

// Training records of guided vertices, in two halves so that the slot's
// atomic is in flight while the vertex is finished.  record_reserve keeps a
// vertex's record with probability 1 - drop (decided by a hash of slot,
// depth and the wave's salt, not by the path's stream; drop =
// ctrl->drop_prob, read once per launch), warp-aggregated over the lanes
// that call it, and returns the record index or ~0u; record_write fills it.
__device__ __forceinline__ bool record_keep(const WaveBufs& b, int depth, float drop, uint32_t slot, bool want) {
  if (b.rec_cap == 0) return false;  // a wave that does not train keeps no records
  const float u = (float)(tea<4>(slot * 16u + (uint32_t)depth, b.rec_salt) >> 8) * (1.0f / 16777216.0f);
  return want && u >= drop;
}

__device__ __forceinline__ uint32_t record_reserve(const WaveBufs& b, int depth, float drop, uint32_t slot,
                                                   bool want) {
  if (b.rec_cap == 0) return ~0u;
  const bool keep = record_keep(b, depth, drop, slot, want);
  const uint32_t active = __activemask();
  const uint32_t mask = __ballot_sync(active, keep);
  if (!mask) return ~0u;
  const int leader = __ffs(mask) - 1;
  const int lane = threadIdx.x & 31;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(&b.ctrl->rec_count, (uint32_t)__popc(mask));
  base = __shfl_sync(active, base, leader);
  const uint32_t k = base + __popc(mask & lanemask_lt());
  return keep && k < b.rec_cap ? k : ~0u;
}

struct Record {
  float4 r[4];
  float4 col;  // see WaveBufs
};
__device__ __forceinline__ void record_fill(Record& rec, uint32_t slot, float flag, float4 r0, float4 r1, float4 r2,
                                            float4 r3, V3 c0) {
  rec.r[0] = r0;
  rec.r[1] = r1;
  rec.r[2] = r2;
  rec.r[3] = r3;
  rec.col = make_float4(c0.x, c0.y, c0.z, __uint_as_float((slot << 1) | (flag != 0.0f ? 1u : 0u)));
}
__device__ __forceinline__ void record_write(const WaveBufs& b, uint32_t k, const Record& rec) {
  if (k == ~0u) return;
  for (int j = 0; j < 4; ++j) b.rec_list[4ull * k + j] = rec.r[j];
  b.rec_col[k] = rec.col;
}

// ---------------------------------------------------------------------------
// Guided bounces, in the epilogue of the guide's inference (k_guided_infer):
// thread t holds the 40 network outputs of emitter-queue entry i in
// registers and finishes that vertex, so the outputs never reach HBM.
//
// Reference estimator: the opaque vertices with roughness 1, whose bounce
// k_nee deferred until the guide had seen the emitter flag its search left,
// with a training record per vertex (the radiance later gathered along the
// new direction, over the throughput after the bounce, is the incident
// radiance).  Returns whether a continuation ray (p, nd) is wanted.
template <bool NET>
__device__ __forceinline__ bool guided_compat_vertex(const WaveBufs& b, int depth, float drop, uint32_t i,
                                                     const float* o, V3& p, V3& nd, uint32_t& slot, uint32_t& scene,
                                                     uint32_t& guided_n, Record& rec, bool& keep) {
  const float4 a4 = b.nee_a[i], b4 = b.nee_b[i], c4 = b.nee_c[i];
  slot = __float_as_uint(a4.w);
  scene = __float_as_uint(c4.w);
  const SceneDev& sc = b.scenes[scene];
  if (sc.mats[__float_as_int(b4.w)].roughness != 1.0f) return false;  // bounced in k_nee
  keep = !NET && record_keep(b, depth, drop, slot, true);
  const uint32_t rk = NET ? record_reserve(b, depth, drop, slot, true) : ~0u;
  const float4 cw = b.ps_col[slot];
  p = ld3(a4);
  const V3 N = ld3(b4);
  const V3 D = ld3(c4);
  uint32_t seed = b.ps_rng[slot];
  const float4 at = b.ps_att[slot];
  const int stale = __float_as_int(at.w);
  float weight;
  nd = guided_bounce<NET>(o, N, seed, b.bsdf_fraction, weight);
  const V3 att = ld3(at) * weight;
  const float il = rsqrtf(fmaxf(dot(D, D), 1e-30f));
  record_fill(rec, slot, stale >= 0 ? 1.0f : 0.0f, make_float4(p.x, p.y, p.z, weight),
              make_float4(N.x, N.y, N.z, nd.x), make_float4(-D.x * il, -D.y * il, -D.z * il, nd.y),
              make_float4(att.x, att.y, att.z, nd.z), ld3(cw));
  record_write(b, rk, rec);
  b.ps_rng[slot] = seed;
  b.ps_att[slot] = make_float4(att.x, att.y, att.z, at.w);
  ++guided_n;
  return depth + 1 < (int)sc.num_bounces && weight > 0.0f;
}

// ---------------------------------------------------------------------------
// physically based estimator at opaque vertices (opt-in; no reference
// counterpart).  Emitter sampling: one shadow ray toward a point of an
// emitter picked by area x luminance (two-sided emitters), weighted against
// the bounce's density by the power heuristic.  Bounce: the diffuse lobe
// with probability = roughness (cosine-weighted), else a mirror; the
// throughput takes the albedo when the vertex is left.  ps_att.w carries the
// solid-angle density of the last diffuse bounce (0 after a camera ray or a
// specular event) for the weight at an emitter hit (emitter_hit).
//
// Plain mode finishes each vertex here.  Guided mode (SPLIT) only traces the
// shadow ray and leaves (direction, density, cosine, emitter material,
// visibility) in nee_light; k_guided_infer weighs it with the guide's density
// and draws the bounce once the guide's inference has run.

// A warp of k_nee_pb's vertices in shared memory: prepared ones, and each
// lane's own (see NeeLanes).
struct PbVertices {
  float4 p[32];      // position, slot
  float4 n[32];      // normal that faces the incoming ray, material
  float4 w[32];      // direction to the emitter sample, its distance (0: no shadow ray)
  float4 l[32];      // density and cosine of the sample, its emitter's material, scene
  uint4 s[32];       // stream state, ray queue entry, emitter queue entry (SPLIT), -
};

// The whole warp shades 32 consecutive rays and draws the opaque hits'
// emitter samples; returns the number of vertices (see fill_vertices).
template <bool SPLIT>
__device__ __noinline__ uint32_t fill_pb_vertices(const WaveBufs& b, int depth, uint32_t base, uint32_t count,
                                                  PbVertices& vb) {
  const int lane = threadIdx.x & 31;
  const uint32_t i = base + (uint32_t)lane;
  Vertex v;
  const bool vertex = shade_ray<true>(b, depth, i, i < count, v);
  const V3 d = vertex ? ld3(b.rd[depth & 1][i]) : v3(0.0f);
  const uint32_t ventry = SPLIT ? queue_vertex(b, vertex, v, d) : 0u;
  const uint32_t vmask = __ballot_sync(FULL, vertex);
  if (vertex) {
    const uint32_t k = __popc(vmask & lanemask_lt());
    const SceneDev& vs = b.scenes[v.scene];
    uint32_t vseed = b.ps_rng[v.slot];
    const V3 n = dot(v.N, d) < 0.0f ? v.N : -v.N;
    V3 w = v3(0.0f);
    float vpl = 0.0f, vcos = 0.0f, far = 0.0f;
    int vem = 0;
    if (vs.mats[v.mat].roughness > 0.0f && vs.num_emit > 0) {
      V3 y;
      const uint32_t e = sample_emitter(vs, vseed, y);
      const V3 to = y - v.p;
      const float d2 = dot(to, to);
      const float dist = fsqrt(d2);
      w = to * fdiv(1.0f, dist);
      vcos = dot(n, w);
      const float cos_y = fabsf(dot(ld3(__ldg(vs.emit + 4ull * e + 3)), w));
      if (vcos > 0.0f && cos_y > 0.0f && dist > 0.0f) {
        vpl = fdiv(fmul(__ldg(vs.emit + 4ull * e).w, d2), cos_y);
        vem = __float_as_int(__ldg(vs.emit + 4ull * e + 1).w);
        far = dist;
      }
    }
    vb.p[k] = make_float4(v.p.x, v.p.y, v.p.z, __uint_as_float(v.slot));
    vb.n[k] = make_float4(n.x, n.y, n.z, __int_as_float(v.mat));
    vb.w[k] = make_float4(w.x, w.y, w.z, far);
    vb.l[k] = make_float4(vpl, vcos, __int_as_float(vem), __uint_as_float(v.scene));
    vb.s[k] = make_uint4(vseed, i, ventry, 0u);
  }
  return __popc(vmask);
}

template <bool COUNT, bool SPLIT>
__global__ void __launch_bounds__(128, LISA_NEE_PB_MIN_BLOCKS) k_nee_pb(const __grid_constant__ WaveBufs b, int depth) {
  const int q = depth & 1;
  const uint32_t count = *(volatile uint32_t*)&b.ctrl->qcount[q];
  const int lane = threadIdx.x & 31;
  const uint32_t lt = lanemask_lt();
  uint2 stack[TRAV_STACK];
  TravState s;
  TraceScene ts;
  bool have = false, exhausted = false, ray_active = false, pending = false;
  uint32_t nshadow = 0, visits = 0, tests = 0, vertices = 0;
  __shared__ TriPass tri_pass[4];
  TriPass& tp = tri_pass[threadIdx.x >> 5];
  __shared__ PbVertices vertex_buf[4], lane_buf[4];
  PbVertices& vb = vertex_buf[threadIdx.x >> 5];
  PbVertices& vl = lane_buf[threadIdx.x >> 5];
  uint32_t vb_next = 0, vb_count = 0;  // (the same in every lane)
  bool queue_empty = false;
  while (true) {
    const uint32_t busy = __ballot_sync(FULL, ray_active);
    if (__popc(busy) <= (int)b.refill_busy_max) {
      bool want_ray = false;
      V3 nd = v3(0.0f);
      // the lane's vertex (undefined without one)
      const float4 p4 = vl.p[lane];
      const uint32_t slot = __float_as_uint(p4.w), scene = __float_as_uint(vl.l[lane].w);
      if (pending) {
        pending = false;
        const float4 n4 = vl.n[lane], w4 = vl.w[lane], l4 = vl.l[lane];
        const uint4 s4 = vl.s[lane];
        const SceneDev& sc = b.scenes[scene];
        const DevMaterial& m = sc.mats[__float_as_int(n4.w)];
        const V3 Ns = ld3(n4), wi = ld3(w4);
        const float pl = l4.x, cos_x = l4.y;
        const int em_m = __float_as_int(l4.z);
        const uint32_t ray = s4.y, entry = s4.z;
        uint32_t seed = s4.x;
        const bool lit = w4.w > 0.0f && s.best_prim < 0;
        const float4 at = b.ps_att[slot];
        const V3 att = vertex_throughput(at, m);
        if (SPLIT) {
          b.nee_light[2ull * entry] = make_float4(wi.x, wi.y, wi.z, pl);
          b.nee_light[2ull * entry + 1] = make_float4(cos_x, __int_as_float(em_m), lit ? 1.0f : 0.0f, 0.0f);
          b.ps_rng[slot] = seed;
          b.ps_att[slot] = make_float4(att.x, att.y, att.z, at.w);
        } else {
          const float r = m.roughness;
          if (lit) {
            const DevMaterial& em = sc.mats[em_m];
            const float fcos = fmul(r, fdiv(cos_x, PI_F));
            // power heuristic against the bounce (traced at every vertex, the
            // last one's for the emission it reaches only)
            const float wl = fdiv(fmul(pl, pl), fadd(fmul(pl, pl), fmul(fcos, fcos)));
            const float4 c = b.ps_col[slot];
            const V3 col =
                ld3(c) + ((att * v3(em.emission[0], em.emission[1], em.emission[2])) * fdiv(fcos, pl)) * wl;
            b.ps_col[slot] = make_float4(col.x, col.y, col.z, c.w);
          }
          float prev = 0.0f;
          if (r >= 1.0f || (r > 0.0f && rnd(seed) < r)) {
            nd = cosine_dir(Ns, seed);
            prev = fmul(r, fdiv(dot(Ns, nd), PI_F));
          } else {
            nd = reflect(ld3(b.rd[q][ray]), Ns);
          }
          want_ray = !is_zero(nd);
          if (want_ray && depth + 1 == (int)sc.num_bounces) want_ray = final_ray_wanted(sc, ld3(p4), nd);
          b.ps_rng[slot] = seed;
          b.ps_att[slot] = make_float4(att.x, att.y, att.z, prev);
        }
        have = false;
      }
      const uint32_t ri = warp_reserve(&b.ctrl->qcount[q ^ 1], want_ray);
      if (want_ray && queue_fits(b, ri)) {
        b.ro[q ^ 1][ri] = p4;
        b.rd[q ^ 1][ri] = make_float4(nd.x, nd.y, nd.z, __uint_as_float(scene));
      }
      // Idle lanes take their next vertices from the warp's buffer; an empty
      // one is filled by the whole warp, which shades 32 consecutive rays and
      // draws the opaque hits' emitter samples.
      while (__any_sync(FULL, !have && !exhausted)) {
        if (vb_next == vb_count) {
          uint32_t base = 0;
          if (!queue_empty) {
            if (lane == 0) base = atomicAdd(&b.ctrl->head[HEAD_NEE], 32u);
            base = __shfl_sync(FULL, base, 0);
          }
          if (queue_empty || base >= count) {
            queue_empty = true;
            if (!have) exhausted = true;
            break;
          }
          vb_next = 0;
          vb_count = fill_pb_vertices<SPLIT>(b, depth, base, count, vb);
          vertices += vb_count;
          __syncwarp();
        }
        const bool need = !have && !exhausted;
        const uint32_t nmask = __ballot_sync(FULL, need);
        const uint32_t k = vb_next + __popc(nmask & lt);
        vb_next = min(vb_next + (uint32_t)__popc(nmask), vb_count);
        if (need && k < vb_count) {
          const float4 a4 = vb.p[k], w4 = vb.w[k], l4 = vb.l[k];
          vl.p[lane] = a4;
          vl.n[lane] = vb.n[k];
          vl.w[lane] = w4;
          vl.l[lane] = l4;
          vl.s[lane] = vb.s[k];
          have = true;
          s.best_prim = -1;
          if (w4.w > 0.0f) {
            ++nshadow;
            ts = trace_scene(b.scenes[__float_as_uint(l4.w)]);
            // stop short of the emitter itself; any blocker will do
            ray_active = trav_begin(s, ts, ld3(a4), ld3(w4), RAY_TMIN, fmul(w4.w, 0.9990234375f), tp, true);
          }
          pending = !ray_active;  // no shadow ray, or nothing to traverse
        }
        __syncwarp();
      }
      if (!__any_sync(FULL, have)) break;
      if (__popc(__ballot_sync(FULL, ray_active)) <= (int)b.refill_busy_max && __any_sync(FULL, pending)) continue;
    }
    if (trav_step_warp<COUNT, true>(ray_active, s, ts, stack, visits, tests, &b.ctrl->status, tp)) {
      ray_active = false;
      pending = true;
    }
  }
  warp_add64(&b.ctrl->rays_shadow, nshadow);
  warp_add64(&b.ctrl->shadow_walked, nshadow);  // every shadow ray of this estimator is traced
  if (lane == 0 && vertices) atomicAdd(&b.ctrl->nee_total, (unsigned long long)vertices);
  if (COUNT) {
    warp_add64(&b.ctrl->node_visits[1], visits);
    warp_add64(&b.ctrl->tri_tests[1], tests);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) b.ctrl->head[HEAD_TRACE] = 0;  // trace of this depth is done
}

// Physically based estimator: the emitter sample of k_nee_pb weighed
// against the guided density, then the bounce -- the diffuse lobe by
// one-sample MIS between cosine sampling (probability c) and the guide's
// mixture, q = c cos/pi + (1-c) q_guide, throughput x (cos/pi) / q -- with a
// training record per diffuse bounce.
template <bool NET>
__device__ __forceinline__ bool guided_pb_vertex(const WaveBufs& b, int depth, float drop, uint32_t i, const float* o,
                                                 V3& p, V3& nd, uint32_t& slot, uint32_t& scene, uint32_t& guided_n,
                                                 Record& rec, bool& keep) {
  const float c = b.bsdf_fraction;
  const float4 a4 = b.nee_a[i], b4 = b.nee_b[i], c4 = b.nee_c[i];
  p = ld3(a4);
  slot = __float_as_uint(a4.w);
  scene = __float_as_uint(c4.w);
  const V3 N = ld3(b4);
  const V3 D = ld3(c4);
  const V3 Ns = dot(N, D) < 0.0f ? N : -N;
  const float4 cw = b.ps_col[slot];
  const SceneDev& sc = b.scenes[scene];
  const float r = sc.mats[__float_as_int(b4.w)].roughness;
  V3 att = ld3(b.ps_att[slot]);
  V3 col = ld3(cw);
  uint32_t seed = b.ps_rng[slot];
  // the lobe choice is the stream's first draw at this vertex, as when the
  // bounce is drawn in k_nee_pb; decided first so that the training
  // record's slot is reserved while the mixture is evaluated
  const bool diffuse = r >= 1.0f || (r > 0.0f && rnd(seed) < r);
  keep = !NET && record_keep(b, depth, drop, slot, diffuse);
  const uint32_t rk = NET ? record_reserve(b, depth, drop, slot, diffuse) : ~0u;
  guide::Lobe L[guide::LOBES];
  if (NET) guide::decode(o, L);
  const float4 l0 = b.nee_light[2ull * i], l1 = b.nee_light[2ull * i + 1];
  if (l1.z != 0.0f) {
    const float pl = l0.w, cos_x = l1.x;
    const DevMaterial& em = sc.mats[__float_as_int(l1.y)];
    // (fast reciprocals: the guided bounce's densities need no bit-exact
    // agreement with the oracle, only the same values for sampling and weight)
    const float fcos = r * cos_x * (1.0f / PI_F);
    const float px = cos_x * (1.0f / PI_F);
    const float pb = r * (NET ? c * px + (1.0f - c) * guide::mix_pdf(L, l0.x, l0.y, l0.z) : px);
    const float wl = __fdividef(pl * pl, pl * pl + pb * pb);
    col = col + ((att * v3(em.emission[0], em.emission[1], em.emission[2])) * __fdividef(fcos, pl)) * wl;
  }
  float prev = 0.0f;
  bool want;
  if (diffuse) {
    if (rnd(seed) < c || !NET) {
      nd = cosine_dir(Ns, seed);
    } else {
      const float u0 = rnd(seed), u1 = rnd(seed), u2 = rnd(seed);
      guide::mix_sample(L, u0, u1, u2, nd.x, nd.y, nd.z);
    }
    const float cs = dot(Ns, nd);
    const float pc = cs > 0.0f ? cs * (1.0f / PI_F) : 0.0f;
    const float qm = NET ? c * pc + (1.0f - c) * guide::mix_pdf(L, nd.x, nd.y, nd.z) : pc;
    const float weight = (pc > 0.0f && qm > 0.0f && isfinite(qm)) ? __fdividef(pc, qm) : 0.0f;
    att = att * weight;
    prev = r * qm;
    want = weight > 0.0f;
    const float il = rsqrtf(fmaxf(dot(D, D), 1e-30f));
    record_fill(rec, slot, 0.0f, make_float4(p.x, p.y, p.z, weight), make_float4(N.x, N.y, N.z, nd.x),
                make_float4(-D.x * il, -D.y * il, -D.z * il, nd.y), make_float4(att.x, att.y, att.z, nd.z), col);
    record_write(b, rk, rec);
    ++guided_n;
  } else {
    nd = reflect(D, Ns);
    want = true;
  }
  if (want && depth + 1 == (int)sc.num_bounces) want = final_ray_wanted(sc, p, nd);
  b.ps_col[slot] = make_float4(col.x, col.y, col.z, cw.w);
  b.ps_rng[slot] = seed;
  b.ps_att[slot] = make_float4(att.x, att.y, att.z, prev);
  return want;
}

// The guide's inference on the emitter queue of this depth, fused with the
// guided bounces of those vertices (tensor-core layers, guide_infer.cuh;
// bounce in the last layer's epilogue).
template <bool PHYS>
__global__ void __launch_bounds__(INFER_THREADS, INFER_BLOCKS_PER_SM) k_guided_infer(const uint16_t* __restrict__ pack,
                                                                           const float* __restrict__ master,
                                                                           GuideSrc src, uint32_t* status, WaveBufs b,
                                                                           int depth) {
  const int q = depth & 1;
  uint32_t guided_n = 0;
  const float drop = b.ctrl->drop_prob;  // written by the last wave's record collection
  // the path state and emitter sample that the guided bounce reads, brought
  // into L2 while the five layers run
  auto pre = [&](uint32_t i) {
    const uint32_t slot = __float_as_uint(b.nee_a[i].w);
    prefetch_l2(b.ps_col + slot);
    prefetch_l2(b.ps_rng + slot);
    if (PHYS) {
      prefetch_l2(b.ps_att + slot);  // (the reference estimator's flag feature has loaded it)
      prefetch_l2(b.nee_light + 2ull * i);
    }
  };
  infer_tiles<SRC_NEE>(pack, master, src, status, pre, [&](uint32_t i, bool valid, const float* o) {
    bool want = false;
    V3 p = v3(0.0f), nd = v3(0.0f);
    uint32_t slot = 0, scene = 0;
    Record rec;
    bool keep;
    if (valid) {
      if (PHYS) want = guided_pb_vertex<true>(b, depth, drop, i, o, p, nd, slot, scene, guided_n, rec, keep);
      else want = guided_compat_vertex<true>(b, depth, drop, i, o, p, nd, slot, scene, guided_n, rec, keep);
    }
    const uint32_t ri = warp_reserve(&b.ctrl->qcount[q ^ 1], want);
    if (want && queue_fits(b, ri)) {
      b.ro[q ^ 1][ri] = make_float4(p.x, p.y, p.z, __uint_as_float(slot));
      b.rd[q ^ 1][ri] = make_float4(nd.x, nd.y, nd.z, __uint_as_float(scene));
    }
  });
  warp_add32(&b.ctrl->guided_count, guided_n);
  if (blockIdx.x == 0 && threadIdx.x == 0) b.ctrl->infer_rows += *(volatile uint32_t*)&b.ctrl->nee_count;
}

// The same vertices where the BSDF draws every bounce (bsdf_fraction 1: a
// warm-up wave, whose records train the guide): the guide's density has no
// weight, so its network does not run.  Bound by the gathers of path state
// and by the atomics on the queue and record counters, one each for a block
// of 256: 0.91 ms for 14.2 M vertices of eight depths (1.22 with a warp's
// atomics), 2.02 with the network.  Resident blocks only: eight an SM in
// turn took 0.1 ms more, 32 0.7.
constexpr int BOUNCE_BLOCKS_PER_SM = 4;

template <bool PHYS>
__global__ void __launch_bounds__(256, BOUNCE_BLOCKS_PER_SM) k_bsdf_bounce(WaveBufs b, int depth) {
  const int q = depth & 1;
  const uint32_t count = min(*(volatile uint32_t*)&b.ctrl->nee_count, b.capacity);
  const float drop = b.ctrl->drop_prob;
  uint32_t guided_n = 0;
  __shared__ uint2 s_n[8];  // per warp: rays for the next queue, records
  __shared__ uint32_t s_ray, s_rec;
  const uint32_t warp = threadIdx.x >> 5;
  for (uint32_t base = blockIdx.x * blockDim.x; base < count; base += gridDim.x * blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    bool want = false, keep = false;
    V3 p = v3(0.0f), nd = v3(0.0f);
    uint32_t slot = 0, scene = 0;
    Record rec;
    if (i < count) {
      if (PHYS) want = guided_pb_vertex<false>(b, depth, drop, i, nullptr, p, nd, slot, scene, guided_n, rec, keep);
      else want = guided_compat_vertex<false>(b, depth, drop, i, nullptr, p, nd, slot, scene, guided_n, rec, keep);
    }
    // places in both lists, one atomic each for the block
    const uint32_t rays = __ballot_sync(FULL, want), recs = __ballot_sync(FULL, keep);
    if ((threadIdx.x & 31u) == 0) s_n[warp] = make_uint2(__popc(rays), __popc(recs));
    __syncthreads();
    uint2 before = make_uint2(0u, 0u), all = before;
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
      const uint2 v = s_n[k];
      if (k == warp) before = all;
      all.x += v.x;
      all.y += v.y;
    }
    if (threadIdx.x == 0) s_ray = atomicAdd(&b.ctrl->qcount[q ^ 1], all.x);
    if (threadIdx.x == 32 && all.y) s_rec = atomicAdd(&b.ctrl->rec_count, all.y);
    __syncthreads();
    if (want) {
      const uint32_t ri = s_ray + before.x + __popc(rays & lanemask_lt());
      if (queue_fits(b, ri)) {
        b.ro[q ^ 1][ri] = make_float4(p.x, p.y, p.z, __uint_as_float(slot));
        b.rd[q ^ 1][ri] = make_float4(nd.x, nd.y, nd.z, __uint_as_float(scene));
      }
    }
    if (keep) {
      const uint32_t k = s_rec + before.y + __popc(recs & lanemask_lt());
      if (k < b.rec_cap) record_write(b, k, rec);
    }
  }
  warp_add32(&b.ctrl->guided_count, guided_n);
}

// With one stream per pixel: the first path of the wave's pixel `item`, and
// the distance from path `slot` to its pixel's next (0: the last one).
__device__ __forceinline__ uint32_t first_of_pixel(const WaveDesc& w, uint32_t item) {
  const WaveGroup& g = w.groups[find_group(w, item, true)];
  return g.slot0 + (item - g.acc0);
}
__device__ __forceinline__ uint32_t next_of_pixel(const WaveDesc& w, uint32_t slot) {
  const WaveGroup& g = w.groups[find_group(w, slot, false)];
  return slot - g.slot0 + g.npix < g.nplanes * g.npix ? g.npix : 0u;
}

// ---------------------------------------------------------------------------
// whole paths in one kernel (plain sampling, small waves)
//
// A lane takes a path from camera to end: closest hit, shading, emitter
// search and bounce, depth after depth, advancing one BVH node per loop trip
// like the stage kernels, whose routines it calls in the same order -- the
// paths are the same bit for bit.  Nothing passes through memory but the
// path's final radiance.  With CHAIN (one stream per pixel) a lane takes a
// pixel's paths in turn, each going on with the stream of the one before.
//
// For small waves, whose time is the latency of the stages and not their
// throughput: each stage launch ends with the wave's longest ray (up to a
// hundred node visits of about a microsecond), and a frame is a chain of
// three such launches per depth.  Here a path waits only for itself: a
// 160 x 90 preview of the Cornell box takes 163 us instead of 397, a
// 333 x 217 frame of eight samples with one stream per pixel 1.9 instead of 8.3.  It is
// bound by issue (58 % of the slots) and by instruction fetch: the loop is
// 42 KB of code, so a routine is written once and shared by the ray kinds
// (two more copies of trav_begin and of the triangle test cost 10 %).
template <bool PHYS, bool CHAIN>
__global__ void __launch_bounds__(128, LISA_PATHS_MIN_BLOCKS) k_paths(WaveBufs b, const WaveDesc* __restrict__ wave,
                                                                      uint32_t lanes) {
  const WaveDesc& w = *wave;
  const uint32_t count = CHAIN ? w.acc_items : w.paths;
  const int lane = threadIdx.x & 31;
  const uint32_t lt = lanemask_lt();
  uint2 stack[TRAV_STACK];
  TravState s;
  TraceScene ts;
  const SceneDev* sc = nullptr;
  // a lane with a path traces a radiance ray, or (shadow) an emitter-search
  // ray from the vertex p; its ray's origin is s.r.o
  bool have = false, exhausted = (uint32_t)lane >= lanes, ray_active = false, pending = false, shadow = false;
  bool emit_pass = false;  // the finished traversal was of the emitters' own BVH
  uint32_t slot = 0, seed = 0, cand = 0;
  int depth = 0, tries = 0, mat_idx = 0;
  int stale = -1;             // reference estimator: stale emitter flag
  float pdf = 0.0f;           // physically based: density of the last diffuse bounce
  int em_m = 0;               // physically based: the sampled emitter's material, density and cosine
  float pl = 0.0f, cos_x = 0.0f;
  V3 att = v3(0.0f), col = v3(0.0f);
  V3 N = v3(0.0f), D = v3(0.0f), dir = v3(0.0f);  // normal; radiance ray; current ray
  s.r.ox = s.r.oy = s.r.oz = 0.0f;
  uint32_t nbounce = 0, nshadow = 0, nwalked = 0, nvertex = 0;
  uint32_t visits = 0, tests = 0;
  __shared__ uint2 s_jump[32];
  if (threadIdx.x < 32) {
    const LcgJump j = lcg_jump(3u * threadIdx.x);
    s_jump[threadIdx.x] = make_uint2(j.a, j.c);
  }
  __syncthreads();
  __shared__ TriPass tri_pass[4];
  TriPass& tp = tri_pass[threadIdx.x >> 5];
  while (true) {
    const uint32_t busy = __ballot_sync(FULL, ray_active);
    if (__popc(busy) <= (int)b.refill_busy_max) {
      bool vertex = false;   // a new opaque vertex
      bool search = false;   // a vertex that needs its next try (reference estimator)
      bool leave = false;    // a vertex whose emitter search is over: draw the bounce
      bool lit = false, start = false, over = false;
      bool fresh = false;    // a new path
      bool nearer = false;   // look for a triangle nearer than the emitter hit
      float tmax = RAY_TMAX;
      V3 p = v3(s.r.ox, s.r.oy, s.r.oz);
      if (pending && shadow) {
        pending = false;
        if (PHYS) {
          lit = s.best_prim < 0;
          leave = true;
        } else if (emit_pass && s.best_prim >= 0) {
          // the emitters' BVH gave the nearest emitter on the ray: the scene's
          // keeps it unless a triangle is nearer (see k_nee)
          emit_pass = false;
          nearer = true;
          start = true;
        } else {
          emit_pass = false;
          // the occlusion programs: a hit marks only an emitter and otherwise
          // leaves the flag as it was, a miss clears it (shader.cu:172-184)
          if (s.best_prim < 0) stale = -1;
          else if (s.best_mat >= 0) stale = s.best_mat;
          lit = stale >= 0;
          leave = lit || ++tries == NEE_TRIES;
          search = !leave;
        }
      } else if (pending) {
        pending = false;
        over = true;
        const int prim = s.best_prim;
        if (prim >= 0) {  // a miss adds the background, 0, and ends the path
          mat_idx = prim_material(*sc, prim);
          const DevMaterial& m = sc->mats[mat_idx];
          if (m.cls == MAT_EMIT) {
            col = col + emitter_hit<PHYS>(*sc, m, prim, s.best_t, D, make_float4(att.x, att.y, att.z, pdf));
          } else if (!PHYS || depth < (int)sc->num_bounces) {
            p = p + s.best_t * D;
            N = barycentric_normal(p, sc->prims + 5ull * prim);
            if (m.cls == MAT_DIELECTRIC) {
              const V3 nd = dielectric_bounce<PHYS>(m, D, N, att, seed);
              if (PHYS) pdf = 0.0f;
              start = (PHYS || depth + 1 < (int)sc->num_bounces) && !is_zero(nd);
              if (PHYS && start && depth + 1 == (int)sc->num_bounces) start = final_ray_wanted(*sc, p, nd);
              over = !start;
              D = nd;
            } else {
              att = att * v3(m.albedo[0], m.albedo[1], m.albedo[2]);
              over = false;
              vertex = true;
              ++nvertex;
            }
          }
        }
      }
      if (PHYS) {
        if (vertex) {
          N = dot(N, D) < 0.0f ? N : -N;  // faces the incoming ray
          leave = true;
          if (sc->mats[mat_idx].roughness > 0.0f && sc->num_emit > 0) {
            V3 y;
            const uint32_t k = sample_emitter(*sc, seed, y);
            const V3 to = y - p;
            const float d2 = dot(to, to);
            const float dist = fsqrt(d2);
            dir = to * fdiv(1.0f, dist);
            cos_x = dot(N, dir);
            const float cos_y = fabsf(dot(ld3(__ldg(sc->emit + 4ull * k + 3)), dir));
            if (cos_x > 0.0f && cos_y > 0.0f && dist > 0.0f) {
              pl = fdiv(fmul(__ldg(sc->emit + 4ull * k).w, d2), cos_y);
              em_m = __float_as_int(__ldg(sc->emit + 4ull * k + 1).w);
              ++nshadow;
              // stop short of the emitter itself; any blocker will do
              tmax = fmul(dist, 0.9990234375f);
              shadow = true;
              start = true;
              leave = false;
            }
          }
        }
      } else {
        // the tries of each new vertex that may reach an emitter: lane j
        // tests try j of one vertex after another
        uint32_t vmask = __ballot_sync(FULL, vertex);
        if (vmask) {
          const EmitBounds e = vertex ? emit_bounds(*sc, p) : EmitBounds{};
          while (vmask) {
            const int owner = __ffs(vmask) - 1;
            vmask &= vmask - 1;
            EmitBounds o;
            o.c = v3(__shfl_sync(FULL, e.c.x, owner), __shfl_sync(FULL, e.c.y, owner), __shfl_sync(FULL, e.c.z, owner));
            o.h = v3(__shfl_sync(FULL, e.h.x, owner), __shfl_sync(FULL, e.h.y, owner), __shfl_sync(FULL, e.h.z, owner));
            const V3 on = v3(__shfl_sync(FULL, N.x, owner), __shfl_sync(FULL, N.y, owner), __shfl_sync(FULL, N.z, owner));
            const uint2 j = s_jump[lane];
            uint32_t st = j.x * __shfl_sync(FULL, seed, owner) + j.y;
            const uint32_t mask = __ballot_sync(FULL, emit_candidate(o, on, st));
            if (lane == owner) cand = mask;
          }
          if (vertex) {
            cand = (sc->has_emit_box ? cand & ((1u << (NEE_TRIES - 1)) - 1u) : 0u) | (1u << (NEE_TRIES - 1));
            tries = 0;
            shadow = true;
            search = true;
          }
        }
        // The next try that is traced (see k_nee): with the flag unset, tries
        // that cannot reach an emitter are only counted.
        while (search) {
          if (stale < 0) {
            const uint32_t skip = (uint32_t)__ffs((int)(cand >> tries)) - 1u;  // (the last try is always a candidate)
            const uint2 j = s_jump[skip];
            seed = j.x * seed + j.y;
            tries += (int)skip;
            nshadow += skip;
          }
          ++nshadow;
          const float hx = rng11(seed);
          const float hy = rng11(seed);
          const float hz = rng11(seed);
          dir = bsdf::hemisphere_direction(N, hx, hy, hz);
          const bool capable = emit_may_hit(*sc, p, dir);
          if (!capable && stale < 0) {
            leave = ++tries == NEE_TRIES;
            search = !leave;
          } else {
            emit_pass = stale < 0 && sc->num_etris >= EMIT_BVH_MIN_TRIS;
            s.any = !capable;
            start = true;
            search = false;
          }
        }
      }
      if (leave) {
        const DevMaterial& m = sc->mats[mat_idx];
        V3 nd;
        if (PHYS) {
          const float r = m.roughness;
          if (lit) {
            const DevMaterial& em = sc->mats[em_m];
            const float fcos = fmul(r, fdiv(cos_x, PI_F));
            // power heuristic against the bounce
            const float wl = fdiv(fmul(pl, pl), fadd(fmul(pl, pl), fmul(fcos, fcos)));
            col = col + ((att * v3(em.emission[0], em.emission[1], em.emission[2])) * fdiv(fcos, pl)) * wl;
          }
          pdf = 0.0f;
          if (r >= 1.0f || (r > 0.0f && rnd(seed) < r)) {
            nd = cosine_dir(N, seed);
            pdf = fmul(r, fdiv(dot(N, nd), PI_F));
          } else {
            nd = reflect(D, N);
          }
          start = !is_zero(nd);
          if (start && depth + 1 == (int)sc->num_bounces) start = final_ray_wanted(*sc, p, nd);
        } else {
          if (lit) {
            const DevMaterial& em = sc->mats[stale];
            col = col + (v3(em.emission[0], em.emission[1], em.emission[2]) * bsdf::BRDF(N, dir, m)) * att;
          }
          nd = bsdf::bounce(D, N, seed, m);
          start = depth + 1 < (int)sc->num_bounces && !is_zero(nd);
        }
        shadow = false;
        over = !start;
        D = nd;
      }
      if (over) {
        b.ps_col[slot] = make_float4(col.x, col.y, col.z, 0.0f);
        have = false;
        if (CHAIN) {
          const uint32_t next = next_of_pixel(w, slot);
          if (next) {
            slot += next;
            have = fresh = true;
          } else {
            b.ps_rng[slot] = seed;
          }
        }
      } else if (start && !shadow) {
        ++depth;
        ++nbounce;
      }
      const bool need = !have && !exhausted;
      const uint32_t nmask = __ballot_sync(FULL, need);
      if (nmask) {
        const int leader = __ffs(nmask) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(&b.ctrl->head[HEAD_TRACE], (uint32_t)__popc(nmask));
        base = __shfl_sync(FULL, base, leader);
        if (need) {
          slot = base + __popc(nmask & lt);
          have = fresh = slot < count;
          exhausted = !have;
          if (CHAIN && have) slot = first_of_pixel(w, slot);
        }
      }
      if (fresh) {
        uint32_t scene, pix;
        camera_ray(b, w, slot, scene, pix, seed, p, D);
        sc = b.scenes + scene;
        att = v3(1.0f);
        col = v3(0.0f);
        stale = -1;
        pdf = 0.0f;
        depth = 0;
        shadow = false;
        start = true;
      }
      if (!__any_sync(FULL, have)) break;
      if (start) {
        if (!shadow) dir = D;
        const bool any = shadow && (PHYS || s.any || nearer);
        const float te = s.best_t;
        const int pe = s.best_prim, me = s.best_mat;
        ts = emit_pass ? trace_scene_emit(*sc) : trace_scene(*sc);
        ray_active = trav_begin(s, ts, p, dir, RAY_TMIN, tmax, tp, any);
        s.r.ox = p.x;  // (kept when there is nothing to traverse)
        s.r.oy = p.y;
        s.r.oz = p.z;
        if (!PHYS && nearer) {
          s.best_t = te;
          s.best_prim = pe;
          s.best_mat = me;
          s.cull = fmaf(te, 1.52587890625e-5f, te) + s.r.slack;
        }
        if (ray_active) nwalked += shadow ? 1u : 0u;
        else emit_pass = false;
        pending = !ray_active;
      }
    }
    if (trav_step_warp<false, true>(ray_active, s, ts, stack, visits, tests, &b.ctrl->status, tp)) {
      ray_active = false;
      pending = true;
    }
  }
  warp_add64(&b.ctrl->rays_bounce, nbounce);
  warp_add64(&b.ctrl->rays_shadow, nshadow);
  warp_add64(&b.ctrl->shadow_walked, nwalked);
  warp_add64(&b.ctrl->nee_total, nvertex);
  if (blockIdx.x == 0 && threadIdx.x == 0) b.ctrl->rays_primary += w.paths;
}

// ---------------------------------------------------------------------------
// accumulate: per pixel, the wave's samples in sample order

// A float's double, and its square's (48 bits, so exact), put together from
// integers: the GPU has so few double units that a conversion or a product
// costs as much as thirty integer instructions.  Zeros, which black pixels
// are full of, come out of the general form of the first; subnormals,
// infinities and NaN take the double units.
__device__ __forceinline__ double as_double(float v) {
  const uint32_t u = __float_as_uint(v), e = (u >> 23) & 0xffu;
  if (e == 0xffu || (e == 0u && (u & 0x7fffffu))) return (double)v;
  const uint32_t hi = (u & 0x80000000u) | ((e ? e + 896u : 0u) << 20) | ((u & 0x7fffffu) >> 3);
  return __hiloint2double((int)hi, (int)(u << 29));
}
__device__ __forceinline__ double square_as_double(float v) {
  const uint32_t u = __float_as_uint(v), e = (u >> 23) & 0xffu;
  if (e == 0xffu || e == 0u) return (u << 1) ? __dmul_rn((double)v, (double)v) : 0.0;
  // (1.m x 2^23)^2 has its top bit at 46 or 47; moved to 52 it adds one to
  // the exponent field: 2 (e - 150) + 46 or 47, biased by 1023
  const unsigned long long m = (u & 0x7fffffu) | 0x800000u, p = m * m;
  const uint32_t top = (uint32_t)(p >> 47);
  return __longlong_as_double((long long)((p << (6u - top)) + ((unsigned long long)(2u * e + 768u + top) << 52)));
}

// Per pixel of the wave: its samples in order into the float Kahan sum, the
// FP64 sum of squares and, if asked for, the FP64 sum.  Bound by the double
// additions, three or six a sample: 0.12 ms for 16.8 M samples of 1 Mi
// pixels, 0.39 with the squares in double products.
__global__ void k_accumulate(WaveBufs b, const WaveDesc* __restrict__ wave) {
  const WaveDesc& w = *wave;
  if (blockIdx.x == 0 && threadIdx.x == 0) b.ctrl->head[HEAD_TRACE] = 0;  // for a whole-path wave that follows
  for (uint32_t item = blockIdx.x * blockDim.x + threadIdx.x; item < w.acc_items; item += gridDim.x * blockDim.x) {
    const WaveGroup& g = w.groups[find_group(w, item, true)];
    const SceneDev& sc = b.scenes[g.scene];
    const uint32_t pix = g.pix0 + (item - g.acc0);
    float4 s = sc.acc_sum[pix], c = sc.acc_comp[pix];
    double* sq = sc.acc_sq + 3ull * pix;
    double q0 = sq[0], q1 = sq[1], q2 = sq[2];
    double m0 = 0, m1 = 0, m2 = 0;
    if (sc.acc_sum64) {
      m0 = sc.acc_sum64[3ull * pix];
      m1 = sc.acc_sum64[3ull * pix + 1];
      m2 = sc.acc_sum64[3ull * pix + 2];
    }
    uint32_t last_slot = 0;
    for (uint32_t m = 0; m < g.nplanes; ++m) {
      const uint32_t slot = g.slot0 + m * g.npix + (pix - g.pix0);
      last_slot = slot;
      const float4 v = b.ps_col[slot];
      // Kahan: y = v - c; t = s + y; c = (t - s) - y; s = t
      float y, t;
      y = fsub(v.x, c.x); t = fadd(s.x, y); c.x = fsub(fsub(t, s.x), y); s.x = t;
      y = fsub(v.y, c.y); t = fadd(s.y, y); c.y = fsub(fsub(t, s.y), y); s.y = t;
      y = fsub(v.z, c.z); t = fadd(s.z, y); c.z = fsub(fsub(t, s.z), y); s.z = t;
      q0 = __dadd_rn(q0, square_as_double(v.x));
      q1 = __dadd_rn(q1, square_as_double(v.y));
      q2 = __dadd_rn(q2, square_as_double(v.z));
      if (sc.acc_sum64) {
        m0 = __dadd_rn(m0, as_double(v.x));
        m1 = __dadd_rn(m1, as_double(v.y));
        m2 = __dadd_rn(m2, as_double(v.z));
      }
    }
    sc.acc_sum[pix] = s;
    sc.acc_comp[pix] = c;
    sq[0] = q0;
    sq[1] = q1;
    sq[2] = q2;
    if (sc.acc_sum64) {
      sc.acc_sum64[3ull * pix] = m0;
      sc.acc_sum64[3ull * pix + 1] = m1;
      sc.acc_sum64[3ull * pix + 2] = m2;
    }
    if (w.rng_mode == LISA_RNG_PER_PIXEL) sc.pix_rng[pix] = b.ps_rng[last_slot];
  }
}

// ---------------------------------------------------------------------------
// guide training samples from the wave's kept records
//
// Each record holds the radiance the path had gathered when the vertex was
// left (c0) and the throughput after its bounce (a1); with the path's final
// radiance c, the radiance that arrived along the sampled direction is
// L = (c - c0) / a1.  The training weight is mean(L) * p_bsdf / q, the
// importance weight of the Neural Importance Sampling loss; records with
// weight 0 carry no gradient and are skipped.  At most `cap` samples go to
// the batch.  The keep probability of the next wave's records is set from
// this wave's guided-vertex count, aiming at 90 % of the record capacity.

__global__ void k_guide_collect(WaveBufs b, float4* __restrict__ batch, uint32_t cap) {
  const uint32_t total = *(volatile uint32_t*)&b.ctrl->guided_count;
  const uint32_t nrec = min(*(volatile uint32_t*)&b.ctrl->rec_count, b.rec_cap);
  const uint32_t stride = gridDim.x * blockDim.x;
  const uint32_t end = (nrec + 31u) & ~31u;
  for (uint32_t k = blockIdx.x * blockDim.x + threadIdx.x; k < end; k += stride) {
    bool want = false;
    float4 r0, r1, r2, r3, r4;
    float wt = 0.0f;
    if (k < nrec) {
      r4 = b.rec_col[k];
      const float4 col = b.ps_col[__float_as_uint(r4.w) >> 1];
      // no channel gained radiance after the vertex: every term below is
      // <= 0 (or not a number), so the record is not wanted -- its other
      // four float4 are not read
      if (col.x > r4.x || col.y > r4.y || col.z > r4.z) {
        const float4* rec = b.rec_list + 4ull * k;
        r0 = rec[0];
        r1 = rec[1];
        r2 = rec[2];
        r3 = rec[3];
        float l = 0.0f;
        int nl = 0;
        if (r3.x > 0.0f) { l += (col.x - r4.x) / r3.x; ++nl; }
        if (r3.y > 0.0f) { l += (col.y - r4.y) / r3.y; ++nl; }
        if (r3.z > 0.0f) { l += (col.z - r4.z) / r3.z; ++nl; }
        wt = nl ? l / (float)nl * r0.w : 0.0f;
        want = wt > 0.0f && isfinite(wt);
      }
    }
    const uint32_t i = warp_reserve(&b.ctrl->train_count, want);
    if (want && i < cap) {
      float4* o = batch + 4ull * i;
      o[0] = make_float4(r0.x, r0.y, r0.z, r1.x);
      o[1] = make_float4(r1.y, r1.z, r2.x, r2.y);
      o[2] = make_float4(r2.z, r1.w, r2.w, r3.w);
      o[3] = make_float4(fminf(wt, 1e4f), (float)(__float_as_uint(r4.w) & 1u), 0.0f, 0.0f);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const float keep = total ? fminf(1.0f, 0.9f * (float)b.rec_cap / (float)total) : 1.0f;
    b.ctrl->drop_prob = 1.0f - keep;
  }
}

__global__ void k_init_pixrng(uint32_t* rng, uint32_t npix, uint32_t subframe) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x)
    rng[p] = tea<16>(p, subframe);  // shader.cu:141
}

// ---------------------------------------------------------------------------
// tone map (src/cuda/helpers.h:35-62) and the PPM payload
// (src/sutil/sutil.cpp:533-553: rows flipped, alpha dropped)

__device__ __forceinline__ unsigned char quantize8(float x) {
  x = clampf(x, 0.0f, 1.0f);
  return (unsigned char)min((unsigned)(x * 256.0f), 255u);
}
__device__ __forceinline__ float to_srgb(float c) {
  const float inv_gamma = 1.0f / 2.4f;
  return c < 0.0031308f ? fmul(12.92f, c) : fsub(fmul(1.055f, powf(c, inv_gamma)), 0.055f);
}

__global__ void k_tonemap(const float4* __restrict__ sum, uint32_t npix, float inv_n, uint32_t width,
                          uint32_t height, float* rgb32, uchar4* rgba8, unsigned char* ppm) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < npix; p += gridDim.x * blockDim.x) {
    const float4 s = sum[p];
    const float r = fmul(s.x, inv_n), g = fmul(s.y, inv_n), bl = fmul(s.z, inv_n);
    if (rgb32) {
      rgb32[3ull * p] = r;
      rgb32[3ull * p + 1] = g;
      rgb32[3ull * p + 2] = bl;
    }
    const unsigned char R = quantize8(to_srgb(clampf(r, 0.0f, 1.0f)));
    const unsigned char G = quantize8(to_srgb(clampf(g, 0.0f, 1.0f)));
    const unsigned char B = quantize8(to_srgb(clampf(bl, 0.0f, 1.0f)));
    if (rgba8) rgba8[p] = make_uchar4(R, G, B, 255);
    if (ppm) {
      const uint32_t x = p % width, y = p / width;
      const uint64_t o = 3ull * ((uint64_t)(height - 1 - y) * width + x);
      ppm[o] = R;
      ppm[o + 1] = G;
      ppm[o + 2] = B;
    }
  }
}

// FP64 mean (of acc_sum64, else the float mean) and sample variance of the
// pixels' samples, one value a thread; each double operation rounds once, as
// the same expressions do on a host without contraction.
//
// Bound by the copies to the host behind it.  Formed on the host from copies
// of the sums, the two images of 333 x 217 pixels took 0.9 ms with the float
// mean; now the call takes 0.3 ms, 30 us of it this kernel's double divisions
// (the GPU has few double units).
__global__ void k_moments(const float4* __restrict__ sum, const double* __restrict__ sum64,
                          const double* __restrict__ sq, uint32_t npix, float inv_n, double n, double* var,
                          double* mean) {
  const uint64_t count = 3ull * npix;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < count; i += gridDim.x * (uint64_t)blockDim.x) {
    const double mu = sum64 ? (n > 0.0 ? __ddiv_rn(sum64[i], n) : 0.0)
                            : (double)fmul(reinterpret_cast<const float*>(sum + i / 3)[i % 3], inv_n);
    if (mean) mean[i] = mu;
    if (var) {
      double v = 0.0;
      if (n > 1.0) v = __ddiv_rn(__dmul_rn(__dsub_rn(__ddiv_rn(sq[i], n), __dmul_rn(mu, mu)), n), n - 1.0);
      var[i] = v > 0.0 ? v : 0.0;
    }
  }
}

// ---------------------------------------------------------------------------
// traversal hooks: closest hit / brute force / counting pass of given rays

// Ray i of `rays` (ox oy oz tmin dx dy dz tmax).  A negative tmax gets the
// margin of a best hit (a positive one needs none: its entry distances are
// rounded down).
__device__ __forceinline__ bool begin_given(TravState& s, const TraceScene& ts, const float* rays, uint32_t i, TriPass& tp) {
  const float* r = rays + 8ull * i;
  const bool active = trav_begin(s, ts, v3(r[0], r[1], r[2]), v3(r[4], r[5], r[6]), r[3], r[7], tp);
  if (r[7] < 0.0f) s.cull = fmaf(-r[7], 1.52587890625e-5f, r[7]);
  return active;
}

template <bool COUNT>
__global__ void __launch_bounds__(128) k_trace_rays(const SceneDev* __restrict__ scd, const float* __restrict__ rays,
                                                   uint32_t n, int32_t* prim, float* tout, WaveCtrl* ctrl) {
  // the same warp-wide traversal step as the wavefront kernels (whole
  // warps run each round: `total` is a multiple of 32, as is the stride)
  uint32_t visits = 0, tests = 0;
  __shared__ TriPass tri_pass[4];
  TriPass& tp = tri_pass[threadIdx.x >> 5];
  uint2 stack[TRAV_STACK];
  const TraceScene ts = trace_scene(*scd);
  const uint32_t total = ((n + 31) / 32) * 32;
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
    TravState s;
    bool active = false;
    if (i < n) active = begin_given(s, ts, rays, i, tp);
    while (__any_sync(FULL, active))
      if (trav_step_warp<COUNT, false, true>(active, s, ts, stack, visits, tests, &ctrl->status, tp)) active = false;
    if (i < n) {
      if (prim) prim[i] = s.best_prim;
      if (tout) tout[i] = s.best_prim >= 0 ? s.best_t : __int_as_float(0x7f800000);
    }
  }
  if (COUNT) {
    warp_add64(&ctrl->node_visits[0], visits);
    warp_add64(&ctrl->tri_tests[0], tests);
  }
}

// The same where warps have one ray each or more than 32: warp w takes rays
// share * w .. + share - 1, a lane the next one once at most RAYS_BUSY lanes
// have one.  (No counter in memory, so calls on several streams stay apart.)
// A call takes as long as its longest rays, and a ray alone in its warp steps
// faster: 1,000 rays of 30,001 triangles, with the build, 411 -> 365 us.  With
// more rays than lanes, a lane need not wait for the longest of its warp's:
// 165,000 rays 603 -> 557 us, 400,000 872 -> 756.  Between, 32 rays a warp and
// no more code in the loop are best (50,003 rays: 447 us, 458 in this kernel,
// 499 spread over all warps).
constexpr int RAYS_BUSY = 24;

template <bool COUNT>
__global__ void __launch_bounds__(128, LISA_TRACE_MIN_BLOCKS) k_trace_rays_shared(const SceneDev* __restrict__ scd,
                                                                           const float* __restrict__ rays, uint32_t n,
                                                                           uint32_t share, int32_t* prim, float* tout,
                                                                           WaveCtrl* ctrl) {
  uint32_t visits = 0, tests = 0;
  __shared__ TriPass tri_pass[4];
  TriPass& tp = tri_pass[threadIdx.x >> 5];
  uint2 stack[TRAV_STACK];
  const TraceScene ts = trace_scene(*scd);
  uint32_t next = (uint32_t)min((uint64_t)n, (uint64_t)share * ((blockIdx.x * blockDim.x + threadIdx.x) >> 5));
  const uint32_t end = next + min(share, n - next);
  TravState s;
  bool active = false;
  uint32_t i = 0;
  auto done = [&]() {
    if (prim) prim[i] = s.best_prim;
    if (tout) tout[i] = s.best_prim >= 0 ? s.best_t : __int_as_float(0x7f800000);
  };
  while (true) {
    const uint32_t idle = __ballot_sync(FULL, !active);
    if (next < end && 32 - __popc(idle) <= RAYS_BUSY) {
      const uint32_t at = next + __popc(idle & lanemask_lt());
      if (!active && at < end) {
        i = at;
        active = begin_given(s, ts, rays, i, tp);
        if (!active) done();
      }
      next = min(end, next + __popc(idle));
    }
    if (!__any_sync(FULL, active)) {
      if (next >= end) break;
      continue;
    }
    if (trav_step_warp<COUNT, false, true>(active, s, ts, stack, visits, tests, &ctrl->status, tp)) {
      active = false;
      done();
    }
  }
  if (COUNT) {
    warp_add64(&ctrl->node_visits[0], visits);
    warp_add64(&ctrl->tri_tests[0], tests);
  }
}

template <bool COUNT>
static void launch_trace_rays(const SceneDev* scd, const float* rays, uint32_t n, int32_t* prim, float* t,
                              WaveCtrl* ctrl, int sm_count, cudaStream_t s) {
  const uint32_t warps = 4u * LISA_TRACE_MIN_BLOCKS * (uint32_t)sm_count;  // resident
  const uint32_t share = (uint32_t)(((uint64_t)n + warps - 1u) / warps);
  if (share == 1u || share > 32u) {
    const uint32_t blocks = (uint32_t)(((uint64_t)n + 4ull * share - 1u) / (4ull * share));
    k_trace_rays_shared<COUNT><<<blocks, 128, 0, s>>>(scd, rays, n, share, prim, t, ctrl);
  } else {
    k_trace_rays<COUNT><<<(n + 127) / 128, 128, 0, s>>>(scd, rays, n, prim, t, ctrl);
  }
}

__global__ void k_brute_rays(const SceneDev* __restrict__ scd, const float* __restrict__ rays, uint32_t n,
                             int32_t* prim, float* tout) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float* r = rays + 8ull * i;
    int hp;
    float ht;
    brute_hit(*scd, v3(r[0], r[1], r[2]), v3(r[4], r[5], r[6]), r[3], r[7], hp, ht);
    prim[i] = hp;
    tout[i] = ht;
  }
}

// ---------------------------------------------------------------------------
// host side

// Plain waves of at most this many paths run whole paths in one kernel
// (k_paths), larger ones stage by stage.  Measured device times, k_paths
// against the stages, by wave size (8 bounces; 12 for the 5,000-sphere soup):
//   reference estimator     64 Ki         1 Mi          4 Mi
//     Cornell box           0.25 / 0.60   1.41 / 1.62   4.99 / 4.90 ms
//     icosphere box, 328 k  0.44 / 1.42   2.46 / 3.26   9.09 / 8.32 ms
//     sphere soup           3.18 / 9.16   9.68 / 16.5   29.8 / 33.4 ms
//   physically based        64 Ki         256 Ki        1 Mi
//     hard indirect, 328 k  0.56 / 1.06   1.20 / 1.38   3.44 / 2.76 ms
// The stages win on large waves by their occupancy (32 warps an SM against
// 20) and by running each routine on full warps; the physically based
// estimator's short searches leave less to win.
constexpr uint32_t PATHS_MAX_WAVE = 1u << 21, PATHS_MAX_WAVE_PB = 1u << 18;

// Host view of one planned wave.
struct WaveLaunch {
  uint32_t bounces;  // depth of its deepest scene
  int scene;         // scene of its first group (the only one of a guided wave)
  bool guided;       // the guide samples this wave's bounces
  bool train;        // guided wave: train the guide after it
  bool warm;         // guided wave: warm-up, sample the BSDF only
  uint32_t steps;    // guided wave: Adam steps after it, in proportion to its paths
  uint32_t items;    // paths, or with one stream per pixel the pixels they run through
  bool whole;        // rendered by k_paths, not stage by stage
};

namespace {

// Guided mode guides the scenes with at least guide_min_spp samples per
// pixel, one scene per wave so one network runs its inference, each wave
// holding at most guide_spp_per_wave planes (or as many as make 1 Mi paths,
// for small images) so the guide trains in between; the other scenes are
// packed into plain waves after them.
bool scene_guided(const Renderer& r, uint32_t s) {
  return r.opts.mode == LISA_MODE_GUIDED && r.scenes[s].params.num_samples >= r.opts.guide_min_spp;
}

void plan_waves(Renderer& r, const std::vector<uint32_t>& spp, const std::vector<uint64_t>& sample_base,
                std::vector<WaveDesc>& waves, std::vector<WaveLaunch>& wave_launch) {
  const uint32_t W = r.capacity;
  const bool per_pixel = r.opts.rng == LISA_RNG_PER_PIXEL;
  const bool may_whole = !r.opts.stage_timing && !r.opts.count_traversal;
  const uint32_t max_whole = r.opts.estimator == LISA_ESTIMATOR_PHYSICAL ? PATHS_MAX_WAVE_PB : PATHS_MAX_WAVE;
  waves.clear();
  wave_launch.clear();
  WaveDesc cur;
  std::memset(&cur, 0, sizeof(cur));
  uint32_t cur_b = 0;
  bool cur_guided = false;
  auto close = [&]() {
    if (cur.num_groups == 0) return;
    cur.rng_mode = r.opts.rng;
    cur.seed = r.opts.seed;
    waves.push_back(cur);
    // guide_steps_per_wave steps per 4 Mi paths, at least one
    const uint32_t steps = cur_guided ? std::min<uint32_t>(r.guide_max_steps, std::max<uint32_t>(
                                            1u, (uint32_t)(((uint64_t)cur.paths * r.opts.guide_steps_per_wave +
                                                            (1ull << 21)) >> 22)))
                                      : 0u;
    const uint32_t items = per_pixel ? cur.acc_items : cur.paths;
    const bool whole = may_whole && !cur_guided && items <= max_whole;
    wave_launch.push_back(WaveLaunch{cur_b, (int)cur.groups[0].scene, cur_guided, false, false, steps, items, whole});
    std::memset(&cur, 0, sizeof(cur));
    cur_b = 0;
  };
  auto add = [&](uint32_t s, uint32_t pix0, uint32_t npix, uint32_t sample0, uint32_t k) {
    WaveGroup& g = cur.groups[cur.num_groups++];
    g.scene = s;
    g.pix0 = pix0;
    g.npix = npix;
    g.sample0 = sample0;
    g.nplanes = k;
    g.slot0 = cur.paths;
    g.acc0 = cur.acc_items;
    cur.paths += k * npix;
    cur.acc_items += npix;
    cur_b = std::max(cur_b, r.scenes[s].params.num_bounces);
  };
  for (int pass = 0; pass < 2; ++pass) {
    const bool one_scene = pass == 0;  // pass 0: guided scenes, pass 1: the rest
    cur_guided = one_scene;
    for (uint32_t s = 0; s < r.scenes.size(); ++s) {
      if (scene_guided(r, s) != one_scene) continue;
      const uint32_t npix = r.scenes[s].npix;
      const uint32_t max_planes =
          one_scene && r.opts.guide_spp_per_wave && npix
              ? std::max<uint32_t>(r.opts.guide_spp_per_wave, ((1u << 20) + npix - 1) / npix)
              : UINT32_MAX;
      uint32_t planes = spp[s];
      uint32_t j = (uint32_t)sample_base[s];
      if (npix == 0 || r.scenes[s].params.num_bounces == 0) continue;
      if (one_scene) close();
      bool scene_in_cur = false;
      // With one stream per pixel a pixel's samples are a chain.  k_paths
      // runs it in one launch, each path of a pixel by the lane that ran the
      // one before; stage by stage each sample is a wave.  (333 x 217 pixels,
      // 8 samples: 1.77 ms, bound by the longest chain -- 640 x 360 pixels
      // take 2.24 -- against 2.10 ms in waves of one sample.)
      const bool chain = per_pixel && may_whole && !one_scene && npix <= max_whole;
      while (planes > 0) {
        if (per_pixel && cur.acc_items && (cur.acc_items > max_whole || npix > max_whole - cur.acc_items)) {
          close();  // chains are k_paths' alone
          scene_in_cur = false;
        }
        const uint32_t room = W - cur.paths;
        if (cur.num_groups == MAX_GROUPS || (per_pixel && scene_in_cur)) {
          close();
          scene_in_cur = false;
          continue;
        }
        if (npix <= room) {
          uint32_t k = std::min(std::min(planes, room / npix), max_planes);
          if (per_pixel && !chain) k = 1;
          add(s, 0, npix, j, k);
          scene_in_cur = true;
          planes -= k;
          j += k;
          if (one_scene) {
            close();
            scene_in_cur = false;
          }
        } else if (cur.paths == 0) {
          for (uint32_t p0 = 0; p0 < npix; p0 += W) {
            add(s, p0, std::min(W, npix - p0), j, 1);
            close();
          }
          planes -= 1;
          j += 1;
          scene_in_cur = false;
        } else {
          close();
          scene_in_cur = false;
        }
      }
    }
    close();
  }
}

// own: REFILL_*, of the kernel the buffers go to (0: it does not traverse)
WaveBufs make_bufs(Renderer& r, uint32_t own = 0) {
  WaveBufs b;
  std::memset(&b, 0, sizeof(b));
  b.ro[0] = r.ro[0];
  b.ro[1] = r.ro[1];
  b.rd[0] = r.rd[0];
  b.rd[1] = r.rd[1];
  b.hit = r.hit;
  b.ps_att = r.ps_att;
  b.ps_col = r.ps_col;
  b.ps_rng = r.ps_rng;
  b.nee_a = r.nee_a;
  b.nee_b = r.nee_b;
  b.nee_c = r.nee_c;
  b.ctrl = r.ctrl;
  b.scenes = r.d_scenes;
  b.capacity = r.capacity;
  b.refill_busy_max = 32u - refill_idle_lanes(r.opts.refill_idle, own);
  b.physical = r.opts.estimator == LISA_ESTIMATOR_PHYSICAL;
  b.rec_list = r.rec_list;
  b.rec_col = r.rec_list ? r.rec_list + 4ull * r.rec_cap : nullptr;
  b.rec_cap = r.rec_cap;
  b.nee_light = r.nee_light;
  b.bsdf_fraction = r.opts.guide_bsdf_fraction;
  return b;
}

struct StageTimer {
  Renderer& r;
  bool on;
  bool capturing = false;  // inside stream capture: record external event nodes
  size_t next = 0;
  std::vector<std::pair<int, std::pair<size_t, size_t>>> marks;  // stage, (start ev, end ev)
  explicit StageTimer(Renderer& rr, bool enable) : r(rr), on(enable) {}
  Status ev(size_t* idx) {
    if (next >= r.ev_pool.size()) {
      cudaEvent_t e;
      LISA_CUDA(cudaEventCreate(&e));
      r.ev_pool.push_back(e);
    }
    *idx = next++;
    if (capturing)
      LISA_CUDA(cudaEventRecordWithFlags(r.ev_pool[*idx], r.stream, cudaEventRecordExternal));
    else
      LISA_CUDA(cudaEventRecord(r.ev_pool[*idx], r.stream));
    return Status();
  }
};

}  // namespace

// Dynamic shared memory of the fused inference kernels.
Status guided_infer_setup() {
  LISA_CUDA(cudaFuncSetAttribute(k_guided_infer<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, INFER_SMEM));
  LISA_CUDA(cudaFuncSetAttribute(k_guided_infer<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, INFER_SMEM));
  return Status();
}

Status guide_collect(Renderer& r, int, uint32_t cap, cudaStream_t s) {
  WaveBufs b = make_bufs(r);
  k_guide_collect<<<r.sm_count * 8, 256, 0, s>>>(b, r.guide_batch, cap);
  LISA_CUDA(cudaGetLastError());
  return Status();
}

// Stage indices of the timer: 0 trace, 2 shading and emitter search, 3 other,
// 4 guide inference, 5 guide training (sample collection, training, Adam).
Status launch_wave_sequence(Renderer& r, const std::vector<WaveLaunch>& waves, lisa_render_stats* st,
                            StageTimer* tm) {
  WaveBufs b = make_bufs(r);
  uint32_t launches[5] = {0, 0, 0, 0, 0};  // trace, -, nee, guide, total
  auto stage = [&](int which, auto&& fn) -> Status {
    size_t e0 = 0, e1 = 0;
    if (tm && tm->on) LISA_TRY(tm->ev(&e0));
    LISA_TRY(fn());
    LISA_CUDA(cudaGetLastError());
    if (tm && tm->on) {
      LISA_TRY(tm->ev(&e1));
      tm->marks.push_back({which, {e0, e1}});
    }
    if (which < 3) launches[which]++;
    if (which == 4 || which == 5) launches[3]++;
    launches[4]++;
    return Status();
  };
  const int acc_blocks = r.sm_count * 8;
  const bool counting = r.opts.count_traversal != 0;
  const bool guided_mode = r.opts.mode == LISA_MODE_GUIDED;
  const bool physical = r.opts.estimator == LISA_ESTIMATOR_PHYSICAL;
  for (size_t wv = 0; wv < waves.size(); ++wv) {
    const WaveDesc* wd = r.d_waves + wv;
    GuideSrc infer_src, train_src;
    GuideNet* net = nullptr;
    const bool guided = guided_mode && waves[wv].guided;
    if (guided) {
      const SceneGpu& sg = r.scenes[waves[wv].scene];
      net = r.guides[sg.guide].get();
      std::memset(&infer_src, 0, sizeof(infer_src));
      infer_src.nee_a = r.nee_a;
      infer_src.nee_b = r.nee_b;
      infer_src.nee_c = r.nee_c;
      infer_src.ps_att = r.ps_att;
      infer_src.count = &r.ctrl->nee_count;
      infer_src.n = r.capacity;
      infer_src.no_flag = physical ? 1u : 0u;
      for (int k = 0; k < 3; ++k) {
        infer_src.bmin[k] = sg.bvh.bmin[k];
        infer_src.bmax[k] = sg.bvh.bmax[k];
      }
      train_src = infer_src;
      train_src.nee_a = train_src.nee_b = train_src.nee_c = nullptr;
      train_src.geom = r.guide_batch;
      train_src.count = &r.ctrl->train_count;
      train_src.n = r.guide_batch_cap;
    }
    if (waves[wv].whole) {
      // All resident warps share a wave of up to ten paths each: it takes as
      // long as its longest path, and a warp of few paths steps that one faster.  (160 x 90 paths over 20 warps an SM against
      // eight: Cornell box 112 / 132 us, icosphere box 207 / 230, hard
      // indirect 273 / 315.)  Then warps of 32, at least eight an SM: with
      // more paths the warps' own bookkeeping weighs more (250 x 150 paths
      // over 20 warps an SM against eight: 281 / 275 and 380 / 370).
      const uint32_t wpb = (uint32_t)r.nee_threads / 32u, items = waves[wv].items;
      const uint32_t all = (uint32_t)r.path_blocks, few = (uint32_t)r.sm_count * ((8u + wpb - 1u) / wpb);
      const uint32_t grid = items <= 10u * wpb * all
                                ? all
                                : std::min(all, std::max(few, (items + 32u * wpb - 1u) / (32u * wpb)));
      const uint32_t lanes = std::min<uint32_t>(32u, (items + grid * wpb - 1u) / (grid * wpb));
      LISA_TRY(stage(0, [&] {
        const WaveBufs bp = make_bufs(r, REFILL_PATHS);
        const bool chains = r.opts.rng == LISA_RNG_PER_PIXEL;
        auto* kernel = physical ? (chains ? k_paths<true, true> : k_paths<true, false>)
                                : (chains ? k_paths<false, true> : k_paths<false, false>);
        kernel<<<grid, r.nee_threads, 0, r.stream>>>(bp, wd, lanes);
        return Status();
      }));
      LISA_TRY(stage(3, [&] {
        k_accumulate<<<acc_blocks, 256, 0, r.stream>>>(b, wd);
        return Status();
      }));
      continue;
    }
    LISA_TRY(stage(3, [&] {
      k_raygen<<<r.sm_count * 8, 256, 0, r.stream>>>(b, wd);
      return Status();
    }));
    // the physically based estimator traces one more ray per path, the one
    // leaving its last vertex, for the emission it reaches (no vertex)
    const uint32_t depths = waves[wv].bounces + (physical ? 1u : 0u);
    for (uint32_t d = 0; d < depths; ++d) {
      LISA_TRY(stage(0, [&] {
        const WaveBufs b = make_bufs(r, REFILL_TRACE);
        if (counting) k_trace<true><<<r.trace_blocks, r.trace_threads, 0, r.stream>>>(b, (int)d);
        else k_trace<false><<<r.trace_blocks, r.trace_threads, 0, r.stream>>>(b, (int)d);
        return Status();
      }));
      // the guide draws the bounces of the first guide_max_depth vertices
      // of a path (0 = all); deeper ones sample the BSDF (and, with the
      // reference estimator, never the last one, whose bounce is not traced)
      const bool guided_d = guided && (physical ? d < waves[wv].bounces : d + 1 < waves[wv].bounces) &&
                            (r.opts.guide_max_depth == 0 || d < r.opts.guide_max_depth);
      LISA_TRY(stage(2, [&] {
        const dim3 g(physical ? r.nee_pb_blocks : r.nee_blocks), t(r.nee_threads);
        const WaveBufs b = make_bufs(r, REFILL_NEE);
        if (physical) {
          if (guided_d) {
            if (counting) k_nee_pb<true, true><<<g, t, 0, r.stream>>>(b, (int)d);
            else k_nee_pb<false, true><<<g, t, 0, r.stream>>>(b, (int)d);
          } else {
            if (counting) k_nee_pb<true, false><<<g, t, 0, r.stream>>>(b, (int)d);
            else k_nee_pb<false, false><<<g, t, 0, r.stream>>>(b, (int)d);
          }
        } else if (guided_d) {
          if (counting) k_nee<true, true><<<g, t, 0, r.stream>>>(b, (int)d);
          else k_nee<false, true><<<g, t, 0, r.stream>>>(b, (int)d);
        } else {
          if (counting) k_nee<true><<<g, t, 0, r.stream>>>(b, (int)d);
          else k_nee<false><<<g, t, 0, r.stream>>>(b, (int)d);
        }
        return Status();
      }));
      if (guided_d) {
        LISA_TRY(stage(4, [&] {
          WaveBufs bw = b;  // warm-up waves sample the BSDF only (c = 1)
          if (waves[wv].warm) bw.bsdf_fraction = 1.0f;
          bw.rec_salt = (uint32_t)(r.guide_waves_done + wv) * 2654435761u + 17u;
          if (!waves[wv].train) bw.rec_cap = 0;
          const uint32_t grid = std::min<uint32_t>((r.capacity + 255) / 256, (uint32_t)(r.sm_count * INFER_BLOCKS_PER_SM));
          if (bw.bsdf_fraction == 1.0f) {
            const uint32_t g = std::min<uint32_t>((r.capacity + 255) / 256, (uint32_t)(r.sm_count * BOUNCE_BLOCKS_PER_SM));
            if (physical) k_bsdf_bounce<true><<<g, 256, 0, r.stream>>>(bw, (int)d);
            else k_bsdf_bounce<false><<<g, 256, 0, r.stream>>>(bw, (int)d);
          } else if (physical)
            k_guided_infer<true><<<grid, INFER_THREADS, INFER_SMEM, r.stream>>>(net->w_bf16, net->master, infer_src, net->status,
                                                                       bw, (int)d);
          else
            k_guided_infer<false><<<grid, INFER_THREADS, INFER_SMEM, r.stream>>>(net->w_bf16, net->master, infer_src, net->status,
                                                                        bw, (int)d);
          return Status();
        }));
      }
    }
    LISA_TRY(stage(3, [&] {
      k_accumulate<<<acc_blocks, 256, 0, r.stream>>>(b, wd);
      return Status();
    }));
    if (guided && waves[wv].train) {
      const uint32_t steps = waves[wv].steps;
      LISA_TRY(stage(5, [&] { return guide_collect(r, (int)wv, steps * r.guide_chunk, r.stream); }));
      // one Adam step per slice of the collected samples, all in one
      // cooperative launch
      LISA_TRY(stage(5, [&] {
        return guide_launch_train_rounds(*net, train_src, SRC_GEOM, r.guide_chunk, steps, r.opts.guide_lr, r.guide_grid_bar,
                                         r.stream, &r.ctrl->train_samples);
      }));
    }
  }
  if (st) {
    st->launches_trace += launches[0];
    st->launches_nee += launches[2];
    st->launches_guide += launches[3];
    st->launches_total += launches[4];
  }
  return Status();
}

Status renderer_render(Renderer& r, uint32_t spp_req, bool progressive, lisa_render_stats* st) {
  lisa_render_stats local;
  std::memset(&local, 0, sizeof(local));
  std::vector<uint32_t> spp(r.scenes.size());
  std::vector<uint64_t> base(r.scenes.size());
  for (size_t s = 0; s < r.scenes.size(); ++s) {
    spp[s] = progressive ? spp_req : r.scenes[s].params.num_samples;
    base[s] = r.scenes[s].next_sample;
  }
  std::vector<WaveDesc> waves;
  std::vector<WaveLaunch> wb;
  plan_waves(r, spp, base, waves, wb);
  const bool guided = r.opts.mode == LISA_MODE_GUIDED;
  // warm-up and training flags count the guided waves of each scene (its
  // guide); a scene's Adam steps stop at guide_train_steps
  std::vector<uint64_t> scene_waves(r.scenes.size(), 0), scene_steps(r.scenes.size(), 0);
  if (guided)
    for (size_t i = 0; i < wb.size(); ++i) {
      if (!wb[i].guided) continue;
      const int sc = wb[i].scene;
      const uint64_t k = r.scenes[sc].guide_waves_done + scene_waves[sc]++;
      const uint64_t done = r.scenes[sc].guide_steps_done + scene_steps[sc];
      if (r.opts.guide_train_steps)
        wb[i].steps = (uint32_t)std::min<uint64_t>(wb[i].steps, done < r.opts.guide_train_steps
                                                                    ? r.opts.guide_train_steps - done
                                                                    : 0);
      wb[i].train = (r.opts.guide_train_waves == 0 || k < r.opts.guide_train_waves) && wb[i].steps > 0;
      if (!wb[i].train) wb[i].steps = 0;
      scene_steps[sc] += wb[i].steps;
      wb[i].warm = k < r.opts.guide_warmup_waves;
    }
  if (waves.size() > r.wave_capacity) {
    if (r.d_waves) cudaFree(r.d_waves);
    r.d_waves = nullptr;
    LISA_CUDA(cudaMalloc(&r.d_waves, sizeof(WaveDesc) * waves.size()));
    r.wave_capacity = (uint32_t)waves.size();
  }
  if (!waves.empty())
    LISA_CUDA(cudaMemcpyAsync(r.d_waves, waves.data(), sizeof(WaveDesc) * waves.size(), cudaMemcpyHostToDevice,
                              r.stream));
  // reset ray counters
  LISA_CUDA(cudaMemsetAsync(r.ctrl, 0, sizeof(WaveCtrl), r.stream));
  if (r.opts.rng == LISA_RNG_PER_PIXEL) {
    for (auto& s : r.scenes) {
      const uint32_t subframe = progressive ? s.subframe : 0u;
      k_init_pixrng<<<r.sm_count * 4, 256, 0, r.stream>>>(s.pix_rng, s.npix, subframe);
    }
    LISA_CUDA(cudaGetLastError());
  }
  cudaEvent_t e0, e1;
  LISA_CUDA(cudaEventCreate(&e0));
  LISA_CUDA(cudaEventCreate(&e1));
  LISA_CUDA(cudaEventRecord(e0, r.stream));
  StageTimer tm(r, r.opts.stage_timing != 0);
  Status s;
  if (r.opts.use_graph && !wb.empty()) {
    // one graph per launch-sequence shape; the wave table it reads is
    // refreshed above, outside the graph
    std::vector<uint64_t> key;
    for (const WaveLaunch& w : wb) {
      key.push_back(w.whole ? w.items : 0u);  // (its launch shape)
      key.push_back(((uint64_t)w.steps << 40) | ((uint64_t)w.bounces << 32) | ((uint64_t)w.scene << 3) |
                    ((uint64_t)w.guided << 2) | ((uint64_t)w.warm << 1) | w.train);
    }
    key.push_back(r.opts.count_traversal);
    key.push_back(r.opts.stage_timing);
    key.push_back((uint64_t)(uintptr_t)r.d_waves);
    if (key != r.graph_key || !r.graph_exec) {
      if (tm.on) {  // create the timing events before capture begins
        size_t need = 0;
        for (const WaveLaunch& w : wb) need += 2ull * (5ull * (w.bounces + 1) + 6 + 2ull * w.steps);
        while (r.ev_pool.size() < need) {
          cudaEvent_t e;
          LISA_CUDA(cudaEventCreate(&e));
          r.ev_pool.push_back(e);
        }
      }
      if (r.graph_exec) cudaGraphExecDestroy(r.graph_exec);
      r.graph_exec = nullptr;
      r.graph_key.clear();
      cudaGraph_t g = nullptr;
      LISA_CUDA(cudaStreamBeginCapture(r.stream, cudaStreamCaptureModeThreadLocal));
      lisa_render_stats counts;
      std::memset(&counts, 0, sizeof(counts));
      tm.capturing = true;
      s = launch_wave_sequence(r, wb, &counts, &tm);
      tm.capturing = false;
      const cudaError_t ce = cudaStreamEndCapture(r.stream, &g);
      if (s.ok() && ce != cudaSuccess) s = Status::cuda(ce, "cudaStreamEndCapture");
      if (s.ok()) {
        const cudaError_t ie = cudaGraphInstantiate(&r.graph_exec, g, 0);
        if (ie != cudaSuccess) s = Status::cuda(ie, "cudaGraphInstantiate");
      }
      if (g) cudaGraphDestroy(g);
      if (s.ok()) {
        r.graph_key = key;
        r.graph_marks = tm.marks;
        r.graph_launches[0] = counts.launches_trace;
        r.graph_launches[2] = counts.launches_nee;
        r.graph_launches[3] = counts.launches_total;
        r.graph_launches[4] = counts.launches_guide;
      }
    }
    if (s.ok()) {
      tm.marks = r.graph_marks;
      local.launches_trace = r.graph_launches[0];
      local.launches_nee = r.graph_launches[2];
      local.launches_total = r.graph_launches[3];
      local.launches_guide = r.graph_launches[4];
      const cudaError_t le = cudaGraphLaunch(r.graph_exec, r.stream);
      if (le != cudaSuccess) s = Status::cuda(le, "cudaGraphLaunch");
    }
  } else {
    s = launch_wave_sequence(r, wb, &local, &tm);
  }
  LISA_CUDA(cudaEventRecord(e1, r.stream));
  if (!s.ok()) {
    cudaStreamSynchronize(r.stream);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return s;
  }
  WaveCtrl hc;
  LISA_CUDA(cudaMemcpyAsync(&hc, r.ctrl, sizeof(hc), cudaMemcpyDeviceToHost, r.stream));
  LISA_CUDA(cudaStreamSynchronize(r.stream));
  float ms = 0.0f;
  LISA_CUDA(cudaEventElapsedTime(&ms, e0, e1));
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (tm.on) {
    for (auto& m : tm.marks) {
      float t = 0.0f;
      LISA_CUDA(cudaEventElapsedTime(&t, r.ev_pool[m.second.first], r.ev_pool[m.second.second]));
      if (m.first == 0) local.ms_trace += t;
      else if (m.first == 2) local.ms_nee += t;
      else if (m.first == 4) {
        local.ms_guide += t;
        local.ms_guide_infer += t;
      } else if (m.first == 5) {
        local.ms_guide += t;
        local.ms_guide_train += t;
      }
      else local.ms_other += t;
    }
  }
  for (size_t k = 0; k < r.scenes.size(); ++k) {
    r.scenes[k].samples_done += spp[k];
    r.scenes[k].next_sample += spp[k];
    if (progressive) r.scenes[k].subframe++;
  }
  if (guided) {
    r.guide_waves_done += wb.size();
    for (size_t k = 0; k < r.scenes.size(); ++k) {
      r.scenes[k].guide_waves_done += scene_waves[k];
      r.scenes[k].guide_steps_done += scene_steps[k];
    }
    for (auto& g : r.guides) LISA_TRY(guide_check_status(*g, r.stream));
    for (size_t k = wb.size(); k-- > 0;) {
      if (!wb[k].guided) continue;
      float l = 0.0f;  // loss of the last guided wave's scene
      LISA_CUDA(cudaMemcpy(&l, r.guides[r.scenes[wb[k].scene].guide]->loss_last, sizeof(float),
                           cudaMemcpyDeviceToHost));
      local.guide_loss = l;
      break;
    }
  }
  local.rays_primary = hc.rays_primary;
  local.rays_bounce = hc.rays_bounce;
  local.rays_shadow = hc.rays_shadow;
  local.paths = hc.rays_primary;
  local.samples_total = r.scenes.empty() ? 0 : r.scenes[0].samples_done;
  local.ms_device = ms;
  local.device_status = hc.status;
  local.nee_vertices = hc.nee_total;
  local.node_visits_trace = hc.node_visits[0];
  local.tri_tests_trace = hc.tri_tests[0];
  local.node_visits_nee = hc.node_visits[1];
  local.tri_tests_nee = hc.tri_tests[1];
  local.shadow_traversals = hc.shadow_walked;
  local.guide_infer_rows = hc.infer_rows;
  local.guide_train_samples = hc.train_samples;
  if (st) *st = local;
  if (hc.status) return Status(LISA_ERR_DEVICE, "device status word " + std::to_string(hc.status));
  return Status();
}

Status renderer_reset(Renderer& r) {
  for (auto& s : r.scenes) {
    LISA_CUDA(cudaMemsetAsync(s.acc_sum, 0, sizeof(float4) * s.npix, r.stream));
    LISA_CUDA(cudaMemsetAsync(s.acc_comp, 0, sizeof(float4) * s.npix, r.stream));
    LISA_CUDA(cudaMemsetAsync(s.acc_sq, 0, sizeof(double) * 3 * s.npix, r.stream));
    if (s.acc_sum64) LISA_CUDA(cudaMemsetAsync(s.acc_sum64, 0, sizeof(double) * 3 * s.npix, r.stream));
    s.samples_done = 0;
    s.next_sample = s.sample_offset;
    s.subframe = 0;
  }
  LISA_CUDA(cudaStreamSynchronize(r.stream));
  return Status();
}

Status renderer_get_image(Renderer& r, int scene, float* rgb32, uint8_t* rgba8, double* var, double* mean64) {
  if (scene < 0 || scene >= (int)r.scenes.size()) return Status::invalid("scene index out of range");
  SceneGpu& s = r.scenes[scene];
  const uint32_t npix = s.npix;
  if (npix == 0) return Status();
  const double n = (double)s.samples_done;
  TempDeviceBufs tmp;  // (waits for the stream before the blocks are reused)
  tmp.stream = r.stream;
  float* d_rgb = nullptr;
  uchar4* d_rgba = nullptr;
  double *d_var = nullptr, *d_mean = nullptr;
  const char* w = "image";
  if (rgb32) LISA_TRY(tmp.get((void**)&d_rgb, sizeof(float) * 3ull * npix, w));
  if (rgba8) LISA_TRY(tmp.get((void**)&d_rgba, sizeof(uchar4) * (size_t)npix, w));
  if (var) LISA_TRY(tmp.get((void**)&d_var, sizeof(double) * 3ull * npix, w));
  if (mean64) LISA_TRY(tmp.get((void**)&d_mean, sizeof(double) * 3ull * npix, w));
  const float inv_n = n > 0 ? (float)(1.0 / n) : 0.0f;
  const int blocks = r.sm_count * 4;
  // The mean is the float Kahan sum over n (mean of the samples); rgb32 row 0
  // is the bottom row like the reference accum_buffer.
  if (d_rgb || d_rgba)
    k_tonemap<<<blocks, 256, 0, r.stream>>>(s.acc_sum, npix, inv_n, s.params.width, s.params.height, d_rgb, d_rgba,
                                            nullptr);
  if (d_var || d_mean)
    k_moments<<<blocks, 256, 0, r.stream>>>(s.acc_sum, s.acc_sum64, s.acc_sq, npix, inv_n, n, d_var, d_mean);
  LISA_CUDA(cudaGetLastError());
  if (rgb32) LISA_CUDA(cudaMemcpyAsync(rgb32, d_rgb, sizeof(float) * 3ull * npix, cudaMemcpyDeviceToHost, r.stream));
  if (rgba8)
    LISA_CUDA(cudaMemcpyAsync(rgba8, d_rgba, sizeof(uchar4) * (size_t)npix, cudaMemcpyDeviceToHost, r.stream));
  if (var) LISA_CUDA(cudaMemcpyAsync(var, d_var, sizeof(double) * 3ull * npix, cudaMemcpyDeviceToHost, r.stream));
  if (mean64)
    LISA_CUDA(cudaMemcpyAsync(mean64, d_mean, sizeof(double) * 3ull * npix, cudaMemcpyDeviceToHost, r.stream));
  LISA_CUDA(cudaStreamSynchronize(r.stream));
  return Status();
}

Status renderer_get_ppm(Renderer& r, int scene, uint8_t* rgb8) {
  if (scene < 0 || scene >= (int)r.scenes.size()) return Status::invalid("scene index out of range");
  SceneGpu& s = r.scenes[scene];
  const uint32_t npix = s.npix;
  if (npix == 0) return Status();
  unsigned char* d = nullptr;
  LISA_CUDA(dev_alloc((void**)&d, 3ull * npix));
  const float inv_n = s.samples_done > 0 ? (float)(1.0 / (double)s.samples_done) : 0.0f;
  k_tonemap<<<r.sm_count * 4, 256, 0, r.stream>>>(s.acc_sum, npix, inv_n, s.params.width, s.params.height, nullptr,
                                                   nullptr, d);
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(rgb8, d, 3ull * npix, cudaMemcpyDeviceToHost, r.stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(r.stream);
  else cudaStreamSynchronize(r.stream);
  dev_free(d);
  if (e != cudaSuccess) return Status::cuda(e, "ppm payload");
  return Status();
}

Status launch_trace_closest(const SceneDev* d_scene, WaveCtrl* d_ctrl, const float* d_rays, uint32_t n,
                            int32_t* d_prim, float* d_t, cudaStream_t s, int sm_count, bool brute, bool cleared) {
  if (n == 0) return Status();
  if (!cleared) LISA_CUDA(cudaMemsetAsync(d_ctrl, 0, sizeof(WaveCtrl), s));
  if (brute) {
    const uint32_t blocks = std::min<uint32_t>((n + 127) / 128, (uint32_t)sm_count * 16);
    k_brute_rays<<<blocks, 128, 0, s>>>(d_scene, d_rays, n, d_prim, d_t);
  } else {
    launch_trace_rays<false>(d_scene, d_rays, n, d_prim, d_t, d_ctrl, sm_count, s);
  }
  LISA_CUDA(cudaGetLastError());
  uint32_t status = 0;
  LISA_CUDA(cudaMemcpyAsync(&status, &d_ctrl->status, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
  LISA_CUDA(cudaStreamSynchronize(s));
  if (status) return Status(LISA_ERR_DEVICE, "device status word " + std::to_string(status));
  return Status();
}

Status trace_rays(Renderer& r, const float* d_rays, uint32_t n, int32_t* d_prim, float* d_t, cudaStream_t s,
                  bool brute) {
  if (r.scenes.empty()) return Status::invalid("renderer has no scene");
  return launch_trace_closest(r.d_scenes, r.ctrl, d_rays, n, d_prim, d_t, s, r.sm_count, brute);
}

Status trace_count(Renderer& r, const float* d_rays, uint32_t n, uint64_t* visits, uint64_t* tests) {
  LISA_CUDA(cudaMemsetAsync(r.ctrl, 0, sizeof(WaveCtrl), r.stream));
  if (n) launch_trace_rays<true>(r.d_scenes, d_rays, n, nullptr, nullptr, r.ctrl, r.sm_count, r.stream);
  LISA_CUDA(cudaGetLastError());
  WaveCtrl hc;
  LISA_CUDA(cudaMemcpyAsync(&hc, r.ctrl, sizeof(hc), cudaMemcpyDeviceToHost, r.stream));
  LISA_CUDA(cudaStreamSynchronize(r.stream));
  *visits = hc.node_visits[0];
  *tests = hc.tri_tests[0];
  return Status();
}

Status configure_launch(Renderer& r) {
  int occ = 0;
  const int tthreads = r.opts.threads_per_block ? (int)r.opts.threads_per_block : 128;
  LISA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_trace<false>, tthreads, 0));
  int bps = r.opts.blocks_per_sm ? (int)r.opts.blocks_per_sm : std::max(occ, 1);
  bps = std::min(bps, std::max(occ, 1));
  r.trace_threads = tthreads;
  r.trace_blocks = r.sm_count * bps;
  LISA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_nee<false>, tthreads, 0));
  bps = r.opts.blocks_per_sm ? (int)r.opts.blocks_per_sm : std::max(occ, 1);
  bps = std::min(bps, std::max(occ, 1));
  r.nee_threads = tthreads;
  r.nee_blocks = r.sm_count * bps;
  // the physically based emitter kernel has its own register budget
  LISA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_nee_pb<false, false>, tthreads, 0));
  bps = r.opts.blocks_per_sm ? (int)r.opts.blocks_per_sm : std::max(occ, 1);
  bps = std::min(bps, std::max(occ, 1));
  r.nee_pb_blocks = r.sm_count * bps;
  LISA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_paths<false, false>, tthreads, 0));
  bps = r.opts.blocks_per_sm ? (int)r.opts.blocks_per_sm : std::max(occ, 1);
  r.path_blocks = r.sm_count * std::min(bps, std::max(occ, 1));
  return Status();
}

}  // namespace lisa
