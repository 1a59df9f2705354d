// wavefront.cuh — the renderer's wavefront kernels (device code shared by the
// single-render entry points, render.cu, and the batched renderer, batch.cu).
//
// Paths occupy path slots.  Each step runs three persistent kernels over
// device-side queues: k_extend (closest hit), k_shade (emits shadow rays and the
// continuation ray into queues whose slots are reserved once per warp: a ballot
// and one atomicAdd by the first lane that wants a slot),
// k_shadow (any hit, adds unoccluded contributions).  Queue lengths live in device
// memory.  Paths run in waves (a fixed sequence of launches with no host
// synchronisation, capturable in a CUDA graph), or, with Params::regen_total set,
// a shading step that ends a path starts the next camera path in its slot
// (regenerate).  Kernels are templated on the block size (the traversal stack in
// shared memory is laid out [level][thread]).
//
// Batches: with Params::jobs set, a path carries its job index in meta.w >> 8 and
// the job supplies the camera, the material table offset, the random seed, the
// depth limit and the output pixel base (JobDev).
#pragma once
#include <cuda_fp16.h>

#include <algorithm>

#include "ckr_internal.h"
#include "ltc_table.h"
#include "render_device.cuh"
#include "scene.h"

namespace ckr {
namespace {

constexpr uint32_t kCtrDim = 1024;  // counter dims per (sample, vertex)
constexpr uint32_t kDimBrdf = 1000, kDimRR = 1003, kDimTrain = 1010;
constexpr uint32_t kNoRec = 0xFFFFFFFFu;

// Hooks of the learned light selection (CKR_SHADER_PATH_NEE with a proposal
// network); all null for selection in proportion to power.
struct Learn {
  const uint16_t *sel;       // [queue row x 64] selection CDFs at this bounce's vertices
  const uint16_t *sel_prev;  // the same at the previous bounce (rows by Paths::prev_row)
  float4 *rec;               // training records, 3 float4 each: (x, alpha), (n, value), (wo, cluster)
  uint32_t *rec_count;
  uint32_t rec_cap;
};

__device__ __forceinline__ uint32_t ctr(uint32_t sample, uint32_t depth, uint32_t dim) {
  return ((sample * 64u + depth) * kCtrDim) + dim;
}

// Reference camera (src/main.cpp:77) with the fixed sub-pixel offsets of
// src/main.cpp:23-24 for the first eight samples.
__constant__ float c_jx[8] = {0.34f, 0.86f, 0.20f, 0.86f, 0.66f, 0.34f, 0.20f, 0.66f};
__constant__ float c_jy[8] = {0.20f, 0.66f, 0.66f, 0.34f, 0.86f, 0.86f, 0.34f, 0.20f};

struct Cam {
  F3 pos, dir, cx, cy;
  uint32_t w, h;
};

struct Paths {
  float4 *ray_o;   // ox oy oz tmin
  float4 *ray_d;   // dx dy dz tmax
  float4 *beta;    // throughput rgb, MIS weight of the BRDF sample that made the ray
  uint4 *meta;     // out-pixel index, sample, depth, flags (1 = emission only)
  uint32_t *hit_id;
  float *hit_t;
  uint32_t *q0, *q1;  // path-slot queues
  float4 *sh_o, *sh_d, *sh_c;  // shadow rays and their contributions
  uint32_t *sh_px;
  uint32_t *prev_row;  // learned selection: the path's row in the previous bounce's probabilities
  uint32_t *sh_rec;    // training: per shadow ray, its training record (kNoRec: none)
  // [0] q[0] length, [1] q[1] length, [2] shadow count, [3] [4] work counters of k_extend
  // and k_shadow, [5] next camera path to start, [6] rows that the shading kernel took.  A
  // step's kernels clear them for each other, in launch order: k_camera and the shading
  // kernel [3], k_extend what the shading kernel and k_shadow fill (a memset node costs 3 us of a captured step, a memset 1 us).
  uint32_t *counts;
  unsigned long long *stats;  // cumulative closest-hit rays, shadow rays
  double *accum;     // 3 per output pixel
  uint32_t sh_cap;   // shadow-queue capacity (rays)
  int *status;       // the scene's device status word (first CKR_ERR_*)
};

// One job of a batched render: its paths are the global path indices
// [path_begin, path_begin + npix * spp), its pixels the accumulation rows
// [accum_off, accum_off + npix), its materials sv.mats[mat_off ...].
struct JobDev {
  Cam cam;
  uint64_t path_begin;
  uint64_t seed;
  uint32_t npix, spp, max_depth, mat_off, accum_off;
  double inv_spp;  // 1.0 / spp
  float *rgb;      // output, npix x 3
};

struct Params {
  uint32_t shader, spp, max_depth, n_light, n_brdf;
  float rr_prob;
  uint64_t seed;
  uint32_t npix;
  uint32_t shadow_per_path;
  const JobDev *jobs;  // batched render (nullptr: one render described by the fields above)
  uint32_t njobs;
  // Path regeneration (single render): a shading kernel that ends a path starts
  // camera path P.counts[5]++ in its slot while that index is below regen_total
  // (0: off); cam is the camera of those paths.
  uint32_t regen_total;
  Cam cam;
  // Caller rays (ckr_shade_rays): path g traces ray g % npix (two float4 per ray)
  // as sample g / npix, keyed and accumulated as output row g % npix; nullptr:
  // camera rays.
  const float4 *rays;
};

// Per-path values that a batch takes from the path's job.
struct PathCtx {
  uint64_t seed;
  uint32_t max_depth, px_base, mat_off;
};

__device__ __forceinline__ PathCtx path_ctx(const Params &prm, uint32_t flags) {
  PathCtx c;
  if (prm.jobs) {
    const JobDev &J = prm.jobs[flags >> 8];
    c.seed = J.seed;
    c.max_depth = J.max_depth;
    c.px_base = J.accum_off;
    c.mat_off = J.mat_off;
  } else {
    c.seed = prm.seed;
    c.max_depth = prm.max_depth;
    c.px_base = 0;
    c.mat_off = 0;
  }
  return c;
}

// Job of global path index g (jobs sorted by path_begin).
__device__ __forceinline__ uint32_t job_of(const JobDev *jobs, uint32_t njobs, uint64_t g) {
  uint32_t lo = 0, hi = njobs - 1;
  while (lo < hi) {
    uint32_t mid = (lo + hi + 1) >> 1;
    if (jobs[mid].path_begin <= g) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// One slot of a queue for each lane that wants one; all 32 lanes must call.
__device__ __forceinline__ uint32_t ballot_reserve(uint32_t *counter, bool want) {
  const unsigned m = __ballot_sync(0xffffffffu, want);
  if (m == 0) return 0;
  const uint32_t lane = threadIdx.x & 31u, leader = __ffs(m) - 1;
  uint32_t base = 0;
  if (lane == leader) base = atomicAdd(counter, (uint32_t)__popc(m));
  return __shfl_sync(0xffffffffu, base, leader) + __popc(m & ((1u << lane) - 1u));
}

// Appends one shadow ray for each lane that wants one; all 32 lanes must call.  Rays
// past the queue's capacity are dropped and the status word records
// CKR_ERR_QUEUE_OVERFLOW (the host sizes the queue so that this cannot happen; the
// check keeps a wrong size from writing out of bounds).
__device__ __forceinline__ void emit_shadow(const Paths &P, bool want, F3 o, float4 d, F3 contrib, uint32_t px) {
  const uint32_t at = ballot_reserve(&P.counts[2], want);
  if (!want) return;
  if (at >= P.sh_cap) {
    atomicCAS(P.status, 0, CKR_ERR_QUEUE_OVERFLOW);
    return;
  }
  P.sh_o[at] = make_float4(o.x, o.y, o.z, 0.f);
  P.sh_d[at] = d;
  P.sh_c[at] = make_float4(contrib.x, contrib.y, contrib.z, 0.f);
  P.sh_px[at] = px;
}

__device__ __forceinline__ void add_px(double *accum, uint32_t px, F3 c) {
  atomicAdd(&accum[3 * (size_t)px], (double)c.x);
  atomicAdd(&accum[3 * (size_t)px + 1], (double)c.y);
  atomicAdd(&accum[3 * (size_t)px + 2], (double)c.z);
}

// The state of camera path g (path index = sample * npix + pixel, within a job):
// ray origin (tmin in w), direction (tmax in w), throughput (MIS weight in w) and
// meta (output pixel, sample, depth, flags with the job index above bit 8).
__device__ __forceinline__ void camera_ray(const Cam &cam0, const Params &prm, uint64_t g, float4 &ro, float4 &rd,
                                           float4 &b4, uint4 &meta) {
  b4 = make_float4(1.f, 1.f, 1.f, 1.f);
  if (prm.rays) {
    const uint32_t sample = (uint32_t)(g / prm.npix), row = (uint32_t)(g % prm.npix);
    const float4 o = prm.rays[2 * (size_t)row], d4 = prm.rays[2 * (size_t)row + 1];
    const F3 d = normalize(f3(d4.x, d4.y, d4.z));  // shade() takes normalised directions
    ro = make_float4(o.x, o.y, o.z, fmaxf(o.w, 0.f));  // a negative tmin marks explicit rays
    rd = make_float4(d.x, d.y, d.z, d4.w);
    meta = make_uint4(row, sample, 0u, 0u);
    return;
  }
  Cam cam = cam0;
  uint32_t npix = prm.npix, job = 0, px_base = 0;
  if (prm.jobs) {
    job = job_of(prm.jobs, prm.njobs, g);
    const JobDev &J = prm.jobs[job];
    cam = J.cam;
    npix = J.npix;
    px_base = J.accum_off;
    g -= J.path_begin;
  }
  uint32_t sample = (uint32_t)(g / npix), pix = (uint32_t)(g % npix);
  uint32_t x = pix % cam.w, y = pix / cam.w;
  float jx = sample < 8 ? c_jx[sample] : 0.f, jy = sample < 8 ? c_jy[sample] : 0.f;
  F3 d = cam.cx * (((float)x + jx) / (float)cam.w - 0.5f) + cam.cy * (((float)y + jy) / (float)cam.h - 0.5f) +
         cam.dir;
  d = normalize(d);
  ro = make_float4(cam.pos.x, cam.pos.y, cam.pos.z, 0.f);
  rd = make_float4(d.x, d.y, d.z, 3.0e38f);
  uint32_t out_px = (cam.h - 1 - y) * cam.w + x;
  meta = make_uint4(px_base + out_px, sample, 0u, job << 8);
}

// Starts camera path g in path slot `slot`.
__device__ __forceinline__ void camera_path(const Cam &cam0, const Params &prm, const Paths &P, uint64_t g,
                                            uint32_t slot) {
  float4 ro, rd, b4;
  uint4 meta;
  camera_ray(cam0, prm, g, ro, rd, b4, meta);
  P.ray_o[slot] = ro;
  P.ray_d[slot] = rd;
  P.beta[slot] = b4;
  P.meta[slot] = meta;
}

// Camera paths wave_base + [0, wave_n) into slots [0, wave_n) and queue 0; the
// next path to start (regeneration) is wave_base + wave_n.
template <int TPB>
__global__ void __launch_bounds__(TPB) k_camera(Cam cam0, Paths P, Params prm, uint64_t wave_base,
                                                  uint32_t wave_n) {
  for (uint32_t i = blockIdx.x * TPB + threadIdx.x; i < wave_n; i += gridDim.x * TPB) {
    camera_path(cam0, prm, P, wave_base + i, i);
    P.q0[i] = i;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    P.counts[0] = wave_n;
    P.counts[3] = 0;
    P.counts[5] = (uint32_t)(wave_base + wave_n);
  }
}

// Path regeneration at the end of a shading step: lanes whose path ended take the
// next camera paths (one warp-wide reservation).  Returns true when this lane's
// slot now holds a fresh camera path.  All 32 lanes must call.
__device__ __forceinline__ bool regenerate(const Params &prm, const Paths &P, bool ended, uint32_t slot) {
  if (!prm.regen_total) return false;
  const uint32_t g = ballot_reserve(&P.counts[5], ended);
  if (!ended || g >= prm.regen_total) return false;
  camera_path(prm.cam, prm, P, g, slot);
  return true;
}

// Trees at least this many levels deep are traversed with dynamic fetching
// (trace_dynamic); shallower ones with one ray per thread (trace_static).  Box scene with more
// triangles, PATH, 512^2 x 4 spp, static / dynamic: one level (13 triangles) 584 / 760 us, two (21)
// 761 / 900, three (29) 742 / 895, four (37, 93, 333) 834 / 901, 989 / 978, 1120 / 1050, five
// (1,293) 1246 / 1118; many-light room, eight levels, 640 x 360 x 4 spp, 1829 / 1546.
constexpr uint32_t kDynamicDepth = 4;

// How k_extend / k_shadow walk the tree: one ray per thread, or dynamic fetching with
// or without the scene's spheres.
enum Walk : int { kWalkStatic = 0, kWalkDyn = 1, kWalkDynNoSpheres = 2 };

// Resident blocks of k_extend / k_shadow: 1024 / TPB, i.e. 64 registers.  One ray
// per thread (shallow trees): box frame 1.233 -> 1.208 ms against the compiler's
// choice.  Dynamic fetching (deep trees), where the triangle test's ray data (shear
// rows, direction) sit in shared memory after the stacks (TriShearSmem): with the
// rows in registers the kernels took 92 / 89 registers (five CTAs per SM), with them
// in shared memory 78 / 72 (six / seven CTAs; 1080p 64-spp many-light frame 0.332 ->
// 0.309 s), and capped at 64 registers without spills, eight CTAs: 0.299 s.  Their
// box test is the traversal kernels' (plane bytes by permute, the scene's slot bits), the
// one-ray-per-thread kernels' converts the bytes (with permutes the box frame took 765 us
// for 701).
constexpr int trace_blocks(int tpb) { return 1024 / tpb < 1 ? 1 : 1024 / tpb; }

// Closest hit of the paths in queue `cur`.  Dynamic fetching over the queue takes its
// work from the counter P.counts[3] (zeroed before the launch).
template <int TPB, Walk WALK>
__global__ void __launch_bounds__(TPB, trace_blocks(TPB)) k_extend(SceneView s, Paths P, int cur, int depth) {
  extern __shared__ uint2 smem_trav[];
  const uint32_t *q = cur ? P.q1 : P.q0;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    P.counts[cur ^ 1] = 0;
    P.counts[2] = 0;
    P.counts[4] = 0;
    P.counts[6] = 0;
    atomicAdd(&P.stats[0], (unsigned long long)P.counts[cur]);  // ray statistics: this step's closest-hit rays
  }
  auto fetch = [&](uint32_t i, RayPre &r, float &tmax) {
    const uint32_t slot = q[i];
    const float4 a = P.ray_o[slot], b = P.ray_d[slot];
    if (a.w < 0.f) return false;  // traced by the shading kernel (CKR_SHADER_EXPLICIT)
    r = make_ray(a, b);
    tmax = b.w;
    return true;
  };
  auto finish = [&](uint32_t i, uint32_t best, float t) {
    const uint32_t slot = q[i];
    P.hit_id[slot] = best;
    P.hit_t[slot] = t;
  };
  if constexpr (WALK != kWalkStatic) {
    const auto tri = dynamic_policy<TPB, WALK == kWalkDyn>(smem_trav, depth);
    auto fetch_s = [&](uint32_t i, RayPre &r, float &tmax) {
      if (!fetch(i, r, tmax)) return false;
      store_shear<TPB>(tri.col, r);
      return true;
    };
    trace_dynamic<false>(s, P.counts[cur], P.counts + 3, smem_trav + threadIdx.x, TPB, depth, fetch_s, finish,
                         tri);
  } else
    trace_static<false, TPB>(s, P.counts[cur], smem_trav + threadIdx.x, depth, fetch, finish);
}

// Any hit of the shadow queue: unoccluded rays add their contribution to the
// pixel; occluded ones zero their training record's weight.  Dynamic
// fetching takes its work from the counter P.counts[4] (zeroed before the launch).
template <int TPB, Walk WALK>
__global__ void __launch_bounds__(TPB, trace_blocks(TPB)) k_shadow(SceneView s, Paths P, int depth, float4 *rec) {
  extern __shared__ uint2 smem_trav[];
  const uint32_t n = min(P.counts[2], P.sh_cap);
  if (blockIdx.x == 0 && threadIdx.x == 0)
    atomicAdd(&P.stats[1], (unsigned long long)n);  // ray statistics: this step's shadow rays
  auto fetch = [&](uint32_t i, RayPre &r, float &tmax) {
    const float4 a = P.sh_o[i], b = P.sh_d[i];
    r = make_ray(a, b);
    tmax = b.w;
    return true;
  };
  auto finish = [&](uint32_t i, uint32_t best, float) {
    if (best == kMiss) {
      const float4 c = P.sh_c[i];
      add_px(P.accum, P.sh_px[i], f3(c.x, c.y, c.z));
    } else if (rec) {
      const uint32_t ri = P.sh_rec[i];
      if (ri != kNoRec) rec[3 * (size_t)ri + 1].w = 0.f;  // occluded: the sample contributed nothing
    }
  };
  if constexpr (WALK != kWalkStatic) {
    const auto tri = dynamic_policy<TPB, WALK == kWalkDyn>(smem_trav, depth);
    auto fetch_s = [&](uint32_t i, RayPre &r, float &tmax) {
      fetch(i, r, tmax);
      store_shear<TPB>(tri.col, r);
      return true;
    };
    trace_dynamic<true>(s, n, P.counts + 4, smem_trav + threadIdx.x, TPB, depth, fetch_s, finish,
                        tri);
  } else
    trace_static<true, TPB>(s, n, smem_trav + threadIdx.x, depth, fetch, finish);
}

using ExtendFn = void (*)(SceneView, Paths, int, int);
using ShadowFn = void (*)(SceneView, Paths, int, float4 *);
inline Walk walk_of(const ckr_scene *s) {
  return s->max_depth < kDynamicDepth ? kWalkStatic : s->nsph ? kWalkDyn : kWalkDynNoSpheres;
}
template <int TPB>
ExtendFn extend_fn_of(const ckr_scene *s) {
  const Walk w = walk_of(s);
  return w == kWalkStatic ? k_extend<TPB, kWalkStatic>
         : w == kWalkDyn  ? k_extend<TPB, kWalkDyn>
                          : k_extend<TPB, kWalkDynNoSpheres>;
}
template <int TPB>
ShadowFn shadow_fn_of(const ckr_scene *s) {
  const Walk w = walk_of(s);
  return w == kWalkStatic ? k_shadow<TPB, kWalkStatic>
         : w == kWalkDyn  ? k_shadow<TPB, kWalkDyn>
                          : k_shadow<TPB, kWalkDynNoSpheres>;
}

// The sample of point light L (deterministic, no MIS, src/lightSources.cpp:48-63):
// false below the surface, else the shadow ray's direction and tmax and its contribution.
__device__ __forceinline__ bool point_sample(const DevLight &L, const Surface &S, const Material &M, F3 fcol, F3 beta,
                                             F3 o_off, float4 &d4, F3 &contrib) {
  F3 dl = f3(L.px, L.py, L.pz) - S.x;
  float dist = length(dl);
  F3 w = dl * (1.0f / dist);
  float c = dot(w, S.n);
  if (c < 0.f) return false;
  float f = brdf_eval(M, S.n, S.wo_ref, S.wo, w);
  float sc4 = c * f / (4.0f * kPi * dist * dist);
  contrib = mulc(beta, mulc(fcol, f3(L.pr, L.pg, L.pb))) * sc4;
  d4 = make_float4(w.x, w.y, w.z, shadow_tmax(length(f3(L.px, L.py, L.pz) - o_off)));
  return true;
}

// Direction of the light techniques' sample si of one vertex: n_light samples per
// area and sphere light (lights are stored in the reference's getSamples order, sphere
// sources, mesh sources, triangle sources; src/mis.cpp:100-146, so sample si belongs
// to light si / n_light), then the environment's (EnMpIS, src/mis.cpp:154-166).
template <uint32_t LF>
__device__ __forceinline__ F3 technique_dir(const ShadeView &sv, const Params &prm, F3 x, uint32_t si, uint32_t nls,
                                            float e0, float e1, float e2) {
  if ((LF & kLightEnv) && si >= nls) return env_sample(sv, e0, e1, e2);
  return sample_light<LF>(sv, sv.lights[si / prm.n_light], x, e0, e1, e2);
}

// Of the BRDF samples [i0, i0 + n) of one vertex (n <= 32; sample i draws from the
// sample index sidx0 + i, the first nlobe from the specular lobe, the rest cosine),
// the ones whose direction may meet a light (MESH_ONLY: a mesh light): bit i - i0.  A
// conservative test against each light's bounding sphere, about a tenth of the work of
// the exact one: few of these directions meet a light (one in thirty on the box scene),
// and the ones that do not add nothing.  A cosine direction is formed with the fast
// sine, cosine and square root (within 2e-6 of sample_cosine's); the sphere is widened
// by 2e-4 of its distance and its squared tangent length by 1e-5, well above that and
// the rounding of these sums.  NaN counts as "may meet".
// Out of line: the kernels wait on instruction fetch (a 163 x 121 preview 64.2 -> 62.9 us, 512^2
// DIRECT_MISCV 479 -> 475).
template <bool MESH_ONLY>
__device__ __noinline__ uint32_t may_meet_light(const ShadeView &sv, const Surface &S, const Material &M,
                                                   uint64_t key, uint32_t sample, uint32_t depth, F3 o_off,
                                                   uint32_t sidx0, uint32_t i0, uint32_t n, uint32_t nlobe) {
  const uint32_t all = n >= 32 ? 0xffffffffu : (1u << n) - 1u;
  F3 X, Y;
  ref_frame(S.n, X, Y);
  uint32_t mask = 0;
  for (uint32_t k = 0; k < sv.first_point; ++k) {
    const DevLight &L = sv.lights[k];
    if (MESH_ONLY && L.type != CKR_LIGHT_MESH) continue;
    const F3 l = f3(L.px, L.py, L.pz) - o_off;
    const float ll = dot(l, l), rr = fabsf(L.radius) + 2e-4f * sqrtf(ll);  // a sphere's radius may be negative
    const float thr = ll - rr * rr - 1e-5f * ll;
    if (!(thr > 0.f)) return all;  // inside or at the sphere
    const float lx = dot(l, X), ly = dot(l, Y), ln = dot(l, S.n);
    for (uint32_t j = 0; j < n; ++j) {
      const float e1 = ckr_draw_f(key, ctr(sample, depth, 3 * (sidx0 + i0 + j) + 1));
      const float e2 = ckr_draw_f(key, ctr(sample, depth, 3 * (sidx0 + i0 + j) + 2));
      float b;
      if (i0 + j < nlobe) {
        b = dot(l, sample_dir(M, S.n, S.wo_ref, S.wo, true, e1, e2));
      } else {
        float sp, cp;  // of 2 pi e2 - pi, inside the fast functions' accurate range
        __sincosf(2.0f * kPi * (e2 - 0.5f), &sp, &cp);
        const float st = e1 * rsqrtf(e1), ct = (1.0f - e1) * rsqrtf(1.0f - e1);
        b = ct * ln - st * (cp * lx + sp * ly);
      }
      if (!(b < 0.f || b * b < thr)) mask |= 1u << j;
    }
  }
  return mask;
}

// getLightAnalytic / getLightAnalyticDiffuse over every mesh light
// (src/lightSources_CV.cpp:221-321): spec * amplitude * sum L |I_ltc| / 2pi +
// (1 - spec) * sum L |I_cos| / 2pi.  `no_spec`: the material's spec is 0 and the first part a
// zero.
__device__ __forceinline__ F3 ltc_term(const ShadeView &sv, const Surface &S, const Material &M, const LtcLookup &Lk,
                                       const M3f &minv, bool ltc_on, bool no_spec = false) {
  F3 G = f3(0, 0, 0);
  for (uint32_t k = 0; k < sv.nlights; ++k) {
    DevLight L = sv.lights[k];
    if (L.type != CKR_LIGHT_MESH) continue;
    F3 gs = f3(0, 0, 0), gd = f3(0, 0, 0);
    for (uint32_t j = 0; j < L.count; ++j) {
      const float *t9 = sv.tri9 + 9 * (size_t)(L.first + j);
      F3 A = f3(t9[0], t9[1], t9[2]), B = f3(t9[3], t9[4], t9[5]), C = f3(t9[6], t9[7], t9[8]);
      F3 Le = mat_radiance(sv, sv.tri_mat[L.first + j]);
      float s = ltc_on && !no_spec ? ltc_spec_tri(A, B, C, S.x, minv) : 0.f;
      float d = ltc_diffuse_tri(A, B, C, S.n, S.x);
      gs = gs + Le * s;
      gd = gd + Le * d;
    }
    const float inv2pi = 1.0f / (2.0f * kPi);
    G = G + gs * (inv2pi * (ltc_on ? Lk.amp : 0.f) * M.spec) + gd * (inv2pi * (1.0f - M.spec));
  }
  return G;
}

// The sampled part of getLightFromMeshSource_AnalyticCV (src/lightSources_CV.cpp:335-397):
// per mesh light, n_light points by MeshLight::getSamples (300-bin CDF, sqrt(u1)
// barycentrics), each adding Le (V f - f_ltc) cos cos_l / d^2 * area / n.  The
// unoccluded -f_ltc part is summed into `neg`; each +f part is a shadow ray.  All 32
// lanes must call (`surface`: this lane has a vertex).
__device__ __forceinline__ void cv_samples(const ShadeView &sv, const Paths &P, const Params &prm, bool surface,
                                           const Surface &S, const Material &M, const LtcLookup &Lk, const M3f &minv,
                                           bool ltc_on, uint64_t key, const uint4 &meta, F3 o_off, F3 &neg) {
  uint32_t sidx = 0;
  for (uint32_t k = 0; k < sv.first_point; ++k) {
    DevLight L = sv.lights[k];
    if (L.type != CKR_LIGHT_MESH) continue;
    const float w_area = L.area / (float)prm.n_light;
    for (uint32_t i = 0; i < prm.n_light; ++i, ++sidx) {
      bool want = false;
      float4 d4 = make_float4(0, 0, 0, 0);
      F3 contrib = f3(0, 0, 0);
      if (surface) {
        float e0 = ckr_draw_f(key, ctr(meta.y, 0, 3 * sidx));
        float e1 = ckr_draw_f(key, ctr(meta.y, 0, 3 * sidx + 1));
        float e2 = ckr_draw_f(key, ctr(meta.y, 0, 3 * sidx + 2));
        uint32_t b = (uint32_t)(e0 * (float)kInvCdfBins);
        b = b >= kInvCdfBins ? kInvCdfBins - 1 : b;
        const uint32_t tri = L.first + __ldg(&sv.cdf[L.cdf + b]);
        const float *t9 = sv.tri9 + 9 * (size_t)tri;
        F3 A = f3(__ldg(t9), __ldg(t9 + 1), __ldg(t9 + 2));
        F3 B = f3(__ldg(t9 + 3), __ldg(t9 + 4), __ldg(t9 + 5));
        F3 C = f3(__ldg(t9 + 6), __ldg(t9 + 7), __ldg(t9 + 8));
        F3 Pl = sample_triangle(A, B, C, e1, e2);
        F3 dv = Pl - S.x;
        float d2 = dot(dv, dv), d = sqrtf(d2);
        F3 w = dv * (1.0f / d);
        float c = dot(w, S.n);
        if (!(c < 0.f)) {
          const float4 nm = __ldg(&sv.tri_nm[tri]);
          float c1 = fabsf(dot(w, f3(nm.x, nm.y, nm.z)));
          float g = c * c1 / d2 * w_area;
          F3 Le = mat_radiance(sv, __float_as_uint(nm.w));
          const ckr_material &mm = sv.mats[S.mat];
          float fa = brdf_eval(M, S.n, S.wo_ref, S.wo, w) * mm.reflectance;
          float fl = ltc_on ? brdf_ltc(M, Lk, minv, S.n, w) * mm.reflectance : fa;
          neg = neg - Le * (fl * g);
          if (fa > 0.f) {
            want = true;
            contrib = mulc(f3(mm.color[0], mm.color[1], mm.color[2]), Le) * (fa * g);
            d4 = shadow_dir(o_off, Pl);
          }
        }
      }
      emit_shadow(P, want, o_off, d4, contrib, meta.x);
    }
  }
}

// Continuation dims of CKR_SHADER_EXPLICIT: RR at kDimRR, redraws r < kExplicitTries
// of the hemisphere direction at kDimHemi + 2r, + 2r + 1.
constexpr uint32_t kDimHemi = 1004, kExplicitTries = 8;

// The next 32 queue rows of a warp of a shading kernel, after its first ones: taken from a
// counter, for a vertex costs from nothing (a miss, an emitter) to all its samples, and warps
// that strode over the queue ended far apart (512^2 DIRECT_MISCV: 16.9 of 24 warps resident on
// average, 647 -> 528 us; box path frame 615 -> 606 us; small-batch pass 1822 -> 1798 us).
__device__ __forceinline__ uint32_t next_rows(const Paths &P, uint32_t stride, uint32_t n, int lane) {
  if (stride >= n) return n;
  uint32_t at = 0;
  if (lane == 0) at = atomicAdd(&P.counts[6], 32u);
  return stride + __shfl_sync(0xffffffffu, at, 0);
}

template <uint32_t SHADER, int TPB, uint32_t LF = kLightsAll>
__device__ __forceinline__ void shade(ShadeView sv0, Paths P, Params prm, int cur, int depth,
                                      const LtcEntry *__restrict__ ltc, SceneView scene, int stack_depth) {
  const uint32_t n = P.counts[cur];
  const uint32_t *q = cur ? P.q1 : P.q0;
  uint32_t *qn = cur ? P.q0 : P.q1;
  if (blockIdx.x == 0 && threadIdx.x == 0) P.counts[3] = 0;
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (TPB / 32);
  const uint32_t warp_id = blockIdx.x * (TPB / 32) + (threadIdx.x >> 5);
  for (uint32_t base = warp_id * 32; base < n; base = next_rows(P, warps * 32, n, lane)) {
    uint32_t i = base + lane;
    bool valid = i < n;
    uint32_t slot = valid ? q[i] : 0;
    bool cont = false;
    Surface S;
    Material M;
    F3 fcol = f3(0, 0, 0), beta = f3(0, 0, 0);
    uint4 meta = make_uint4(0, 0, 0, 0);
    ShadeView sv = sv0;  // a batch job's materials replace the scene's
    PathCtx pc = path_ctx(prm, 0u);
    uint64_t key = 0;
    F3 o_off = f3(0, 0, 0);
    bool surface = false, lam = false;
    if (valid) {
      uint32_t id = P.hit_id[slot];
      meta = P.meta[slot];
      pc = path_ctx(prm, meta.w);
      sv.mats = sv0.mats + pc.mat_off;
      if ((LF & kLightEnv) && id == kMiss && SHADER == CKR_SHADER_PATH && sv.env_n && meta.z > 0) {
        // A BRDF-sampled ray left the scene: the environment, with its MIS weight.
        const float4 rd = P.ray_d[slot], b4 = P.beta[slot];
        const float4 e = env_lookup(sv, f3(rd.x, rd.y, rd.z));
        add_px(P.accum, meta.x, mulc(f3(b4.x, b4.y, b4.z), f3(e.x, e.y, e.z)) * b4.w);
      }
      if (id != kMiss) {
        float4 ro = P.ray_o[slot], rd = P.ray_d[slot], b4 = P.beta[slot];
        beta = f3(b4.x, b4.y, b4.z);
        S = make_surface(sv, f3(ro.x, ro.y, ro.z), f3(rd.x, rd.y, rd.z), id, P.hit_t[slot]);
        const ckr_material &mm = sv.mats[S.mat];
        if (mm.light_type != 0) {
          // Emitter.  Camera rays see MaterialType::getRadiance, the radiance
          // divided by its largest component (headers/materialTypes.h:34-38);
          // BRDF-sampled rays carry their MIS weight.
          F3 Le = f3(mm.radiance[0], mm.radiance[1], mm.radiance[2]);
          if (meta.z == 0) {
            float mx = fmaxf(Le.x, fmaxf(Le.y, Le.z));
            // Vec::maxnorm picks the largest component in x, y, z order.
            mx = Le.x;
            if (mx < Le.y) mx = Le.y;
            if (mx < Le.z) mx = Le.z;
            add_px(P.accum, meta.x, Le * (1.0f / mx));
          } else {
            add_px(P.accum, meta.x, mulc(beta, Le) * b4.w);
          }
        } else if (!(meta.w & 1u)) {
          surface = true;
          M = material_of(mm);
          lam = is_lambert(M, dot(S.wo, S.n));
          fcol = f3(mm.color[0], mm.color[1], mm.color[2]) * mm.reflectance;
          key = ckr_key(pc.seed, meta.x - pc.px_base);
          o_off = offset_origin(S.x, S.n);
        }
      }
    }
    // The path continues in its slot; its rows are written as soon as they are known: held to
    // the end of the vertex they were spilled (small-batch pass 1.94 -> 1.87 ms).  A tmin of -1 marks a ray the explicit loop has
    // traced already.
    auto go_on = [&](F3 w, F3 nb, float wb) {
      cont = true;
      const uint32_t nd = meta.z + 1;
      P.ray_o[slot] = make_float4(o_off.x, o_off.y, o_off.z, SHADER == CKR_SHADER_EXPLICIT ? -1.f : 0.f);
      P.ray_d[slot] = make_float4(w.x, w.y, w.z, 3.0e38f);
      P.beta[slot] = make_float4(nb.x, nb.y, nb.z, wb);
      P.meta[slot] = make_uint4(meta.x, meta.y, nd, (meta.w & ~1u) | (nd >= pc.max_depth ? 1u : 0u));
    };
    // ---- direct light ----
    LtcLookup Lk{};
    M3f minv{};
    bool ltc_on = false;
    F3 cv_neg = f3(0, 0, 0);
    if (surface && (SHADER == CKR_SHADER_DIRECT_MISCV || SHADER == CKR_SHADER_DIRECT_CV ||
                    SHADER == CKR_SHADER_EXPLICIT)) {
      auto tab = [&](int idx) { return ltc[idx]; };
      float theta = acosf(fminf(1.0f, fmaxf(-1.0f, dot(S.n, S.wo))));
      Lk = ltc_lookup(tab, theta, M.alpha);
      minv = ltc_minv_world(Lk, S.n, S.wo);
      ltc_on = M.brdf == kGGX || M.brdf == kGGXApprox;
    }
    if (SHADER == CKR_SHADER_DIRECT_CV)
      cv_samples(sv, P, prm, surface, S, M, Lk, minv, ltc_on, key, meta, o_off, cv_neg);
    if (SHADER == CKR_SHADER_PATH || SHADER == CKR_SHADER_DIRECT_MIS) {
      // Point lights, then the MIS set: the light techniques' samples, and the BRDF
      // samples (DIRECT_MIS, N * spec lobe samples, the rest cosine, as
      // getBrdfDirectionSamples, src/materialTypes.cpp:118-134) or the one BRDF sample
      // that continues the path (PATH).  A light's, the environment's and a BRDF sample
      // all take the same query and BRDF evaluation, one copy of their code in one loop,
      // and a sample's shadow ray is appended as soon as it is known (counting the rays
      // first and forming them in a second pass took every sample twice: box path frame
      // 1.049 -> 0.927 ms, small-batch pass 3.52 -> 3.03 ms).  The loop is the same for all lanes of a warp, and every lane
      // takes part in its reservations.
      for (uint32_t k = sv.first_point; (LF & kLightPoint) && k < sv.nlights; ++k) {
        float4 d4 = make_float4(0, 0, 0, 0);
        F3 contrib = f3(0, 0, 0);
        const bool want = surface && point_sample(sv.lights[k], S, M, fcol, beta, o_off, d4, contrib);
        emit_shadow(P, want, o_off, d4, contrib, meta.x);
      }
      const uint32_t nls = sv.first_point * prm.n_light, nlt = nls + ((LF & kLightEnv) ? sv.env_n : 0u);
      const uint32_t nb = SHADER == CKR_SHADER_PATH ? 1u : prm.n_brdf;
      const uint32_t nlobe = surface ? (uint32_t)((float)nb * M.spec) : 0u;
      for (uint32_t s0 = 0; s0 < nlt + nb;) {
        const bool light = s0 < nlt, last = SHADER == CKR_SHADER_PATH && !light;
        const uint32_t cnt = min(32u, (light ? nlt : nlt + nb) - s0);
        uint32_t todo = !surface ? 0u : cnt >= 32 ? 0xffffffffu : (1u << cnt) - 1u;
        // BRDF samples that meet no light add nothing (with an environment all do).
        if (SHADER == CKR_SHADER_DIRECT_MIS && surface && !light && !((LF & kLightEnv) && sv.env_n))
          todo = may_meet_light<false>(sv, S, M, key, meta.y, meta.z, o_off, nlt, s0 - nlt, cnt, nlobe);
        while (__any_sync(0xffffffffu, todo)) {
          bool want = false;
          float4 d4 = make_float4(0, 0, 0, 0);
          F3 contrib = f3(0, 0, 0);
          if (todo) {
            const uint32_t si = s0 + __ffs(todo) - 1;
            todo &= todo - 1;
            const uint32_t dim = last ? kDimBrdf : 3 * si;
            const float e0 = ckr_draw_f(key, ctr(meta.y, meta.z, dim));
            const float e1 = ckr_draw_f(key, ctr(meta.y, meta.z, dim + 1));
            const float e2 = ckr_draw_f(key, ctr(meta.y, meta.z, dim + 2));
            const F3 w = light ? technique_dir<LF>(sv, prm, S.x, si, nls, e0, e1, e2)
                               : sample_dir(M, S.n, S.wo_ref, S.wo,
                                            SHADER == CKR_SHADER_PATH ? e0 < M.spec : si - nlt < nlobe, e1, e2);
            const float c = dot(w, S.n);
            if (last ? c > 0.f && ckr_draw_f(key, ctr(meta.y, meta.z, kDimRR)) >= prm.rr_prob : !(c < 0.f)) {
              const LightQuery lq = query_lights<true, LF>(sv, S.x, o_off, w, prm.n_light);
              if (last || lq.hit) {
                float f, p;
                brdf_pdf_eval(M, S.n, S.wo_ref, S.wo, w, f, p, lam);
                if (!last) {
                  const float denom = lq.pdf_sum + (float)nb * p;
                  contrib = mulc(beta, mulc(fcol, lq.Le)) * (f * c / (denom + 1e-20f));
                  d4 = make_float4(w.x, w.y, w.z, shadow_tmax(lq.d));
                  want = true;
                } else if (p > 0.f && f > 0.f) {
                  const float wb = (float)nb * p / ((float)nb * p + lq.pdf_sum);
                  const F3 nbeta = mulc(beta, fcol) * (f * c / (p * (1.0f - prm.rr_prob)));
                  go_on(w, nbeta, wb);
                }
              }
            }
          }
          if (!last) emit_shadow(P, want, o_off, d4, contrib, meta.x);
        }
        s0 += cnt;
      }
    }
    if (surface && SHADER == CKR_SHADER_DIRECT_CV) {
      // getLightFromMeshSource_AnalyticCV: the LTC term plus the unoccluded part of
      // the sampled residual; the occluded part arrives through the shadow rays.
      const ckr_material &mm = sv.mats[S.mat];
      F3 col = f3(mm.color[0], mm.color[1], mm.color[2]);
      add_px(P.accum, meta.x, mulc(col, ltc_term(sv, S, M, Lk, minv, ltc_on) + cv_neg));
    }
    if (surface && (SHADER == CKR_SHADER_DIRECT_MISCV || SHADER == CKR_SHADER_EXPLICIT)) {
      // getLightFromMeshSource_Analytic_MISCV (src/lightSources_CV.cpp:399-450); at
      // every vertex of the explicit path loop (shadeDI, src/shader.cpp:100-109).
      // Without a specular part the BRDF is its LTC approximation (is_lambert: both are 1 / pi),
      // so a sample's residual is an exact zero and the sample is left out, unless it is a
      // light's below kLambertCos, which is evaluated to see (a cosine direction never is).
      // Box, 512^2 x 4 spp: 1.79 -> 0.70 ms.
      const bool same_brdf = lam && ltc_on && Lk.det > 0.f && Lk.amp < 1e30f && sv.finite_radiance;
      // Lights wholly above or below the surface's plane, by more than kLambertCos and the
      // rounding of a sampled point, have no sample whose cosine must be looked at (521 ->
      // 477 us).
      bool no_samples = same_brdf;
      for (uint32_t k = 0; no_samples && k < sv.first_point; ++k) {
        const DevLight &L = sv.lights[k];
        const F3 v = f3(L.px, L.py, L.pz) - S.x;
        const float r = fabsf(L.radius), h = dot(v, S.n);
        const float reach = 1e-3f * (length(v) + r) + 1e-6f * (fabsf(L.px) + fabsf(L.py) + fabsf(L.pz) + r);
        no_samples = h - r > reach || h + r < -reach;
      }
      F3 G = ltc_term(sv, S, M, Lk, minv, ltc_on, same_brdf);
      // MIS residual over the getSamples set; visibility is 1 in the reference.
      F3 res = f3(0, 0, 0);
      const uint32_t nb = prm.n_brdf, nlobe = (uint32_t)((float)nb * M.spec);
      const uint32_t nls = sv.first_point * prm.n_light;
      // A sample adds nothing unless its direction meets a mesh light: the BRDF samples
      // are first cut down to those that may (may_meet_light), 32 at a time, and only
      // these run the queries and the BRDF's terms (box, 512^2 x 4 spp, 10 light + 60
      // BRDF samples: 4.84 -> 2.63 ms).  The sums' order stays the samples'.
      for (uint32_t s0 = 0; s0 < nls + nb;) {
        const bool lights = s0 < nls;
        const uint32_t cnt = min(32u, (lights ? nls : nls + nb) - s0);
        uint32_t todo = cnt >= 32 ? 0xffffffffu : (1u << cnt) - 1u;
        if (lights ? no_samples : same_brdf) todo = 0;
        else if (!lights) todo = may_meet_light<true>(sv, S, M, key, meta.y, meta.z, o_off, nls, s0 - nls, cnt, nlobe);
        while (todo) {
          const uint32_t si = s0 + __ffs(todo) - 1;
          todo &= todo - 1;
          float e0 = ckr_draw_f(key, ctr(meta.y, meta.z, 3 * si));
          float e1 = ckr_draw_f(key, ctr(meta.y, meta.z, 3 * si + 1));
          float e2 = ckr_draw_f(key, ctr(meta.y, meta.z, 3 * si + 2));
          F3 w = lights ? sample_light<LF>(sv, sv.lights[si / prm.n_light], S.x, e0, e1, e2)
                        : sample_dir(M, S.n, S.wo_ref, S.wo, si - nls < nlobe, e1, e2);
          float c = dot(w, S.n);
          if (c < 0.f || (same_brdf && c > kLambertCos)) continue;
          LightQuery lq = query_lights<false, LF>(sv, S.x, o_off, w, prm.n_light);
          if (lq.mesh == kMiss) continue;
          // lq.mesh: of the first mesh light in list order that the direction meets.
          float f, p;
          brdf_pdf_eval(M, S.n, S.wo_ref, S.wo, w, f, p, lam);
          float denom = lq.pdf_sum + (float)nb * p;
          float fa = f * sv.mats[S.mat].reflectance;
          float fl = ltc_on ? brdf_ltc(M, Lk, minv, S.n, w) * sv.mats[S.mat].reflectance : fa;
          res = res + mat_radiance(sv, sv.tri_mat[lq.mesh]) * ((fa - fl) * c / (denom + 1e-20f));
        }
        s0 += cnt;
      }
      const ckr_material &mm = sv.mats[S.mat];
      F3 col = f3(mm.color[0], mm.color[1], mm.color[2]);
      add_px(P.accum, meta.x, mulc(beta, mulc(col, res + G)));
    }
    // ---- continuation of the explicit path loop (shadeExplicit, src/shader.cpp:111-207):
    // Russian roulette 0.3 after the vertex's direct light, then a uniform hemisphere
    // direction, redrawn while it meets an emitter (emitters only count through the
    // direct term), traced here; beta *= c 2 pi cos f / 0.7.
    if (SHADER == CKR_SHADER_EXPLICIT) {
      extern __shared__ uint2 smem_trav[];
      uint32_t hit = kMiss;
      float th = 0.f;
      F3 wn = f3(0, 0, 0);
      const bool go = surface && meta.z + 1 < pc.max_depth &&
                      ckr_draw_f(key, ctr(meta.y, meta.z, kDimRR)) >= prm.rr_prob;
      // Every lane runs the same number of traversals (the stack is per thread, the
      // loop has no barrier, but keeping lanes together keeps the warp converged).
      bool done = !go;
      for (uint32_t r = 0; r < kExplicitTries; ++r) {
        if (!done) {
          wn = sample_hemisphere(S.n, ckr_draw_f(key, ctr(meta.y, meta.z, kDimHemi + 2 * r)),
                                 ckr_draw_f(key, ctr(meta.y, meta.z, kDimHemi + 2 * r + 1)));
          RayPre rp = ray_pre(o_off, wn, 0.f);
          th = 3.0e38f;
          hit = trace_ray<false>(scene, rp, th, smem_trav + threadIdx.x, TPB, stack_depth);
          if (hit == kMiss) {
            done = true;  // escapes the scene
          } else {
            const uint32_t hm = (hit & kSphereBit) ? __ldg(&sv.sph_mat[hit & ~kSphereBit]) : __ldg(&sv.tri_mat[hit]);
            if (sv.mats[hm].light_type == 0) done = true;  // accepted
            else hit = kMiss;                              // an emitter: draw again
          }
        }
      }
      if (go && hit != kMiss) {
        const ckr_material &mm = sv.mats[S.mat];
        float f = brdf_eval(M, S.n, S.wo_ref, S.wo, wn) * mm.reflectance;
        float k = 2.0f * kPi * dot(wn, S.n) * f / (1.0f - prm.rr_prob);
        F3 nb = mulc(beta, f3(mm.color[0], mm.color[1], mm.color[2])) * k;
        go_on(wn, nb, 1.f);
        P.hit_id[slot] = hit;
        P.hit_t[slot] = th;
      }
    }
    const bool fresh = regenerate(prm, P, valid && !cont, slot);
    uint32_t cbase = ballot_reserve(&P.counts[cur ^ 1], cont || fresh);
    if (cont || fresh) qn[cbase] = slot;
  }
}

// Shading kernels.  The MIS path tracer's vertex is register hungry but short, and what it
// spills costs more than resident warps give: at 512 / TPB resident blocks (128 registers at
// 128 threads, nothing spilled) the box frame takes 586 us, at 640 592 (at 768 / 384, when
// it took 628, 670 / 684).  The direct-light shaders run at 1024 / TPB resident blocks (64 registers at
// 128 threads): box, 1080p x 2 spp, DIRECT_MIS of 1 light + 2 BRDF samples, at 512 / 640 / 768 / 1024 /
// 1280: 835 / 854 / 844 / 821 / 889 us; DIRECT_CV, 17 lights, 256^2, 643 / 635 / 655 / 635 / 668; small
// frames want fewer (163 x 121 with an environment 58 / 59 / 60 / 63 / 65).  The explicit path loop, which
// traverses inside the kernel, at 512 / TPB (128 registers; box 192^2 x 4 spp, depth 4, spec
// 0.6: 301 us, at 384 / 640 328 / 323).
constexpr int shade_blocks(uint32_t shader, int tpb) {
  return shader == CKR_SHADER_EXPLICIT ? (512 / tpb > 1 ? 512 / tpb : 1) : (1024 / tpb > 1 ? 1024 / tpb : 1);
}

template <uint32_t SHADER, int TPB, uint32_t LF = kLightsAll>
__global__ void __launch_bounds__(TPB, shade_blocks(SHADER, TPB)) k_shade(ShadeView sv0, Paths P, Params prm, int cur, int depth,
                                                 const LtcEntry *__restrict__ ltc, SceneView scene = SceneView{},
                                                 int stack_depth = 0) {
  shade<SHADER, TPB, LF>(sv0, P, prm, cur, depth, ltc, scene, stack_depth);
}

// LF: the light kinds compiled in (kLightsMeshOnly for scenes whose lights are all
// MESH / TRI lights, see mesh_lights_only).
template <int TPB, uint32_t LF = kLightsAll>
__global__ void __launch_bounds__(TPB, (512 / TPB > 1 ? 512 / TPB : 1))
    k_shade_path(ShadeView sv0, Paths P, Params prm, int cur, int depth, const LtcEntry *__restrict__ ltc) {
  shade<CKR_SHADER_PATH, TPB, LF>(sv0, P, prm, cur, depth, ltc, SceneView{}, 0);
}

// Whether a scene's lights are all MESH / TRI lights (no point or sphere light, no
// environment): its path shader can leave the other kinds' code out.
inline bool mesh_lights_only(const ckr_scene *s) {
  if (s->env_n) return false;
  for (const DevLight &L : s->host_lights)
    if (L.type != CKR_LIGHT_MESH && L.type != CKR_LIGHT_TRI) return false;
  return true;
}

// The reference's default shader (MISCV) at 512 / TPB resident blocks (128 registers at
// 128 threads): box, 512^2 x 4 spp, 10 light + 60 BRDF samples, at 384 / 512 / 640 / 768 / 1024:
// 487 / 447 / 464 / 469 / 458 us; 200^2 x 3 spp 152 / 160 / 176 / 190 / -.
template <int TPB, uint32_t LF = kLightsAll>
__global__ void __launch_bounds__(TPB, (512 / TPB > 1 ? 512 / TPB : 1))
    k_shade_miscv(ShadeView sv0, Paths P, Params prm, int cur, int depth, const LtcEntry *__restrict__ ltc) {
  shade<CKR_SHADER_DIRECT_MISCV, TPB, LF>(sv0, P, prm, cur, depth, ltc, SceneView{}, 0);
}

// CKR_SHADER_PATH_NEE: one light sample and one BRDF sample per vertex over many
// lights.  The light technique draws an emitter light from the selection
// distribution, one of its triangles in proportion to power and a uniform point
// on it; the BRDF sample continues the path and, if it meets an emitter, is
// weighted at the next vertex with the light technique's pdf of the previous
// vertex (its pdf is carried in beta.w).  Balance heuristic throughout.  Launched
// with 1024 / TPB resident blocks (64 registers at 128 threads, a few spills): the
// many-light frame, 1920 x 1080 x 8 spp, at 1024 / 1280 / 1536 takes 34.4 / 35.1 / 36.1 ms,
// the resident warps hiding the vertex's dependent loads.
template <int TPB>
__global__ void __launch_bounds__(TPB, (1024 / TPB > 1 ? 1024 / TPB : 1))
    k_shade_nee(ShadeView sv0, Paths P, Params prm, int cur, Learn lr) {
  const uint32_t n = P.counts[cur];
  const uint32_t *q = cur ? P.q1 : P.q0;
  uint32_t *qn = cur ? P.q0 : P.q1;
  if (blockIdx.x == 0 && threadIdx.x == 0) P.counts[3] = 0;
  const int lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (TPB / 32);
  const uint32_t warp_id = blockIdx.x * (TPB / 32) + (threadIdx.x >> 5);
  const float train_frac = lr.rec && n ? fminf(1.0f, (float)lr.rec_cap / (float)n) : 0.f;
  for (uint32_t base = warp_id * 32; base < n; base += warps * 32) {
    const uint32_t i = base + lane;
    const bool valid = i < n;
    const uint32_t slot = valid ? q[i] : 0;
    uint32_t nshadow = 0;
    bool cont = false, rec_ok = false;
    float4 sd = make_float4(0, 0, 0, 0), sc = sd, r0 = sd, r1 = sd, r2 = sd;
    F3 o_off = f3(0, 0, 0);
    uint4 meta = make_uint4(0, 0, 0, 0);
    ShadeView sv = sv0;  // a batch job's materials replace the scene's
    PathCtx pc = path_ctx(prm, 0u);
    if (valid) {
      uint32_t id = P.hit_id[slot];
      meta = P.meta[slot];
      pc = path_ctx(prm, meta.w);
      sv.mats = sv0.mats + pc.mat_off;
      if (id != kMiss) {
        float4 ro = P.ray_o[slot], rd = P.ray_d[slot], b4 = P.beta[slot];
        F3 beta = f3(b4.x, b4.y, b4.z);
        Surface S = make_surface(sv, f3(ro.x, ro.y, ro.z), f3(rd.x, rd.y, rd.z), id, P.hit_t[slot]);
        const ckr_material &mm = sv.mats[S.mat];
        if (mm.light_type != 0) {
          F3 Le = f3(mm.radiance[0], mm.radiance[1], mm.radiance[2]);
          if (meta.z == 0) {
            float mx = Le.x;  // Vec::maxnorm, as the other shaders
            if (mx < Le.y) mx = Le.y;
            if (mx < Le.z) mx = Le.z;
            add_px(P.accum, meta.x, Le * (1.0f / mx));
          } else {
            float wb = 1.0f;
            uint32_t k = (id & kSphereBit) ? kNoLight : __ldg(&sv.tri_light[id]);
            if (k != kNoLight && b4.w > 0.f) {
              DevLight L = sv.lights[k];
              Select sel{lr.sel_prev ? lr.sel_prev + 64 * (size_t)P.prev_row[slot] : nullptr};
              const float *t9 = sv.tri9 + 9 * (size_t)id;
              F3 A = f3(__ldg(t9), __ldg(t9 + 1), __ldg(t9 + 2));
              F3 B = f3(__ldg(t9 + 3), __ldg(t9 + 4), __ldg(t9 + 5));
              F3 C = f3(__ldg(t9 + 6), __ldg(t9 + 7), __ldg(t9 + 8));
              F3 nrm = cross_rn(C - A, B - A);
              float len = length(nrm);
              float cl = fabsf(dot(nrm, f3(rd.x, rd.y, rd.z))) / len;
              float pl = nee_pdf(sv, select_prob(sv, sel, k - sv.first_emit), L, id, P.hit_t[slot], 0.5f * len, cl);
              if (pl > 0.f && pl < 3.0e38f) wb = b4.w / (b4.w + pl);
            }
            add_px(P.accum, meta.x, mulc(beta, Le) * wb);
          }
        } else if (!(meta.w & 1u)) {
          Material M = material_of(mm);
          F3 fcol = f3(mm.color[0], mm.color[1], mm.color[2]) * mm.reflectance;
          uint64_t key = ckr_key(pc.seed, meta.x - pc.px_base);
          o_off = offset_origin(S.x, S.n);
          // ---- light technique: one sample ----
          float e0 = ckr_draw_f(key, ctr(meta.y, meta.z, 0)), e1 = ckr_draw_f(key, ctr(meta.y, meta.z, 1));
          float e2 = ckr_draw_f(key, ctr(meta.y, meta.z, 2)), e3 = ckr_draw_f(key, ctr(meta.y, meta.z, 3));
          Select sel{lr.sel ? lr.sel + 64 * (size_t)i : nullptr};
          uint32_t j = select_pick(sv, sel, e0);
          DevLight L = sv.lights[sv.first_emit + j];
          uint32_t tri = L.first + cdf_pick(sv.pcdf + L.pcdf, L.count, e1);
          const float *t9 = sv.tri9 + 9 * (size_t)tri;
          F3 A = f3(__ldg(t9), __ldg(t9 + 1), __ldg(t9 + 2));
          F3 B = f3(__ldg(t9 + 3), __ldg(t9 + 4), __ldg(t9 + 5));
          F3 C = f3(__ldg(t9 + 6), __ldg(t9 + 7), __ldg(t9 + 8));
          F3 Pl = sample_triangle(A, B, C, e2, e3);
          F3 dv = Pl - S.x;
          float dist = length(dv);
          F3 w = dv * (1.0f / dist);
          float c = dot(w, S.n);
          F3 nrm = cross_rn(C - A, B - A);
          float len = length(nrm);
          float cl = fabsf(dot(nrm, w)) / len;
          if (c > 0.f && cl > 0.f && len > 0.f && dist > 0.f) {
            float pl = nee_pdf(sv, select_prob(sv, sel, j), L, tri, dist, 0.5f * len, cl);
            float f, pb;
            brdf_pdf_eval(M, S.n, S.wo_ref, S.wo, w, f, pb);
            if (pl > 0.f && f > 0.f) {
              F3 Le = mat_radiance(sv, sv.tri_mat[tri]);
              float g = f * c / pl;
              F3 contrib = mulc(beta, mulc(fcol, Le)) * (g * (pl / (pl + pb)));
              nshadow = 1;
              sd = shadow_dir(o_off, Pl);
              sc = make_float4(contrib.x, contrib.y, contrib.z, 0.f);
              if (train_frac > 0.f && ckr_draw_f(key, ctr(meta.y, meta.z, kDimTrain)) < train_frac) {
                // Training sample: the unweighted estimate of cluster j's direct light
                // (luminance), zeroed by the shadow kernel if the ray is blocked.
                F3 fl = mulc(fcol, Le);
                rec_ok = true;
                r0 = make_float4(S.x.x, S.x.y, S.x.z, M.alpha);
                r1 = make_float4(S.n.x, S.n.y, S.n.z, (fl.x + fl.y + fl.z) * (1.0f / 3.0f) * g);
                r2 = make_float4(S.wo.x, S.wo.y, S.wo.z, __uint_as_float(j));
              }
            }
          }
          // ---- BRDF technique: continues the path ----
          if (meta.z + 1 <= pc.max_depth) {
            float b0 = ckr_draw_f(key, ctr(meta.y, meta.z, kDimBrdf));
            float b1 = ckr_draw_f(key, ctr(meta.y, meta.z, kDimBrdf + 1));
            float b2 = ckr_draw_f(key, ctr(meta.y, meta.z, kDimBrdf + 2));
            F3 wn = sample_brdf(M, S.n, S.wo_ref, S.wo, b0, b1, b2);
            float cn = dot(wn, S.n);
            float err = ckr_draw_f(key, ctr(meta.y, meta.z, kDimRR));
            if (cn > 0.f && err >= prm.rr_prob) {
              float f, pb;
              brdf_pdf_eval(M, S.n, S.wo_ref, S.wo, wn, f, pb);
              if (pb > 0.f && f > 0.f) {
                F3 nb = mulc(beta, fcol) * (f * cn / (pb * (1.0f - prm.rr_prob)));
                // Its rows are written at once: held to the vertex's end they were spilled
                // (many-light frame 34.4 -> 34.15 ms).
                const uint32_t nd = meta.z + 1;
                cont = true;
                P.ray_o[slot] = make_float4(o_off.x, o_off.y, o_off.z, 0.f);
                P.ray_d[slot] = make_float4(wn.x, wn.y, wn.z, 3.0e38f);
                P.beta[slot] = make_float4(nb.x, nb.y, nb.z, pb);
                P.meta[slot] = make_uint4(meta.x, meta.y, nd, (meta.w & ~1u) | (nd >= pc.max_depth ? 1u : 0u));
                if (lr.sel) P.prev_row[slot] = i;
              }
            }
          }
        }
      }
    }
    uint32_t rbase = kNoRec;
    if (lr.rec) {
      rbase = ballot_reserve(lr.rec_count, rec_ok);
      if (rec_ok && rbase < lr.rec_cap) {
        lr.rec[3 * (size_t)rbase] = r0;
        lr.rec[3 * (size_t)rbase + 1] = r1;
        lr.rec[3 * (size_t)rbase + 2] = r2;
      } else {
        rbase = kNoRec;
      }
    }
    const uint32_t sbase = ballot_reserve(&P.counts[2], nshadow != 0);
    if (nshadow && sbase >= P.sh_cap) {
      atomicCAS(P.status, 0, CKR_ERR_QUEUE_OVERFLOW);
    } else if (nshadow) {
      P.sh_o[sbase] = make_float4(o_off.x, o_off.y, o_off.z, 0.f);
      P.sh_d[sbase] = sd;
      P.sh_c[sbase] = sc;
      P.sh_px[sbase] = meta.x;
      if (lr.rec) P.sh_rec[sbase] = rbase;
    }
    const bool fresh = regenerate(prm, P, valid && !cont, slot);
    uint32_t cbase = ballot_reserve(&P.counts[cur ^ 1], cont || fresh);
    if (cont || fresh) qn[cbase] = slot;
  }
}

// Batched resolve: accumulation row p belongs to the job whose rows contain it.  The FP64
// pipe bounds it (a division per pixel, where the job now holds the quotient: 1.24M pixels of
// 512 jobs 35 -> 24 us).
__global__ void k_resolve_jobs(const double *accum, const JobDev *jobs, uint32_t njobs, uint32_t npix_total) {
  for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < npix_total; p += gridDim.x * blockDim.x) {
    uint32_t lo = 0, hi = njobs - 1;
    while (lo < hi) {
      uint32_t mid = (lo + hi + 1) >> 1;
      if (jobs[mid].accum_off <= p) lo = mid;
      else hi = mid - 1;
    }
    const JobDev &J = jobs[lo];
    const double inv = J.inv_spp;
    const uint32_t q = p - J.accum_off;
    for (int c = 0; c < 3; ++c) J.rgb[3 * (size_t)q + c] = (float)(accum[3 * (size_t)p + c] * inv);
  }
}

__global__ void k_resolve(const double *accum, float *rgb, uint32_t n3, double inv_spp) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n3; i += gridDim.x * blockDim.x)
    rgb[i] = (float)(accum[i] * inv_spp);
}


// Blocks for up to n items: the persistent grid g, or fewer where n fill fewer (an
// empty block of a full grid costs about as much as one that works).
inline unsigned grid_of(int g, uint64_t n, int tpb) { return (unsigned)std::min<uint64_t>(g, std::max<uint64_t>(1, (n + tpb - 1) / tpb)); }

int grid_for(const void *fn, size_t smem, int tpb) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, fn, tpb, smem);
  return std::max(1, sms * std::max(1, per));
}

// Blocks of k_extend / k_shadow: the resident ones take their rays from a counter (dynamic
// fetching); with one ray per thread up to eight times as many, so that blocks whose rays
// end early make room for others (resident blocks alone, which stride over the queue: box
// path frame 605 us for 597, small-batch pass 1.80 ms for 1.77).
inline int walk_grid(Walk walk, const void *fn, size_t smem, int tpb) {
  return (walk == kWalkStatic ? 8 : 1) * grid_for(fn, smem, tpb);
}

}  // namespace
}  // namespace ckr
