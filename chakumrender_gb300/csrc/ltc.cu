// ltc.cu — LTC polygon-light shading of a G-buffer (getLightFromMeshSource_Analytic,
// src/lightSources_CV.cpp:323-333, per pixel).
//
// The kernel is FP32 issue bound (per pixel and emitter triangle: three
// transformed vertices, horizon clipping, 3-4 edge integrals, for both the
// specular LTC lobe and the diffuse cosine lobe) and its lanes disagree on the
// path a triangle takes (above, below or across the horizon), so triangles across
// the horizon are queued per warp and clipped by all lanes together (k_ltc_shade).
// Blocks stride over pixels; the 64x64 LTC table is read from global memory (two entries per
// pixel), the emitters from shared memory, where each warp stages them 32 at a time (stage_list).
#include <algorithm>

#include "ckr_internal.h"
#include "ckr_rng.h"
#include "ltc_table.h"
#include "shading_device.cuh"

namespace ckr {
namespace {

// Blocks of two warps, which share nothing, at 128 registers without spills: 1024^2 pixels and 8
// quads take 238 us, with four, eight warps a block 239, 252; at ten blocks an SM 235, but 1,000 quads
// on 5,000 pixels 2.49 ms for 2.39.  Small blocks spread small images: 22 x 771 pixels on 58
// blocks of eight warps 19.8 us, on 265 blocks of two 10.2.
constexpr int kLtcTPB = 64, kLtcWarps = kLtcTPB / 32;
// Deferred triangles per warp and batch of 32 pixels (7.3 KB of shared memory per warp; 384
// entries at two blocks of 256 threads ran as 256).
constexpr uint32_t kLtcQueue = 256;
// Distances whose squares may overflow: no test of spheres.
constexpr float kLtcFar = 1e17f;

// The clipped integrals for a lane whose warp's queue is full.  Out of line: inlined
// into the classifying loop they pushed it past 128 registers (60 bytes of spills,
// 1.20 ms per 1024^2 frame against 0.84 ms).
__device__ __noinline__ float clipped_diffuse_here(F3 A, F3 B, F3 C, F3 n, F3 x) {
  return ltc_diffuse_clipped(A, B, C, n, x);
}
__device__ __noinline__ float clipped_spec_here(F3 A, F3 B, F3 C, F3 x, M3f m) {
  return ltc_spec_clipped(A, B, C, x, m);
}

// LTC table entries straight from global memory: two per pixel, through L1.
struct GlobalTable {
  const LtcEntry *t;
  SHD LtcEntry operator()(int i) const { return t[i]; }
};

// Per warp: the emitter triangles at hand (stage_list), its 32 pixels' shading frames and the
// triangles it deferred.
struct LtcWarp {
  float4 tri[32][3];         // (A, r) (B, g) (C, b)
  float4 group[32];          // a sphere around the group that starts here, its kind in the radius' low bits
  float px[32][17];          // x (3), n (3), Minv in world space (9); padded against bank conflicts
  float res[kLtcQueue][3];   // a deferred triangle's contribution, colour-weighted
  uint2 item[kLtcQueue];     // (lane | light << 5, previous item of the same lane or ~0)
};
static_assert(sizeof(LtcWarp) % 16 == 0, "the next warp's rows are 16-byte aligned");

// ---- both lobes at once -------------------------------------------------------------
// A pair of FP32 numbers in one 64-bit register pair, the specular lobe's in the low half,
// the diffuse one's in the high half: one FFMA2 does both lobes' multiply-add, each rounded
// as the scalar instruction rounds it.
using f2 = unsigned long long;
__device__ __forceinline__ f2 pk(float lo, float hi) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float lo2(f2 a) {
  return __uint_as_float((uint32_t)a);
}
__device__ __forceinline__ float hi2(f2 a) {
  return __uint_as_float((uint32_t)(a >> 32));
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
  f2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
  f2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}

// A corner of an emitter triangle as the two lobes see it: unit vectors (specular in the
// LTC's canonical space), and its height over the horizon of each (the specular one before
// normalisation, as ltc_spec_case tests it).
struct Corner {
  f2 x, y, z;
  float hs, hd;
};

__device__ __forceinline__ Corner corner(F3 P, F3 x, F3 n, const M3f &minv) {
  const F3 d = P - x, q = mul(minv, d);
  const f2 X = pk(q.x, d.x), Y = pk(q.y, d.y), Z = pk(q.z, d.z);
  // dot() and normalize(), pairwise and in their order of rounding: the edge factor
  // amplifies a last bit of these where an edge passes close to the point.
  const f2 nn = fma2(Z, Z, fma2(X, X, mul2(Y, Y)));
  const f2 r = pk(rsqrtf(lo2(nn)), rsqrtf(hi2(nn)));
  Corner c;
  c.x = mul2(X, r);
  c.y = mul2(Y, r);
  c.z = mul2(Z, r);
  c.hs = q.z;
  c.hd = dot(f3(hi2(c.x), hi2(c.y), hi2(c.z)), n);
  return c;
}

// theta_over_sin's coefficients, negated, in pairs.
__constant__ float2 c_theta[10] = {
    {-1.570796251296997f, -1.570796251296997f},
    {0.9999964833259583f, 0.9999964833259583f},
    {-0.7852754592895508f, -0.7852754592895508f},
    {0.6649839878082275f, 0.6649839878082275f},
    {-0.5770568251609802f, -0.5770568251609802f},
    {0.48246079683303833f, 0.48246079683303833f},
    {-0.35151180624961853f, -0.35151180624961853f},
    {0.19518974423408508f, 0.19518974423408508f},
    {-0.06951962411403656f, -0.06951962411403656f},
    {0.011529042385518551f, 0.011529042385518551f}};

// The edge integrals of both lobes (integrate_edge_z, integrate_edge; theta_over_sin's
// polynomial in pairs).
__device__ __forceinline__ void edge2(const Corner &a, const Corner &b, F3 n, float &s, float &d) {
  const f2 cc = fma2(a.z, b.z, fma2(a.x, b.x, mul2(a.y, b.y)));
  const float cs = lo2(cc), cd = hi2(cc);
  const float us = fminf(fabsf(cs), 1.0f), ud = fminf(fabsf(cd), 1.0f);
  const f2 u = pk(us, ud);
  const f2 *k = reinterpret_cast<const f2 *>(c_theta);
  f2 g = k[9];  // the negated polynomial
#pragma unroll
  for (int i = 8; i >= 0; --i) g = fma2(g, u, k[i]);
  // Both cases of theta_over_sin: some lane of a warp nearly always has an obtuse angle.
  const f2 one = pk(1.0f, 1.0f), q = mul2(fma2(u, pk(-1.0f, -1.0f), one), fma2(u, one, one));
  const f2 obtuse = fma2(pk(kPi, kPi), pk(rsqrtf(lo2(q)), rsqrtf(hi2(q))), g);
  const float gs = cs >= 0.0f ? -lo2(g) : lo2(obtuse), gd = cd >= 0.0f ? -hi2(g) : hi2(obtuse);
  const float ax = hi2(a.x), ay = hi2(a.y), az = hi2(a.z), bx = hi2(b.x), by = hi2(b.y), bz = hi2(b.z);
  s = (lo2(a.x) * lo2(b.y) - lo2(a.y) * lo2(b.x)) * gs;
  d = dot(cross(f3(ax, ay, az), f3(bx, by, bz)), n) * gd;
}

// Least and greatest of three numbers, NaN if one is.
__device__ __forceinline__ float min3_nan(float a, float b, float c) {
  float r;
  asm("{\n\t.reg .f32 t;\n\tmin.NaN.f32 t, %1, %2;\n\tmin.NaN.f32 %0, t, %3;\n\t}" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
  float r;
  asm("{\n\t.reg .f32 t;\n\tmax.NaN.f32 t, %1, %2;\n\tmax.NaN.f32 %0, t, %3;\n\t}" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// Whether two corners of the emitter list are the same point.
__device__ __forceinline__ bool same(F3 a, F3 b) { return a.x == b.x && a.y == b.y && a.z == b.z; }

// One emitter triangle and its radiance.
struct LtcTri {
  F3 A, B, C, col;
};
__device__ __forceinline__ LtcTri global_tri(const float *tri9, const float *rgb, uint32_t k) {
  const float *t = tri9 + 9 * (size_t)k, *c = rgb + 3 * (size_t)k;
  return {f3(__ldg(t), __ldg(t + 1), __ldg(t + 2)), f3(__ldg(t + 3), __ldg(t + 4), __ldg(t + 5)),
          f3(__ldg(t + 6), __ldg(t + 7), __ldg(t + 8)), f3(__ldg(c), __ldg(c + 1), __ldg(c + 2))};
}
__device__ __forceinline__ LtcTri staged_tri(const LtcWarp &W, uint32_t j) {
  const float4 a = W.tri[j][0], b = W.tri[j][1], c = W.tri[j][2];
  return {f3(a.x, a.y, a.z), f3(b.x, b.y, b.z), f3(c.x, c.y, c.z), f3(a.w, b.w, c.w)};
}
__device__ __forceinline__ void put_tri(LtcWarp &W, uint32_t j, const LtcTri &t) {
  W.tri[j][0] = make_float4(t.A.x, t.A.y, t.A.z, t.col.x);
  W.tri[j][1] = make_float4(t.B.x, t.B.y, t.B.z, t.col.y);
  W.tri[j][2] = make_float4(t.C.x, t.C.y, t.C.z, t.col.z);
}

// Kinds of groups: a triangle alone; two that share the edge from their first corner, staged as
// (a, p, m), (a, m, q); the same, which the list holds in the other order.
constexpr uint32_t kAlone = 0, kPair = 1, kPairSwapped = 3;

// Stages the triangles [from, from + 32) of the list of n in the warp's shared memory and
// takes them apart into groups: from the first on, a triangle and the next are a pair if they share
// the edge.  Returns where the next stage starts: a last triangle with more to come after it may be
// the first of a pair.  t: this lane's triangle, from + lane.  All lanes must call.  Taken apart here, and with pairs in one order, the
// shading loop has no corners to compare and to choose: 8 quads 245.9 -> 238.1 us (1024^2 pixels), 1,000
// quads 2.63 -> 2.39 ms (5,000 pixels), one quad 65.7 -> 63.9 us.  16 triangles that share no edge
// 270 -> 275.
__device__ __forceinline__ uint32_t stage_list(LtcWarp &W, LtcTri t, uint32_t from, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31u, held = min(32u, n - from);
  LtcTri u{};
  __syncwarp();
  if (lane < held) put_tri(W, lane, t);
  __syncwarp();
  uint32_t kind = kAlone;
  if (lane + 1 < held) {
    u = staged_tri(W, lane + 1);
    if (same(t.A, u.A)) kind = same(t.C, u.B) ? kPair : same(t.B, u.C) ? kPairSwapped : kAlone;
  }
  // The second of a pair starts none: the lanes ahead that could start one alternate.
  const uint32_t could = __ballot_sync(0xffffffffu, kind != kAlone);
  const uint32_t other = ~could & ((1u << lane) - 1u);  // lanes ahead that could not
  const bool second = (__clz(other) - (32u - lane)) & 1u;
  if (second) kind = kAlone;
  __syncwarp();  // all have read the next one's row
  if (kind == kPairSwapped) {
    put_tri(W, lane, u);
    put_tri(W, lane + 1, t);
  }
  // A sphere around the group about its corners' mean; its radius is infinite where a colour is
  // not finite (whose product with a zero is not zero).
  const F3 q = kind == kAlone ? t.A : kind == kPair ? u.C : u.B;
  const F3 c = (t.A + t.B + t.C + q) * 0.25f;
  auto d2 = [&](F3 p) { return dot(p - c, p - c); };
  const float rr = max3_nan(max3_nan(d2(t.A), d2(t.B), d2(t.C)), d2(q), 1e-32f);
  const float r = 1.00001f * rr * rsqrtf(rr);
  float sum = fabsf(t.col.x) + fabsf(t.col.y) + fabsf(t.col.z);
  if (kind != kAlone) sum += fabsf(u.col.x) + fabsf(u.col.y) + fabsf(u.col.z);
  const float w = r < kLtcFar && sum < 3e38f ? r : __int_as_float(0x7f800000);
  W.group[lane] = make_float4(c.x, c.y, c.z, __uint_as_float((__float_as_uint(w) & ~3u) | kind));
  __syncwarp();
  return from + held < n ? from + 31u : n;
}

// getLightFromMeshSource_Analytic per pixel, one pixel per lane.  Per emitter
// triangle and lobe a lane settles the triangles wholly above or below its horizon
// at once; a triangle across the horizon (clipping, four edge integrals) is queued,
// and the warp then works through its queue with every lane busy instead of letting
// the few lanes that clip hold up the rest.  Each lane adds its queued terms in a
// fixed order (newest first), so the result does not depend on scheduling.  A full
// queue falls back to clipping in place.
// FP32 issue bound.  The two lobes run in pairs (FFMA2, above), and two consecutive
// triangles that share the edge from their first corner, (a, p, m) and (a, m, q) in either
// order -- a quad, a fan; what polygon emitters are made of -- take their common corners and
// edge once: 4 corners and 5 edges instead of 6 and 6.  The test is the same for all lanes.
// Triangles across the horizon are queued by lobe, so that a warp clips one lobe at a time,
// and clipped without branches (clip_edges); with one mixed queue and a branch per crossed
// edge the clipping was half of all instructions.  1024^2 pixels, 8 quads: 370 -> 246 us,
// warp instructions 344 M -> 249 M, active lanes 20.0 -> 26.7; 238 us with the list taken apart as
// it is staged (stage_list).
template <bool FITS>
__global__ void __launch_bounds__(kLtcTPB, 8) k_ltc_shade(const float4 *__restrict__ gbuf, uint32_t npx,
                                                       const float *__restrict__ light_tri9,
                                                       const float *__restrict__ light_rgb, uint32_t nlight,
                                                       float *__restrict__ rgb, const LtcEntry *__restrict__ table) {
  extern __shared__ __align__(16) unsigned char ltc_smem[];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  LtcWarp &W = reinterpret_cast<LtcWarp *>(ltc_smem)[warp];
  const GlobalTable tab{table};
  // A list that fits stays staged; its queue items hold staged places, those of a longer one
  // places in the list.
  auto fetch = [&](uint32_t k) {
    if constexpr (FITS) return staged_tri(W, k);
    else return global_tri(light_tri9, light_rgb, k);
  };
  auto lane_tri = [&](uint32_t k) {
    return k + lane < nlight ? global_tri(light_tri9, light_rgb, k + lane) : LtcTri{};
  };
  uint32_t from = 0, to = 0;  // triangles at hand
  const float inv2pi = 1.0f / (2.0f * kPi);
  const uint32_t stride = gridDim.x * (uint32_t)kLtcTPB;
  for (uint32_t base = (blockIdx.x * kLtcWarps + warp) * 32u; base < npx;
       base = npx - base > stride ? base + stride : npx) {
    const uint32_t p = base + lane;
    const bool active = p < npx;
    F3 x = f3(0, 0, 0), n = f3(0, 0, 1);
    M3f minv{};
    float amp = 0.f, spec = 0.f;
    // The list's first triangles load while the pixel's rows and table entries do (35 x 45
    // pixels, 11 quads: 16.8 us without, 16.5 with).
    const bool stage = !FITS || to == 0;
    LtcTri first{};
    if (stage) first = lane_tri(0);
    if (active) {
      const float4 g0 = gbuf[3 * (size_t)p], g1 = gbuf[3 * (size_t)p + 1], g2 = gbuf[3 * (size_t)p + 2];
      x = f3(g0.x, g0.y, g0.z);
      n = f3(g1.x, g1.y, g1.z);
      const F3 wo = f3(g2.x, g2.y, g2.z);
      const float theta = acosf(fminf(1.0f, fmaxf(-1.0f, dot(n, wo))));
      const LtcLookup L = ltc_lookup(tab, theta, g0.w);
      minv = ltc_minv_world(L, n, wo);
      amp = L.amp;
      spec = g2.w;
    }
    float *mine = W.px[lane];
    mine[0] = x.x; mine[1] = x.y; mine[2] = x.z;
    mine[3] = n.x; mine[4] = n.y; mine[5] = n.z;
    for (int i = 0; i < 9; ++i) mine[6 + i] = minv.a[i];
    float s3[3] = {0.f, 0.f, 0.f}, d3[3] = {0.f, 0.f, 0.f};
    // Queued triangles: specular ones from the front, diffuse ones from the back, so that a
    // warp clips one lobe at a time.  The counts are the same in every lane.
    uint32_t head = ~0u, count[2] = {0, 0};
    // Adds triangle k: the lobes' integrals `is`, `id` if it is above their horizon; across
    // it, its queue entries.
    auto add = [&](uint32_t k, F3 col, const Corner &a, const Corner &b, const Corner &c, float is, float id) {
      const float r = col.x, g = col.y, bl = col.z;
      // A NaN height is neither above nor below: queued.
      const bool us = min3_nan(a.hs, b.hs, c.hs) > 0.f, ud = min3_nan(a.hd, b.hd, c.hd) > 0.f;
      const float s = us ? fabsf(is) : 0.f, d = ud ? fabsf(id) : 0.f;
      s3[0] += r * s; s3[1] += g * s; s3[2] += bl * s;
      d3[0] += r * d; d3[1] += g * d; d3[2] += bl * d;
      const bool qs = active && !us && !(max3_nan(a.hs, b.hs, c.hs) < 0.f);
      const bool qd = active && !ud && !(max3_nan(a.hd, b.hd, c.hd) < 0.f);
#pragma unroll
      for (uint32_t lobe = 0; lobe < 2; ++lobe) {
        const bool want = lobe ? qd : qs;
        const unsigned m = __ballot_sync(0xffffffffu, want);
        if (m == 0) continue;
        const uint32_t rank = count[lobe] + (uint32_t)__popc(m & ((1u << lane) - 1u));
        if (want) {
          if (rank + count[lobe ^ 1u] < kLtcQueue) {
            const uint32_t slot = lobe ? kLtcQueue - 1u - rank : rank;
            W.item[slot] = make_uint2(lane | k << 5, head);
            head = slot;
          } else {
            const LtcTri t = fetch(k);
            const float v = lobe ? clipped_diffuse_here(t.A, t.B, t.C, n, x) : clipped_spec_here(t.A, t.B, t.C, x, minv);
            float *acc = lobe ? d3 : s3;
            acc[0] += r * v; acc[1] += g * v; acc[2] += bl * v;
          }
        }
        count[lobe] = min(count[lobe] + (uint32_t)__popc(m), kLtcQueue - count[lobe ^ 1u]);
      }
    };
    // Surfaces that face away from an emitter: a group whose sphere is below both horizons of
    // every lane adds nothing and is passed over.  Below by a margin several times the rounding of
    // these sums and of `corner`, so that the corners' own heights come out negative.  A floor of
    // 1024^2 pixels with 8 quads, all below it 167 -> 60 us, half of them 160 -> 101, all above 160
    // -> 153 (with a branch per lane ahead of each triangle's edges 118, 154, 201; with a vote on the
    // corners 101, 131, 168).
    const F3 z = f3(minv.a[6], minv.a[7], minv.a[8]);
    const float n2 = dot(n, n), z2 = dot(z, z);
    float nn = n2 * rsqrtf(n2) * 1.00001f, nz = z2 * rsqrtf(z2) * 1.00001f;
    if (!active) nn = nz = __int_as_float(0xff800000);  // -inf: below
    if (stage) {
      from = 0;
      to = stage_list(W, first, 0, nlight);
    }
    for (uint32_t k = 0; k < nlight;) {
      if (!FITS && k >= to) {
        from = k;
        to = stage_list(W, lane_tri(k), k, nlight);
      }
      const uint32_t j = k - from;
      const float4 g = W.group[j];
      const uint32_t kind = __float_as_uint(g.w) & 3u;
      const F3 l = f3(g.x, g.y, g.z) - x;
      const float l1 = fabsf(l.x) + fabsf(l.y) + fabsf(l.z), m = fmaf(4e-6f, l1, g.w);
      const float hs = fmaf(z.x, l.x, fmaf(z.y, l.y, fmaf(z.z, l.z, nz * m)));
      const float hd = fmaf(n.x, l.x, fmaf(n.y, l.y, fmaf(n.z, l.z, nn * m)));
      const uint32_t k0 = k;
      k += kind ? 2 : 1;
      if (__all_sync(0xffffffffu, max3_nan(hs, hd, l1 - kLtcFar) < 0.f)) continue;
      const uint32_t back = FITS ? 0u : kind >> 1;  // the list's order of a staged pair
      const LtcTri t = staged_tri(W, j);
      const Corner a = corner(t.A, x, n, minv), b = corner(t.B, x, n, minv), c = corner(t.C, x, n, minv);
      float s0, d0, s1, d1, sm, dm;
      edge2(a, b, n, s0, d0);
      edge2(b, c, n, s1, d1);
      edge2(c, a, n, sm, dm);
      add(k0 + back, t.col, a, b, c, s0 + s1 + sm, d0 + d1 + dm);
      if (kind) {
        const LtcTri u = staged_tri(W, j + 1);
        const Corner q = corner(u.C, x, n, minv);
        edge2(c, q, n, s0, d0);
        edge2(q, a, n, s1, d1);
        add(k0 + 1 - back, u.col, a, c, q, s0 + s1 - sm, d0 + d1 - dm);
      }
    }
    __syncwarp();
    // The warp's queued triangles, every lane taking the next one.
#pragma unroll
    for (uint32_t lobe = 0; lobe < 2; ++lobe)
      for (uint32_t i = lane; i < count[lobe]; i += 32) {
        const uint32_t slot = lobe ? kLtcQueue - 1u - i : i;
        const uint2 it = W.item[slot];
        const uint32_t k = it.x >> 5;
        const float *q = W.px[it.x & 31u];
        const LtcTri t = fetch(k);
        const F3 qx = f3(q[0], q[1], q[2]);
        float v;
        if (lobe) {
          v = ltc_diffuse_clipped(t.A, t.B, t.C, f3(q[3], q[4], q[5]), qx);
        } else {
          M3f qm;
          for (int j = 0; j < 9; ++j) qm.a[j] = q[6 + j];
          v = ltc_spec_clipped(t.A, t.B, t.C, qx, qm);
        }
        W.res[slot][0] = t.col.x * v;
        W.res[slot][1] = t.col.y * v;
        W.res[slot][2] = t.col.z * v;
      }
    __syncwarp();
    for (uint32_t i = head; i != ~0u; i = W.item[i].y) {
      if (i >= count[0]) {
        for (int j = 0; j < 3; ++j) d3[j] += W.res[i][j];
      } else {
        for (int j = 0; j < 3; ++j) s3[j] += W.res[i][j];
      }
    }
    if (active)
      for (int j = 0; j < 3; ++j) rgb[3 * (size_t)p + j] = s3[j] * inv2pi * amp * spec + d3[j] * inv2pi * (1.0f - spec);
    __syncwarp();  // the next batch reuses the warp's shared memory
  }
}

// ---- Monte Carlo reference for the LTC integral -----------------------------------
// Per pixel, the integral over the emitter triangles of brdf x cos x radiance,
// treating the emitters as the LTC integral does: two-sided and unoccluded, a
// direction that crosses several emitters collecting each one's radiance.
// Half of the samples pick an emitter point by area, half sample the BRDF
// (getBrdfDirectionSampleRandomized); both are weighted by the balance heuristic,
// f cos L / (n_a p_area(w) + n_b p_brdf(w)) with p_area(w) = sum over the
// emitters w crosses of t^2 / (A_total |cos_l|).  Sums are FP64 per pixel.

constexpr int kMcTPB = 128;
constexpr uint32_t kMcMaxLights = 256;

// Two-sided ray/triangle distance (Moller & Trumbore 1997); 0 on a miss.
__device__ __forceinline__ float emitter_t(F3 o, F3 w, F3 a, F3 e1, F3 e2) {
  F3 p = cross(w, e2);
  float det = dot(e1, p);
  if (fabsf(det) < 1e-20f) return 0.f;
  float inv = 1.0f / det;
  F3 tv = o - a;
  float u = dot(tv, p) * inv;
  if (u < 0.f || u > 1.f) return 0.f;
  F3 q = cross(tv, e1);
  float v = dot(w, q) * inv;
  if (v < 0.f || u + v > 1.f) return 0.f;
  float t = dot(e2, q) * inv;
  return t > 0.f ? t : 0.f;
}

__global__ void __launch_bounds__(kMcTPB) k_ltc_mc(const float4 *__restrict__ gbuf, uint32_t npx,
                                                   const float *__restrict__ light_tri9,
                                                   const float *__restrict__ light_rgb, uint32_t nlight, uint32_t spp,
                                                   uint64_t seed, int fresnel, double *__restrict__ rgb) {
  __shared__ float4 s_a[kMcMaxLights], s_e1[kMcMaxLights], s_e2[kMcMaxLights];  // .w: r, g, b
  __shared__ float4 s_n[kMcMaxLights];  // unit normal, 1 / A_total
  __shared__ float s_cdf[kMcMaxLights];
  for (uint32_t k = threadIdx.x; k < nlight; k += kMcTPB) {
    const float *t = light_tri9 + 9 * (size_t)k;
    F3 a = f3(t[0], t[1], t[2]), b = f3(t[3], t[4], t[5]), c = f3(t[6], t[7], t[8]);
    F3 e1 = b - a, e2 = c - a, nn = cross_rn(e1, e2);
    float len = length(nn);
    s_a[k] = make_float4(a.x, a.y, a.z, light_rgb[3 * k]);
    s_e1[k] = make_float4(e1.x, e1.y, e1.z, light_rgb[3 * k + 1]);
    s_e2[k] = make_float4(e2.x, e2.y, e2.z, light_rgb[3 * k + 2]);
    F3 un = len > 0.f ? nn * (1.0f / len) : f3(0.f, 0.f, 0.f);
    s_n[k] = make_float4(un.x, un.y, un.z, 0.f);
    s_cdf[k] = 0.5f * len;  // area, turned into the CDF below
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float total = 0.f;
    for (uint32_t k = 0; k < nlight; ++k) total += s_cdf[k];
    float run = 0.f;
    for (uint32_t k = 0; k < nlight; ++k) {
      run += s_cdf[k];
      s_cdf[k] = run / total;
      s_n[k].w = 1.0f / total;
    }
  }
  __syncthreads();
  const uint32_t p = blockIdx.x * kMcTPB + threadIdx.x;
  if (p >= npx) return;
  float4 g0 = gbuf[3 * (size_t)p], g1 = gbuf[3 * (size_t)p + 1], g2 = gbuf[3 * (size_t)p + 2];
  F3 x = f3(g0.x, g0.y, g0.z), n = f3(g1.x, g1.y, g1.z), wo = f3(g2.x, g2.y, g2.z);
  Material M;
  M.brdf = kGGX;
  M.alpha = g0.w;
  M.phong_exp = 0.f;
  M.spec = g2.w;
  float sf = sqrtf(g1.w);
  M.int_ior = fresnel ? (1.0f + sf) / (1.0f - sf) : 1e5f;
  M.ext_ior = 1.0f;
  F3 wo_ref = normalize(n * (2.0f * dot(n, wo)) - wo);
  const uint64_t key = ckr_key(seed, p);
  const float half = 0.5f * (float)spp;
  double acc0 = 0.0, acc1 = 0.0, acc2 = 0.0;
  for (uint32_t s = 0; s < spp; ++s) {
    float e0 = ckr_draw_f(key, 4 * s), e1 = ckr_draw_f(key, 4 * s + 1), e2 = ckr_draw_f(key, 4 * s + 2);
    F3 w;
    if ((s & 1u) == 0) {
      uint32_t k = 0;
      while (k + 1 < nlight && s_cdf[k] <= e0) ++k;
      float4 a = s_a[k], u = s_e1[k], v = s_e2[k];
      F3 A = f3(a.x, a.y, a.z);
      F3 P = sample_triangle(A, A + f3(u.x, u.y, u.z), A + f3(v.x, v.y, v.z), e1, e2);
      w = normalize(P - x);
    } else {
      w = sample_brdf(M, n, wo_ref, wo, e0, e1, e2);
    }
    float c = dot(w, n);
    if (!(c > 0.f)) continue;
    float pa = 0.f, L0 = 0.f, L1 = 0.f, L2 = 0.f;
    for (uint32_t k = 0; k < nlight; ++k) {
      float4 a = s_a[k], u = s_e1[k], v = s_e2[k];
      float t = emitter_t(x, w, f3(a.x, a.y, a.z), f3(u.x, u.y, u.z), f3(v.x, v.y, v.z));
      if (t > 0.f) {
        float4 un = s_n[k];
        float cl = fabsf(un.x * w.x + un.y * w.y + un.z * w.z);
        pa += t * t * un.w / cl;
        L0 += a.w;
        L1 += u.w;
        L2 += v.w;
      }
    }
    if (!(pa > 0.f)) continue;
    float f = brdf_eval(M, n, wo_ref, wo, w);
    float pb = pdf_eval(M, n, wo_ref, wo, w);
    float wgt = f * c / (half * (pa + pb));
    if (!(wgt < 3.0e38f)) continue;
    acc0 += (double)(L0 * wgt);
    acc1 += (double)(L1 * wgt);
    acc2 += (double)(L2 * wgt);
  }
  rgb[3 * (size_t)p] = acc0;
  rgb[3 * (size_t)p + 1] = acc1;
  rgb[3 * (size_t)p + 2] = acc2;
}

}  // namespace
}  // namespace ckr

using namespace ckr;

extern "C" int ckr_ltc_shade(const float *gbuf, uint32_t npx, const float *light_tri9, const float *light_rgb,
                             uint32_t nlight, float *rgb, void *stream) {
  if ((npx && (!gbuf || !rgb)) || (nlight && (!light_tri9 || !light_rgb)) || ((uintptr_t)gbuf & 15u))
    return CKR_ERR_INVALID_ARGUMENT;
  if (npx == 0) return CKR_OK;
  int st = CKR_OK;
  const LtcEntry *table = device_ltc_table(&st);
  if (!table) return st;
  if (nlight >= (1u << 26)) return CKR_ERR_TOO_LARGE;  // light index in a queue item
  const size_t smem = kLtcWarps * sizeof(LtcWarp);
  const auto fn = nlight <= 32 ? k_ltc_shade<true> : k_ltc_shade<false>;
  static bool attr_set[64] = {false};
  int dev = 0, sms = 0, per_sm = 0;
  CKR_CUDA_TRY(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    for (const void *k : {(const void *)k_ltc_shade<true>, (const void *)k_ltc_shade<false>})
      CKR_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    attr_set[dev] = true;
  }
  CKR_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  CKR_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kLtcTPB, smem));
  if (per_sm < 1) return CKR_ERR_CUDA;
  // Two tiles of pixels to a block once there are more than the resident blocks hold: the
  // tiles' work differs (how many triangles are clipped), and blocks that stride over 13 tiles
  // each end far apart.  1024^2 pixels, 8 quads: resident blocks alone 241.5 us, blocks of four
  // tiles 249, two 238, one (each staging the emitters) 240.  Up to eight triangles staging weighs more:
  // resident blocks alone 63.9 us for 67.7 at one quad, 136.5 for 137.6 at four.
  const uint64_t tiles = ceil_div(npx, kLtcTPB);
  const int grid = (int)std::max(std::min(tiles, (uint64_t)sms * per_sm), nlight > 8 ? tiles / 2 : 0);
  fn<<<grid, kLtcTPB, smem, (cudaStream_t)stream>>>(reinterpret_cast<const float4 *>(gbuf), npx, light_tri9, light_rgb,
                                                    nlight, rgb, table);
  CKR_CUDA_TRY(cudaGetLastError());
  return CKR_OK;
}

extern "C" int ckr_ltc_mc(const float *gbuf, uint32_t npx, const float *light_tri9, const float *light_rgb,
                          uint32_t nlight, uint32_t spp, uint64_t seed, int fresnel, double *rgb, void *stream) {
  if ((npx && (!gbuf || !rgb)) || !light_tri9 || !light_rgb || nlight == 0 || ((uintptr_t)gbuf & 15u) ||
      spp == 0 || (spp & 1u) || spp > (1u << 28))
    return CKR_ERR_INVALID_ARGUMENT;
  if (nlight > kMcMaxLights) return CKR_ERR_TOO_LARGE;
  if (npx == 0) return CKR_OK;
  k_ltc_mc<<<(unsigned)ceil_div(npx, kMcTPB), kMcTPB, 0, (cudaStream_t)stream>>>(
      reinterpret_cast<const float4 *>(gbuf), npx, light_tri9, light_rgb, nlight, spp, seed, fresnel, rgb);
  CKR_CUDA_TRY(cudaGetLastError());
  return CKR_OK;
}
