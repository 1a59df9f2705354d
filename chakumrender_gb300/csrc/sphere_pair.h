// sphere_pair.h — the sphere's roots in pairs of FP32 numbers (usable from device and
// host code).
//
// Sphere::intersect (src/geometryPrimitives.cpp:12-27) is FP64, and FP64 runs at 1.6
// lanes per clock and SM on this part (an FP32 multiply-add at 122): one FP64 test held
// its SM for about 900 cycles per warp and was most of the closest-hit time of scenes
// with spheres.  Here the same quantities are pairs hi + lo of FP32 numbers (Dekker 1971,
// Knuth's two-sum, products by fused multiply-add), about 150 FP32 operations, with a
// bound on their error.  The result -- miss or hit, the root rounded to FP32, and the
// side the root lies on -- is used only where the bound shows it to be the one FP64
// gives; otherwise the caller runs the FP64 test (about one in 1,200 of the rays that
// meet a sphere at the box scene's scale).  Box path frame 0.927 -> 0.748 ms, 512-job batch
// 3.03 -> 2.31 ms.
#pragma once
#include <math.h>
#include <stdint.h>
#if defined(__CUDACC__)
#include <cuda_runtime.h>
#define CKR_SPH __host__ __device__ __forceinline__
#else
#include <cstring>
#define CKR_SPH inline
#endif

namespace ckr {

// A root: t rounded to FP32, rem the sign of (root - t); code 0: no root above eps,
// 1: hit, 2: undecided (the caller's FP64 test decides).
struct SphereRoot {
  float t, rem;
  int code;
};

namespace pair {

// Separately rounded operations, whatever the compiler's contraction setting.
CKR_SPH float add(float a, float b) {
#if defined(__CUDA_ARCH__)
  return __fadd_rn(a, b);
#else
  return a + b;
#endif
}
CKR_SPH float mul(float a, float b) {
#if defined(__CUDA_ARCH__)
  return __fmul_rn(a, b);
#else
  return a * b;
#endif
}
CKR_SPH uint32_t bits(float x) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(x);
#else
  uint32_t u;
  memcpy(&u, &x, 4);
  return u;
#endif
}
CKR_SPH float from_bits(uint32_t u) {
#if defined(__CUDA_ARCH__)
  return __uint_as_float(u);
#else
  float x;
  memcpy(&x, &u, 4);
  return x;
#endif
}

struct P2 {
  float h, l;
};
// a + b exactly (Knuth).
CKR_SPH P2 two_sum(float a, float b) {
  const float s = add(a, b), bb = add(s, -a);
  return P2{s, add(add(a, -add(s, -bb)), add(b, -bb))};
}
// x + y to about 2^-46 of |x| + |y|.
CKR_SPH P2 plus(P2 x, P2 y) {
  const P2 s = two_sum(x.h, y.h);
  const float l = add(s.l, add(x.l, y.l));
  const float h = add(s.h, l);
  return P2{h, add(l, -add(h, -s.h))};
}
// x times the FP32 number b, to about 2^-47.
CKR_SPH P2 times(P2 x, float b) {
  const float p = mul(x.h, b);
  return P2{p, fmaf(x.l, b, fmaf(x.h, b, -p))};
}
// x * x to about 2^-47.
CKR_SPH P2 square(P2 x) {
  const float p = mul(x.h, x.h);
  return P2{p, fmaf(2.0f * x.h, x.l, fmaf(x.h, x.h, -p))};
}

}  // namespace pair

// The nearest root above max(tmin, 1e-4) of the ray (o, d) and the sphere (c, r), as the
// reference's FP64 test finds it.  T bounds the squared magnitudes involved,
//   T >= (max(|c|, |o|)_inf^2 + |c - o|^2) max(1, |d|^2) + b^2 + r^2,   b = (c - o).d,
// to within its rounding.  Errors, with u = 2^-24: c - o is exact; b and its square,
// |c - o|^2 and r^2 are sums of at most three products, each within a few u^2 of its
// terms, so the discriminant is within 2^-42 T of its exact value, many times over; the
// root of the discriminant adds the derivative 1 / (2 s) of that and 2^-46 of s; the FP64
// test's own error is thousands of times smaller.  The decisions taken (sign of the
// discriminant, root above eps, rounding to FP32, side) are accepted only when they hold
// over that whole interval.
CKR_SPH SphereRoot sphere_root_pair(float ox, float oy, float oz, float dx, float dy, float dz, float cx, float cy,
                                    float cz, float r, float tmin, float T) {
  using namespace pair;
  const SphereRoot undecided{0.f, 0.f, 2};
  // Scenes of large magnitudes leave few roots decided: FP64 at once.
  if (!(T < 4096.f)) return undecided;
  const P2 px = two_sum(cx, -ox), py = two_sum(cy, -oy), pz = two_sum(cz, -oz);
  const P2 b = plus(plus(times(px, dx), times(py, dy)), times(pz, dz));
  const P2 oo = plus(plus(square(px), square(py)), square(pz));
  const P2 rr = square(P2{r, 0.f});
  const P2 det = plus(plus(square(b), P2{-oo.h, -oo.l}), rr);
  const float E = 2.2737367544323206e-13f * T;  // 2^-42 T
  if (det.h < -E) return SphereRoot{0.f, 0.f, 0};
  if (!(det.h > 4.0f * E)) return undecided;
  // s = sqrt(det): the FP32 root and one correction from the exact residual.
  const float s0 = sqrtf(det.h), inv = 0.5f / s0;
  const float res = add(fmaf(-s0, s0, det.h), det.l);
  const P2 s{s0, mul(res, inv)};
  // 2^-44 (|b| + s) + E / s: twice E / (2 s), and the pairs' own rounding.
  const float Et = fmaf(5.6843418860808015e-14f, fabsf(b.h) + s0, 2.0f * E * inv);
  const float eps = fmaxf(1e-4f, tmin);
  // The FP64 test compares with (double)1e-4 or tmin: within u of eps.
  const float slack = fmaf(eps, 1.2e-7f, Et);
  for (int k = 0; k < 2; ++k) {
    const P2 t = plus(b, k ? s : P2{-s.h, -s.l});
    if (t.h < eps - 2.0f * slack) continue;
    if (!(t.h > eps + 2.0f * slack)) return undecided;
    // t.h is the FP32 number nearest to the root unless the root may lie within Et of
    // the midpoint to a neighbour (half a unit in the last place away; a power of two
    // has a closer neighbour below).
    const uint32_t u = bits(t.h);
    const float half = from_bits((u & 0x7f800000u) - (24u << 23));
    const bool ok = (u & 0x007fffffu) != 0 && fabsf(t.l) + 2.0f * Et < half && fabsf(t.l) > 2.0f * Et;
    if (!ok) return undecided;
    return SphereRoot{t.h, t.l, 1};
  }
  return SphereRoot{0.f, 0.f, 0};
}

// The FP64 test itself.
CKR_SPH SphereRoot sphere_root_f64(float ox, float oy, float oz, float dx, float dy, float dz, float cx, float cy,
                                   float cz, float r, float tmin) {
  const double px = (double)cx - ox, py = (double)cy - oy, pz = (double)cz - oz;
  const double ex = dx, ey = dy, ez = dz;
  const double b = px * ex + py * ey + pz * ez, rr = (double)r;
  double det = b * b - (px * px + py * py + pz * pz) + rr * rr;
  if (det < 0.0) return SphereRoot{0.f, 0.f, 0};
  det = sqrt(det);
  const double eps = fmax(1e-4, (double)tmin);
  double t = b - det;
  if (!(t > eps)) {
    t = b + det;
    if (!(t > eps)) return SphereRoot{0.f, 0.f, 0};
  }
  const float f = (float)t;
  return SphereRoot{f, t < (double)f ? -1.f : t > (double)f ? 1.f : 0.f, 1};
}

}  // namespace ckr
