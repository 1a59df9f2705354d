// mlp.cu — the learned light-selection network on the fifth-generation tensor
// cores: inference over the renderer's queue (k_mlp_infer) and on records
// (k_mlp_infer_rec), training forward + backward (k_mlp_train) and the Adam update
// (k_mlp_adam), all for tiles of 128 rows.
//
// In inference a group of 128 threads owns a tile: thread t computes row t's features and
// epilogues; in training a block of 256 does, two threads a row.  One thread issues the
// tcgen05.mma chain of each layer (M = 128 rows,
// N = 64 outputs, K = 96, or 80 for the hidden layers whose operands carry a
// constant 1 that multiplies the bias) into tensor memory and commits it to an
// mbarrier that the group waits on with a bounded poll.  Row t of the
// accumulator lives in TMEM lane t, which warp (t / 32) % 4 reads with
// tcgen05.ld.  Groups of a CTA share the weights, and one's epilogue overlaps the others'
// MMAs: two groups over the renderer's queue, seven on records.
//
// Backward pass, per layer l with input activations X (rows b) and output
// gradient G (rows b):  dW^T = X^T G  (M = input features padded to 128,
// N = 64, K = the 128 rows of the tile), accumulated in TMEM across all tiles a
// CTA processes, and dX = G W  (M = 128 rows, N = 64, K = 64) for the layer
// below.  X^T and G^T are X and G read as MN-major operands.  Column 64 of X is all
// ones, so row 64 of dW^T is the bias gradient (the first layer's bias is the weight of
// its constant feature).
//
// Bounds: every mbarrier wait gives up after kWaitTries polls, records
// CKR_ERR_ITERATION_LIMIT, waits once more (bounded) for the MMAs in flight,
// frees the CTA's tensor memory and returns.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <utility>
#include <vector>

#include "ckr_internal.h"
#include "ckr_rng.h"
#include "mlp.h"
#include "render_device.cuh"
#include "tc05.cuh"

namespace ckr {
namespace mlp {
namespace {

constexpr uint32_t kWaitTries = 1u << 22;
constexpr uint32_t kIdesc = tc::idesc_bf16(128, 64), kIdescT = tc::idesc_bf16(128, 64, true);

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t *>(&h);
}
__device__ __forceinline__ float bf16_lo(uint32_t u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t u) { return __uint_as_float(u & 0xFFFF0000u); }

// Writes 8 consecutive K entries (k0 % 8 == 0) of row r of a K-major operand.
__device__ __forceinline__ void st8(uint8_t *op, uint32_t r, uint32_t k0, uint32_t K, const float *v) {
  uint4 q = make_uint4(pack_bf16(v[0], v[1]), pack_bf16(v[2], v[3]), pack_bf16(v[4], v[5]), pack_bf16(v[6], v[7]));
  *reinterpret_cast<uint4 *>(op + tc::kmaj(r, k0, K)) = q;
}
__device__ __forceinline__ void ld8(const uint8_t *op, uint32_t r, uint32_t k0, uint32_t K, float *v) {
  uint4 q = *reinterpret_cast<const uint4 *>(op + tc::kmaj(r, k0, K));
  v[0] = bf16_lo(q.x); v[1] = bf16_hi(q.x); v[2] = bf16_lo(q.y); v[3] = bf16_hi(q.y);
  v[4] = bf16_lo(q.z); v[5] = bf16_hi(q.z); v[6] = bf16_lo(q.w); v[7] = bf16_hi(q.w);
}
// Rows to process: n_max, or what the device count leaves after n_off.
__device__ __forceinline__ uint32_t rows(uint32_t n_max, const uint32_t *n_dev, uint32_t n_off) {
  if (!n_dev) return n_max;
  const uint32_t c = *n_dev;
  return c > n_off ? min(c - n_off, n_max) : 0u;
}

struct Params {
  float cx, cy, cz, scale;
  uint32_t nclusters;
  // Test hook: when non-zero, the first layer's MMAs are not issued and every
  // mbarrier wait gives up after this many polls (a phase nothing completes).
  uint32_t stall_tries;
};

// Row features into the first-layer operand (K = 96): the 8-feature groups of PART 0 (the
// first two coordinates), 1 (the third and the rest) or 2 (all).
template <int PART = 2>
__device__ __forceinline__ void write_features(uint8_t *x0, uint32_t t, float4 r0, float4 r1, float4 r2,
                                               const Params &p) {
  float f[kIn];
  const float pc[3] = {(r0.x - p.cx) * p.scale, (r0.y - p.cy) * p.scale, (r0.z - p.cz) * p.scale};
  // sin, cos of 2^k pi p: the base frequency, then the double-angle recurrences
  // sin 2a = 2 sin a cos a, cos 2a = (cos a - sin a)(cos a + sin a); the error
  // (about 1e-6 at the base) roughly doubles per octave, a few 1e-3 after eleven,
  // at the level of BF16's rounding of the features.
#pragma unroll
  for (int c = PART == 1 ? 2 : 0; c < (PART == 0 ? 2 : 3); ++c) {
    float sn, cs;
    __sincosf(3.14159265358979f * pc[c], &sn, &cs);  // |argument| <= pi inside the scene box
#pragma unroll
    for (int k = 0; k < (int)kFreqs; ++k) {
      f[24 * c + 2 * k] = sn;
      f[24 * c + 2 * k + 1] = cs;
      const float s2 = 2.0f * sn * cs;
      cs = (cs - sn) * (cs + sn);
      sn = s2;
    }
  }
  f[72] = r1.x; f[73] = r1.y; f[74] = r1.z;
  f[75] = r2.x; f[76] = r2.y; f[77] = r2.z;
  f[78] = r0.w;
  f[79] = 1.0f;
#pragma unroll
  for (int j = 80; j < (int)kIn; ++j) f[j] = 0.f;
#pragma unroll
  for (int q = PART == 1 ? 6 : 0; q < (PART == 0 ? 6 : (int)kIn / 8); ++q) st8(x0, t, 8 * q, kIn, f + 8 * q);
}

// Two FP32 values to a BF16 pair with ReLU (lower half = first value).
__device__ __forceinline__ uint32_t pack_relu_bf16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// Accumulator row t (64 columns, bias included by the MMA) through ReLU into row t
// of a hidden-layer operand (K = 80): columns 0..63, then the constant 1 at 64 and
// zeros to 79.
__device__ __forceinline__ void epilogue_relu(uint32_t taddr, uint8_t *dst, uint32_t t, int h0 = 0, int h1 = 2) {
#pragma unroll 2
  for (int h = h0; h < h1; ++h) {
    float v[32];
    tc::tmem_ld32(taddr + 32 * h, v);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float *x = v + 8 * q;
      *reinterpret_cast<uint4 *>(dst + tc::kmaj(t, 32 * h + 8 * q, kHidK)) =
          make_uint4(pack_relu_bf16(x[0], x[1]), pack_relu_bf16(x[2], x[3]), pack_relu_bf16(x[4], x[5]),
                     pack_relu_bf16(x[6], x[7]));
    }
  }
  if (h1 < 2) return;  // halves [h0, h1) of the columns; the constants go with the second
  *reinterpret_cast<uint4 *>(dst + tc::kmaj(t, 64, kHidK)) = make_uint4(0x3F80u, 0u, 0u, 0u);  // BF16 1.0
  *reinterpret_cast<uint4 *>(dst + tc::kmaj(t, 72, kHidK)) = make_uint4(0u, 0u, 0u, 0u);
}

// exp(z) as 2^(z log2 e), zero where that is below the normal range (the flushing form of the
// instruction).  Relative error for |z| <= 80: 2^-22 of the instruction (its PTX
// specification) and, from the product's rounding, 116 2^-24 ln 2 = 4.8e-6;
// tested through the probabilities, against FP64 (tests/test_proposal.py).
__device__ __forceinline__ float exp_ftz(float z) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__fmul_rn(z, 1.4426950408889634f)));
  return r;
}

// Terms of a softmax over 64 logits without their maximum: exp(z) with z clamped to [-80, 80],
// so that neither the terms nor their sum leave FP32's range.
__device__ __forceinline__ float exp_80(float z) { return exp_ftz(fminf(fmaxf(z, -80.f), 80.f)); }
// Whether the clamp may show in a row whose terms sum to `sum`: a logit of 80 or more
// (exp(80) = 5.5e34), or none large enough to leave those below -80 (1.8e-35) without weight.
// Such rows are taken from their maximum instead, exp(z - max), which serves all logits.
__device__ __forceinline__ bool clamped(float sum) { return !(sum > 1e-20f && sum < 5e34f); }
// A logit as those rows take it, finite: a NaN as the least.
__device__ __forceinline__ float finite_logit(float z) { return fminf(fmaxf(z, -3.0e38f), 3.0e38f); }

// exp(z) over the logits of row t when all 64 are clusters; returns the sum.
__device__ __forceinline__ float softmax_exp64(uint32_t taddr, float *p) {
  tc::tmem_ld32(taddr, p);
  tc::tmem_ld32(taddr + 32, p + 32);
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < 64; ++j) {
    p[j] = exp_80(p[j]);
    sum += p[j];
  }
  return sum;
}

// Eight probabilities in FP16: terms times `inv`.
__device__ __forceinline__ uint4 half8(const float *x, float inv) {
  __half2 h[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2half2_rn(x[2 * i] * inv, x[2 * i + 1] * inv);
  return *reinterpret_cast<uint4 *>(h);
}

// Cumulative 16-bit table of the selection mixture (1 - delta) softmax + delta / 64: entries
// j and j + 1 from the terms e, with keep = (1 - delta) / sum and `run` the sum so far.
__device__ __forceinline__ uint32_t cdf_pair(const float *e, int j, float keep, float unif, float &run) {
  run += fmaf(keep, e[j], unif);
  const uint32_t c0 = min(65535u, __float2uint_rn(65535.0f * run));
  run += fmaf(keep, e[j + 1], unif);
  const uint32_t c1 = j + 2 == 64 ? 65535u : min(65535u, __float2uint_rn(65535.0f * run));
  return c0 | (c1 << 16);
}

// The selection tables of a warp with rows that the clamp would change (`far`): those rows'
// softmaxes from their maximum, the others' as before; dst null: no row.  Out of line and in local
// memory, so that it costs the usual warp no registers (frozen learned frame of 640 x 360 x 4
// 2.07 ms with and without it, 2.08 with it in the kernel).  All lanes must call.
__device__ __noinline__ void far_cdf(uint32_t taddr, bool far, float delta, uint32_t *dst) {
  float p[64];
  tc::tmem_ld32(taddr, p);
  tc::tmem_ld32(taddr + 32, p + 32);
  float mx = -3.0e38f, sum = 0.f;
#pragma unroll 1
  for (int j = 0; j < 64; ++j) mx = fmaxf(mx, finite_logit(p[j]));
#pragma unroll 1
  for (int j = 0; j < 64; ++j) {
    p[j] = far ? exp_ftz(finite_logit(p[j]) - mx) : exp_80(p[j]);
    sum += p[j];
  }
  const float unif = delta / 64.0f, keep = (1.0f - delta) / sum;
  float run = 0.f;
#pragma unroll 1
  for (int j = 0; j < 64; j += 2) {
    const uint32_t w = cdf_pair(p, j, keep, unif, run);
    if (dst) dst[j / 2] = w;
  }
}

// exp(z - max) over the first C logits of row t (0 beyond); returns their sum.
__device__ __forceinline__ float softmax_exp(uint32_t taddr, uint32_t C, float *p) {
  tc::tmem_ld32(taddr, p);
  tc::tmem_ld32(taddr + 32, p + 32);
  float mx = -3.0e38f;
#pragma unroll
  for (int j = 0; j < 64; ++j)
    if ((uint32_t)j < C) mx = fmaxf(mx, p[j]);
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < 64; ++j) {
    p[j] = (uint32_t)j < C ? __expf(p[j] - mx) : 0.f;
    sum += p[j];
  }
  return sum;
}

__device__ __forceinline__ void issue(uint32_t d, uint32_t a, uint32_t b, uint32_t K, uint32_t accumulate_first) {
  for (uint32_t s = 0; s < K / 16; ++s)
    tc::mma_bf16(d, tc::sdesc(a, K, s), tc::sdesc(b, K, s), kIdesc, (s > 0 || accumulate_first) ? 1u : 0u);
}

// D (+)= X^T G over the 128 rows of a tile: X stored [128 x C], G [128 x 64].
__device__ __forceinline__ void issue_t(uint32_t d, uint32_t x, uint32_t C, uint32_t g, uint32_t accumulate_first) {
  for (uint32_t s = 0; s < 8; ++s)
    tc::mma_bf16(d, tc::sdesc_t(x, C, s), tc::sdesc_t(g, 64, s), kIdescT, (s > 0 || accumulate_first) ? 1u : 0u);
}

// Barrier of one 128-thread group (named barrier 1 + g; 0 is __syncthreads).
// Immediate ids, so that the kernel reserves only the barriers it uses.
__device__ __forceinline__ void group_sync(uint32_t g) {
  if (g == 0) asm volatile("bar.sync 1, 128;" ::: "memory");
  else asm volatile("bar.sync 2, 128;" ::: "memory");
}

// Every thread of the group: shared-memory writes visible to the tensor core,
// TMEM reads done before the next MMA overwrites the accumulator.
__device__ __forceinline__ void sync_for_mma(uint32_t g) {
  tc::fence_proxy_async();
  tc::fence_before_sync();
  group_sync(g);
}

// Waits for the group's committed MMAs; false (uniformly within the group) when
// the wait gave up.
__device__ __forceinline__ bool wait_mma(uint32_t g, uint32_t mbar, uint32_t &phase, int *abort, int *err,
                                         uint32_t tries = kWaitTries) {
  if (!tc::mbar_wait(mbar, phase, tries)) {
    *abort = 1;
    atomicExch(err, CKR_ERR_ITERATION_LIMIT);
  }
  group_sync(g);
  if (*abort) {
    tc::mbar_wait(mbar, phase, tries);  // let the MMAs in flight land before TMEM is freed
    return false;
  }
  phase ^= 1u;
  tc::fence_after_sync();
  return true;
}

// ---- inference ------------------------------------------------------------------
// kGroups independent 128-thread groups per CTA share the weights in shared memory;
// each owns a 128-row tile, an activation buffer, an mbarrier and 64 TMEM columns,
// so one group's epilogue overlaps another's MMAs.
constexpr uint32_t kGroups = 2, kInferTPB = 128 * kGroups;

struct SmemInfer {
  uint8_t w[kImgForward];
  uint8_t a[kGroups][128 * kIn * 2];
  uint64_t mbar[kGroups], mbar_w;
  uint32_t tmem;
  int abort[kGroups];
};

// A queue entry's path state, gathered in three dependent steps (the path slot from
// the queue, the slot's hit and ray, the hit triangle's normal and alpha) so that
// each step's latency can overlap other work of the tile before it.
struct PathGather {
  uint32_t slot, id, flags;
  float4 ro, rd;
  float t;
  float4 na;
};

__device__ __forceinline__ void gather_slot(const PathRows &pr, uint32_t row, uint32_t n, PathGather &g) {
  g.slot = row < n ? pr.queue[row] : 0xFFFFFFFFu;
}

__device__ __forceinline__ void gather_hit(const PathRows &pr, PathGather &g) {
  g.id = kMiss;
  if (g.slot == 0xFFFFFFFFu) return;
  g.id = pr.hit_id[g.slot];
  g.flags = pr.meta[g.slot].w;
  g.ro = pr.ray_o[g.slot];
  g.rd = pr.ray_d[g.slot];
  g.t = pr.hit_t[g.slot];
}

// The hit triangle's normal and material index (ShadeView::tri_nm, a third
// dependent step).
__device__ __forceinline__ void gather_na(const PathRows &pr, PathGather &g) {
  if (g.id != kMiss && !(g.id & kSphereBit)) g.na = pr.sv.tri_nm[g.id];
}

// Network input of a gathered queue entry: its shading point (zeros where the entry is
// not a shaded surface).
__device__ __forceinline__ void path_row(const PathRows &pr, const PathGather &g, float4 &r0, float4 &r1,
                                         float4 &r2) {
  r0 = r1 = r2 = make_float4(0, 0, 0, 0);
  if (g.id == kMiss || (g.flags & 1u)) return;
  if (!(g.id & kSphereBit)) {
    const ckr_material &mm = pr.sv.mats[__float_as_uint(g.na.w)];
    if (mm.light_type != 0) return;  // an emitter
    const F3 d = f3(g.rd.x, g.rd.y, g.rd.z), x = f3(g.ro.x, g.ro.y, g.ro.z) + d * g.t;
    F3 nn = f3(g.na.x, g.na.y, g.na.z);
    if (dot(d, nn) > 0.f) nn = -nn;
    r0 = make_float4(x.x, x.y, x.z, mm.alpha);
    r1 = make_float4(nn.x, nn.y, nn.z, 0.f);
    r2 = make_float4(-d.x, -d.y, -d.z, 0.f);
    return;
  }
  Surface S = make_surface(pr.sv, f3(g.ro.x, g.ro.y, g.ro.z), f3(g.rd.x, g.rd.y, g.rd.z), g.id, g.t);
  const ckr_material &mm = pr.sv.mats[S.mat];
  if (mm.light_type != 0) return;
  r0 = make_float4(S.x.x, S.x.y, S.x.z, mm.alpha);
  r1 = make_float4(S.n.x, S.n.y, S.n.z, 0.f);
  r2 = make_float4(S.wo.x, S.wo.y, S.wo.z, 0.f);
}

// The renderer's queue entries to selection CDFs.
__global__ void __launch_bounds__(kInferTPB, 2) k_mlp_infer(PathRows pr, uint32_t n_max, const uint32_t *n_dev,
                                                         const uint8_t *__restrict__ img, Params p, float delta,
                                                         uint16_t *__restrict__ cdf16, int *err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  SmemInfer &S = *reinterpret_cast<SmemInfer *>(smem_raw);
  const uint32_t g = threadIdx.x >> 7, t = threadIdx.x & 127u, warp = threadIdx.x >> 5;
  // The weights by one bulk copy, waited for before a group's first MMA.
  const uint32_t mbar = tc::smem_u32(&S.mbar[g]), mbar_w = tc::smem_u32(&S.mbar_w);
  if (threadIdx.x == 0) {
    tc::mbar_init(mbar_w, 1);
    tc::bulk_load(tc::smem_u32(S.w), img, kImgForward, mbar_w);
  }
  if (t == 0) {
    tc::mbar_init(mbar, 1);
    S.abort[g] = 0;
  }
  if (warp == 0) tc::tmem_alloc(&S.tmem, 64 * kGroups);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  // Warp w reads TMEM lanes 32 (w % 4) .. +31; group g owns columns 64 g .. +63.
  const uint32_t tmem = S.tmem + 64u * g, lane_addr = tmem + (((warp & 3u) * 32u) << 16);
  const uint32_t n = rows(n_max, n_dev, 0);
  uint8_t *A = S.a[g];
  const uint32_t a_addr = tc::smem_u32(A), w_addr = tc::smem_u32(S.w);
  uint32_t phase = 0;
  const uint32_t stride = gridDim.x * kGroups;
  // The gather of the next tile's rows runs one tile ahead -- its queue load
  // from the start of this tile's MMA chain, its hit and ray loads from the second
  // layer, its triangle's normal and material (ShadeView::tri_nm) during the softmax --
  // so that a row's inputs are in registers when its tile starts (spheres still
  // read the scene through make_surface).  Two CTAs per SM: 128 registers.
  PathGather cur{}, nxt{};
  const uint32_t row0 = (blockIdx.x * kGroups + g) * 128u + t;
  gather_slot(pr, row0, n, cur);
  gather_hit(pr, cur);
  gather_na(pr, cur);
  bool ok = true;
  for (uint32_t tile = blockIdx.x * kGroups + g; tile * 128u < n; tile += stride) {
    const uint32_t row = tile * 128u + t;
    float4 r0, r1, r2;
    path_row(pr, cur, r0, r1, r2);
    gather_slot(pr, (tile + stride) * 128u + t, n, nxt);
    write_features(A, t, r0, r1, r2, p);
    if (row == row0 && t == 0 && !tc::mbar_wait(mbar_w, 0, kWaitTries)) {
      S.abort[g] = 1;
      atomicExch(err, CKR_ERR_ITERATION_LIMIT);
    }
    for (int l = 0; l < 4 && ok; ++l) {
      sync_for_mma(g);
      if (S.abort[g]) {
        ok = false;  // the weights never arrived
        break;
      }
      if (t == 0 && !(p.stall_tries && l == 0)) {
        tc::fence_after_sync();
        if (l == 0) issue(tmem, a_addr, w_addr + kImgW1, kIn, 0);
        else issue(tmem, a_addr, w_addr + kImgW2 + 10240u * (l - 1), kHidK, 0);
        tc::mma_commit(mbar);
      }
      ok = wait_mma(g, mbar, phase, &S.abort[g], err, p.stall_tries ? p.stall_tries : kWaitTries);
      if (ok && l < 3) epilogue_relu(lane_addr, A, t);
      if (l == 1) gather_hit(pr, nxt);
    }
    if (!ok) break;
    gather_na(pr, nxt);
    float e[64];
    const bool full = p.nclusters == 64;
    const float sum = full ? softmax_exp64(lane_addr, e) : softmax_exp(lane_addr, p.nclusters, e);
    const bool far = full && clamped(sum);
    if (__any_sync(0xffffffffu, far)) {
      far_cdf(lane_addr, far, delta, row < n ? reinterpret_cast<uint32_t *>(cdf16 + 64 * (size_t)row) : nullptr);
    } else if (row < n && full) {
      const float unif = delta / 64.0f, keep = (1.0f - delta) / sum;
      float run = 0.f;
      uint32_t w[32];
#pragma unroll
      for (int j = 0; j < 64; j += 2) w[j / 2] = cdf_pair(e, j, keep, unif, run);
      uint4 *dst = reinterpret_cast<uint4 *>(cdf16 + 64 * (size_t)row);
#pragma unroll
      for (int q = 0; q < 8; ++q) dst[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
    } else if (row < n) {
      // Selection mixture (1 - delta) softmax + delta / C as a 16-bit cumulative
      // table: entry j = round(65535 * sum_{i <= j} q_i), the last cluster's 65535.
      const float unif = delta / (float)p.nclusters, keep = (1.0f - delta) / sum;
      float run = 0.f;
      uint32_t w[32];
#pragma unroll
      for (int j = 0; j < 64; j += 2) {
        run += (uint32_t)j < p.nclusters ? keep * e[j] + unif : 0.f;
        uint32_t c0 = (uint32_t)j + 1 >= p.nclusters ? 65535u : min(65535u, __float2uint_rn(65535.0f * run));
        run += (uint32_t)j + 1 < p.nclusters ? keep * e[j + 1] + unif : 0.f;
        uint32_t c1 = (uint32_t)j + 2 >= p.nclusters ? 65535u : min(65535u, __float2uint_rn(65535.0f * run));
        w[j / 2] = c0 | (c1 << 16);
      }
      uint4 *dst = reinterpret_cast<uint4 *>(cdf16 + 64 * (size_t)row);
#pragma unroll
      for (int q = 0; q < 8; ++q) dst[q] = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
    }
    cur = nxt;
    tc::fence_before_sync();
    group_sync(g);
  }
  tc::mbar_wait(mbar_w, 0, kWaitTries);  // a group without a tile: the copy has to land before the block ends
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(S.tmem, 64 * kGroups);
}

// ---- inference on records ----------------------------------------------------------
// Latency bound: what a tile takes is a chain of features, four MMA groups and their
// epilogues, so as many tiles as fit run side by side: seven groups of 128 threads in one
// block per SM (shared memory: the weights and 24 KB a group; 72 registers, which the softmax
// meets by reading its logits from tensor memory once for the sum and again for the
// probabilities).  The next tile's records load during this one, the weights come by one bulk
// copy.  262,144 records: 39.0 us at two blocks of two groups and 128 registers, 36.6 with
// the copy and the early loads (two threads a row at 64 registers: 36.5), 33.1 so.
constexpr uint32_t kRecGroups = 7, kRecTPB = 128 * kRecGroups;

struct SmemInferRec {
  uint8_t w[kImgForward];
  uint8_t a[kRecGroups][128 * kIn * 2];
  uint64_t mbar[kRecGroups], mbar_w;
  uint32_t tmem;
  int abort[kRecGroups];
};

__device__ __forceinline__ void rec_group_sync(uint32_t g) {
  asm volatile("bar.sync %0, 128;" ::"r"(g + 1u) : "memory");
}

__global__ void __launch_bounds__(kRecTPB, 1) k_mlp_infer_rec(const float4 *__restrict__ rec, uint32_t n,
                                                             const uint8_t *__restrict__ img, Params p,
                                                             __half *__restrict__ probs, int *err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  SmemInferRec &S = *reinterpret_cast<SmemInferRec *>(smem_raw);
  const uint32_t g = threadIdx.x >> 7, t = threadIdx.x & 127u, warp = threadIdx.x >> 5;
  const uint32_t mbar = tc::smem_u32(&S.mbar[g]), mbar_w = tc::smem_u32(&S.mbar_w);
  if (threadIdx.x == 0) {
    tc::mbar_init(mbar_w, 1);
    tc::bulk_load(tc::smem_u32(S.w), img, kImgForward, mbar_w);
  }
  if (t == 0) {
    tc::mbar_init(mbar, 1);
    S.abort[g] = 0;
  }
  if (warp == 0) tc::tmem_alloc(&S.tmem, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = S.tmem + 64u * g, lane_addr = tmem + (((warp & 3u) * 32u) << 16);
  uint8_t *A = S.a[g];
  const uint32_t a_addr = tc::smem_u32(A), w_addr = tc::smem_u32(S.w);
  const uint32_t tries = p.stall_tries ? p.stall_tries : kWaitTries;
  uint32_t phase = 0;
  // Few tiles go to different SMs.
  const uint32_t tile0 = g * gridDim.x + blockIdx.x, stride = gridDim.x * kRecGroups;
  float4 r0, r1, r2;
  auto load = [&](uint32_t row) {
    r0 = r1 = r2 = make_float4(0, 0, 0, 0);
    if (row >= n) return;
    r0 = __ldg(rec + 3 * (size_t)row);
    r1 = __ldg(rec + 3 * (size_t)row + 1);
    r2 = __ldg(rec + 3 * (size_t)row + 2);
  };
  load(tile0 * 128u + t);
  bool ok = true;
  for (uint32_t tile = tile0; tile * 128u < n; tile += stride) {
    const uint32_t row = tile * 128u + t;
    write_features(A, t, r0, r1, r2, p);
    load((tile + stride) * 128u + t);
    if (tile == tile0 && t == 0 && !tc::mbar_wait(mbar_w, 0, kWaitTries)) {
      S.abort[g] = 1;
      atomicExch(err, CKR_ERR_ITERATION_LIMIT);
    }
    for (int l = 0; l < 4 && ok; ++l) {
      tc::fence_proxy_async();
      tc::fence_before_sync();
      rec_group_sync(g);
      if (S.abort[g]) {
        ok = false;  // the weights never arrived
        break;
      }
      if (t == 0 && !(p.stall_tries && l == 0)) {
        tc::fence_after_sync();
        if (l == 0) issue(tmem, a_addr, w_addr + kImgW1, kIn, 0);
        else issue(tmem, a_addr, w_addr + kImgW2 + 10240u * (l - 1), kHidK, 0);
        tc::mma_commit(mbar);
      }
      if (!tc::mbar_wait(mbar, phase, tries)) {
        S.abort[g] = 1;
        atomicExch(err, CKR_ERR_ITERATION_LIMIT);
      }
      rec_group_sync(g);
      if (S.abort[g]) {
        tc::mbar_wait(mbar, phase, tries);  // let the MMAs in flight land before TMEM is freed
        ok = false;
        break;
      }
      phase ^= 1u;
      tc::fence_after_sync();
      if (l < 3) epilogue_relu(lane_addr, A, t);
    }
    if (!ok) break;
    // Softmax over the first C logits, 32 columns at a time: with all 64, exp of the clamped
    // logit (as softmax_exp64), else of its distance from the largest (softmax_exp).  Columns that are
    // no cluster's are not read: 262,144 records with 8 clusters 39.7 -> 32.3 us, with 33
    // 39.6 -> 34.2 (the exp without denormal results).
    const uint32_t C = p.nclusters;
    const int halves = C > 32 ? 2 : 1;
    float mx = -3.0e38f, sum = 0.f, e[32];
    if (C != 64)
      for (int h = 0; h < halves; ++h) {
        tc::tmem_ld32(lane_addr + 32u * h, e);
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (32u * h + j < C) mx = fmaxf(mx, e[j]);
      }
    auto exps = [&](int h) {
      tc::tmem_ld32(lane_addr + 32u * h, e);
#pragma unroll
      for (int j = 0; j < 32; ++j)
        e[j] = C == 64           ? exp_80(e[j])
               : 32u * h + j < C ? exp_ftz(e[j] - mx)
                                 : 0.f;
    };
    for (int h = 0; h < halves; ++h) {
      exps(h);
#pragma unroll
      for (int j = 0; j < 32; ++j) sum += e[j];
    }
    const bool far = C == 64 && clamped(sum);
    auto store = [&](int h, float inv) {
      uint4 *dst = reinterpret_cast<uint4 *>(probs + 64 * (size_t)row + 32 * h);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint4 v = half8(e + 8 * q, inv);
        if (row < n) dst[q] = v;
      }
    };
    if (__any_sync(0xffffffffu, far)) {
      // As far_cdf, 32 columns at a time in the registers of the usual path (262,144 records 32.8 us
      // with and without it; out of line, its caller's registers saved, 35.2).
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        tc::tmem_ld32(lane_addr + 32u * h, e);
#pragma unroll
        for (int j = 0; j < 32; ++j) mx = fmaxf(mx, finite_logit(e[j]));
      }
      sum = 0.f;
#pragma unroll 1
      for (int h = 0; h < 4; ++h) {
        tc::tmem_ld32(lane_addr + 32u * (h & 1), e);
#pragma unroll
        for (int j = 0; j < 32; ++j) e[j] = far ? exp_ftz(finite_logit(e[j]) - mx) : exp_80(e[j]);
        if (h < 2) {
#pragma unroll
          for (int j = 0; j < 32; ++j) sum += e[j];
        } else {
          store(h - 2, 1.0f / sum);
        }
      }
    } else {
      const float inv = 1.0f / sum;
      for (int h = 0; h < 2; ++h) {
        if (h < halves) exps(h);
        else
#pragma unroll
          for (int j = 0; j < 32; ++j) e[j] = 0.f;
        store(h, inv);
      }
    }
    tc::fence_before_sync();
    rec_group_sync(g);
  }
  tc::mbar_wait(mbar_w, 0, kWaitTries);  // a group without a tile: the copy has to land before the block ends
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(S.tmem, 512);
}

// ---- training -------------------------------------------------------------------
// Two threads per row: thread (t, hf) of a tile computes half hf of row t's features,
// epilogues and transposes (columns 32 hf .. +31), the halves in warps w and w + 4, which
// read the same TMEM lanes.  The softmax's sum runs over all 64 columns in both, in the
// same order.
constexpr uint32_t kTrainTPB = 256;

struct SmemTrain {
  uint8_t w[kImgBytes];
  uint8_t x0[128 * kIn * 2];
  uint8_t h[3][128 * kHidK * 2];  // H1, H2, H3 with the constant-1 column (K = 80)
  // X^T reads up to 768 bytes past x0 and h (sdesc_t): into what follows here.
  uint8_t g[128 * 64 * 2];        // G [128 rows x K 64]
  float loss[4];
  uint64_t mbar, mbar_w;
  uint32_t tmem;
  int abort;
};

constexpr uint32_t kColD = 0;
// TMEM column of the dW^T accumulator of layer l = 0..3 (dW1..dW4).
__device__ __forceinline__ uint32_t col_w(int l) { return 256u - 64u * (uint32_t)l; }

// As sync_for_mma and wait_mma, for the whole block.
__device__ __forceinline__ void block_sync_for_mma() {
  tc::fence_proxy_async();
  tc::fence_before_sync();
  __syncthreads();
}
__device__ __forceinline__ bool block_wait_mma(uint32_t mbar, uint32_t &phase, int *abort, int *err) {
  if (!tc::mbar_wait(mbar, phase, kWaitTries)) {
    *abort = 1;
    atomicExch(err, CKR_ERR_ITERATION_LIMIT);
  }
  __syncthreads();
  if (*abort) {
    tc::mbar_wait(mbar, phase, kWaitTries);  // let the MMAs in flight land before TMEM is freed
    return false;
  }
  phase ^= 1u;
  tc::fence_after_sync();
  return true;
}

// Latency bound: a CTA's tile is a chain of eight MMA groups with an epilogue between each
// two.  So: two threads a row; the weight images by one bulk copy beside the features; X^T
// and G^T read in place as MN-major operands (copied by the threads, 2 bytes a store and
// four-way bank conflicts, they were 5 of the kernel's 20 us); and the batch's weight sum
// (k_mlp_wsum, the launch before), which only the loss needs, overlapping the forward pass
// (programmatic dependent launch).  A step of 4,096 records: 39.4 -> 21.8 us, this kernel
// 24.0 -> 14.6 us.
__global__ void __launch_bounds__(kTrainTPB) k_mlp_train(const float4 *__restrict__ rec, uint32_t n_max,
                                                         const uint32_t *n_dev, uint32_t n_off,
                                                         const uint8_t *__restrict__ img, const float *scalars,
                                                         Params p, float *__restrict__ part, float *loss_part,
                                                         int *err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  SmemTrain &S = *reinterpret_cast<SmemTrain *>(smem_raw);
  const uint32_t t = threadIdx.x & 127u, hf = threadIdx.x >> 7, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  tc::launch_dependents();
  const uint32_t mbar = tc::smem_u32(&S.mbar), mbar_w = tc::smem_u32(&S.mbar_w);
  if (threadIdx.x == 0) {
    tc::mbar_init(mbar, 1);
    tc::mbar_init(mbar_w, 1);
    S.abort = 0;
    tc::bulk_load(tc::smem_u32(S.w), img, kImgBytes, mbar_w);
  }
  if (warp == 0) tc::tmem_alloc(&S.tmem, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = S.tmem, lane_addr = tmem + (((warp & 3u) * 32u) << 16);
  const uint32_t n = rows(n_max, n_dev, n_off);
  const uint32_t w_addr = tc::smem_u32(S.w), x0_addr = tc::smem_u32(S.x0), g_addr = tc::smem_u32(S.g);
  const uint32_t h0_addr = tc::smem_u32(S.h[0]);  // H1, H2, H3 are 20 KB apart
  uint32_t phase = 0, tiles = 0;
  float loss = 0.f, wsum = 0.f;
  bool ok = true;
  for (uint32_t tile = blockIdx.x; ok && tile * 128u < n; tile += gridDim.x, ++tiles) {
    const uint32_t row = tile * 128u + t;
    float4 r0 = make_float4(0, 0, 0, 0), r1 = r0, r2 = r0;
    if (row < n) {
      r0 = rec[3 * (size_t)row];
      r1 = rec[3 * (size_t)row + 1];
      r2 = rec[3 * (size_t)row + 2];
    }
    const uint32_t k = min(__float_as_uint(r2.w), 63u);
    const uint32_t acc = tiles ? 1u : 0u;
    // ---- forward ----
    if (hf == 0) write_features<0>(S.x0, t, r0, r1, r2, p);
    else write_features<1>(S.x0, t, r0, r1, r2, p);
    if (tiles == 0 && threadIdx.x == 0 && !tc::mbar_wait(mbar_w, 0, kWaitTries)) {
      S.abort = 1;
      atomicExch(err, CKR_ERR_ITERATION_LIMIT);
    }
    for (int l = 0; l < 4 && ok; ++l) {
      block_sync_for_mma();
      if (S.abort) {
        ok = false;  // the weights never arrived
        break;
      }
      if (threadIdx.x == 0) {
        tc::fence_after_sync();
        if (l == 0) issue(tmem + kColD, x0_addr, w_addr + kImgW1, kIn, 0);
        else issue(tmem + kColD, h0_addr + 20480u * (l - 1), w_addr + kImgW2 + 10240u * (l - 1), kHidK, 0);
        tc::mma_commit(mbar);
      }
      ok = block_wait_mma(mbar, phase, &S.abort, err);
      if (ok && l < 3) epilogue_relu(lane_addr + kColD, S.h[l], t, hf, hf + 1);
    }
    if (!ok) break;
    // ---- loss gradient at the logits: a (softmax - onehot(k)) ----
    if (tiles == 0) {
      tc::wait_dependencies();
      wsum = __ldcg(scalars);
      if (!(wsum > 0.f)) break;  // nothing to learn: no partial sums
    }
    const float a = (row < n && r1.w > 0.f) ? r1.w / wsum : 0.f;
    {
      float pr[64];
      const float inv = 1.0f / softmax_exp(lane_addr + kColD, p.nclusters, pr);
      float pk = 0.f;
#pragma unroll
      for (int j = 0; j < 64; ++j) {
        pr[j] *= inv;
        pk = (uint32_t)j == k ? pr[j] : pk;
      }
      if (a > 0.f && hf == 0) loss -= a * __logf(fmaxf(pk, 1e-30f));
#pragma unroll
      for (int j = 0; j < 64; ++j) pr[j] = (uint32_t)j < p.nclusters ? a * (pr[j] - ((uint32_t)j == k ? 1.f : 0.f)) : 0.f;
      if (hf == 0) {
#pragma unroll
        for (int q = 0; q < 4; ++q) st8(S.g, t, 8 * q, 64, pr + 8 * q);
      } else {
#pragma unroll
        for (int q = 4; q < 8; ++q) st8(S.g, t, 8 * q, 64, pr + 8 * q);
      }
    }
    const uint32_t j0 = 32u * hf;
    // ---- backward, layers 4, 3, 2 (input H3, H2, H1) ----
    for (int l = 2; l >= 0 && ok; --l) {
      block_sync_for_mma();
      if (threadIdx.x == 0) {
        tc::fence_after_sync();
        issue_t(tmem + col_w(l + 1), h0_addr + 20480u * l, kHidK, g_addr, acc);  // dW^T += X^T G
        issue(tmem + kColD, g_addr, w_addr + kImgW2t + 8192u * l, 64, 0);        // dX = G W
        tc::mma_commit(mbar);
      }
      // The layer's ReLU mask, while the MMAs run.
      float hv[32], d[32];
#pragma unroll
      for (int q = 0; q < 4; ++q) ld8(S.h[l], t, j0 + 8 * q, kHidK, hv + 8 * q);
      if (!(ok = block_wait_mma(mbar, phase, &S.abort, err))) break;
      // G of the layer below: dX masked by its ReLU.
      tc::tmem_ld32(lane_addr + kColD + j0, d);
#pragma unroll
      for (int j = 0; j < 32; ++j) d[j] = hv[j] > 0.f ? d[j] : 0.f;
#pragma unroll
      for (int q = 0; q < 4; ++q) st8(S.g, t, j0 + 8 * q, 64, d + 8 * q);
    }
    if (!ok) break;
    // ---- layer 1: dW1^T += X0^T G1 ----
    block_sync_for_mma();
    if (threadIdx.x == 0) {
      tc::fence_after_sync();
      issue_t(tmem + col_w(0), x0_addr, kIn, g_addr, acc);
      tc::mma_commit(mbar);
    }
    if (!(ok = block_wait_mma(mbar, phase, &S.abort, err))) break;
    tc::fence_before_sync();
    __syncthreads();
  }
  // A block without a tile has not waited for its weights, nor for the launch before.
  if (tiles == 0) {
    tc::mbar_wait(mbar_w, 0, kWaitTries);
    tc::wait_dependencies();
  }
  // ---- per-CTA partial sums ----
  for (int o = 16; o; o >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, o);
  if (lane == 0 && hf == 0) S.loss[warp] = loss;
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  float *my = part + (size_t)blockIdx.x * kNParams;
  const bool have = ok && tiles > 0;
  if (threadIdx.x == 0) loss_part[blockIdx.x] = have ? S.loss[0] + S.loss[1] + S.loss[2] + S.loss[3] : 0.f;
  // Row t (a TMEM lane) of each dW^T accumulator: weights of input t, or (row 64 of
  // layers 2-4) the bias.
  for (int l = 0; l < 4; ++l) {
    const uint32_t fan = l == 0 ? kIn : 64;
    float v[32];
    if (have) {
      tc::tmem_ld32(lane_addr + col_w(l) + 32u * hf, v);
    } else {
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = 0.f;
    }
    const uint32_t offW = l == 0 ? kOffW1 : l == 1 ? kOffW2 : l == 2 ? kOffW3 : kOffW4;
    const uint32_t offB = l == 1 ? kOffB2 : l == 2 ? kOffB3 : kOffB4;
    if (t < fan) {
#pragma unroll
      for (int o = 0; o < 32; ++o) my[offW + (32u * hf + o) * fan + t] = v[o];
    } else if (l > 0 && t == 64) {
#pragma unroll
      for (int o = 0; o < 32; ++o) my[offB + 32u * hf + o] = v[o];
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
}

// Weight sum of the batch (one CTA; deterministic order).
__global__ void k_mlp_wsum(const float4 *__restrict__ rec, uint32_t n_max, const uint32_t *n_dev, uint32_t n_off,
                           float *scalars) {
  __shared__ float red[32];
  tc::launch_dependents();  // the training kernel's forward pass does not need the sum
  const uint32_t n = rows(n_max, n_dev, n_off);
  float s = 0.f;
  for (uint32_t r = threadIdx.x; r < n; r += blockDim.x) {
    float w = rec[3 * (size_t)r + 1].w;
    s += w > 0.f ? w : 0.f;
  }
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    float tot = 0.f;
    for (uint32_t w = 0; w < blockDim.x / 32; ++w) tot += red[w];
    scalars[0] = tot;
  }
}

// Image slots of parameter j (kmaj offsets in bytes; -1: none).
__device__ __forceinline__ void image_slots(uint32_t j, int &a, int &b) {
  a = b = -1;
  if (j < kOffW2) {
    uint32_t o = j / kIn, i = j % kIn;
    a = kImgW1 + tc::kmaj(o, i, kIn);
  } else {
    const uint32_t offs[3] = {kOffW2, kOffW3, kOffW4}, img[3] = {kImgW2, kImgW3, kImgW4},
                   imgt[3] = {kImgW2t, kImgW3t, kImgW4t};
    for (int l = 0; l < 3; ++l) {
      if (j >= offs[l] && j < offs[l] + 4096) {
        uint32_t o = (j - offs[l]) / 64, i = (j - offs[l]) % 64;
        a = img[l] + tc::kmaj(o, i, kHidK);
        b = imgt[l] + tc::kmaj(i, o, 64);
      } else if (j >= offs[l] + 4096 && j < offs[l] + 4096 + 64) {  // bias of output o at K = 64
        a = img[l] + tc::kmaj(j - offs[l] - 4096, 64, kHidK);
      }
    }
  }
}

// Sums the per-CTA gradients, applies Adam (when the batch had weight) and
// rewrites the BF16 images.  update = 0: images only.
__global__ void k_mlp_adam(float *params, float *m, float *v, const float *part, uint32_t grid,
                           const float *loss_part, float *scalars, uint8_t *img, int update, float lr, float b1,
                           float b2, float eps, float c1, float c2) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (update) tc::wait_dependencies();
  if (update && blockIdx.x == 0 && threadIdx.x == 0 && scalars[0] > 0.f) {
    float l = 0.f;
#pragma unroll 16
    for (uint32_t c = 0; c < grid; ++c) l += loss_part[c];
    scalars[1] = l;
  }
  if (j >= kNParams) return;
  float w = params[j];
  if (update && scalars[0] > 0.f) {
    float g = 0.f;
#pragma unroll 16
    for (uint32_t c = 0; c < grid; ++c) g += part[(size_t)c * kNParams + j];
    float mj = b1 * m[j] + (1.f - b1) * g, vj = b2 * v[j] + (1.f - b2) * g * g;
    m[j] = mj;
    v[j] = vj;
    w -= lr * (mj / c1) / (sqrtf(vj / c2) + eps);
    params[j] = w;
  }
  int a, b;
  image_slots(j, a, b);
  __nv_bfloat16 h = __float2bfloat16_rn(w);
  if (a >= 0) *reinterpret_cast<__nv_bfloat16 *>(img + a) = h;
  if (b >= 0) *reinterpret_cast<__nv_bfloat16 *>(img + b) = h;
}

Params params_of(const Net &net) {
  Params p;
  p.cx = net.centre[0];
  p.cy = net.centre[1];
  p.cz = net.centre[2];
  p.scale = net.scale;
  p.nclusters = net.nclusters;
  p.stall_tries = net.stall_tries;
  return p;
}

int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return std::max(1, sms);
}

}  // namespace

int create(Net &net, uint64_t seed) {
  std::vector<float> w(kNParams, 0.f);
  // He-uniform initialisation from the counter stream (seed, layer); the output
  // layer is scaled by 0.1 so that the first proposals are close to uniform.
  auto init = [&](uint32_t off, uint32_t nout, uint32_t nin, uint32_t fan, uint32_t layer, double gain) {
    uint64_t key = ckr_key(seed, layer);
    double lim = gain * std::sqrt(6.0 / fan);
    for (uint32_t o = 0; o < nout; ++o)
      for (uint32_t i = 0; i < nin; ++i)
        w[off + o * (nin == 79 ? kIn : nin) + i] =
            (float)((2.0 * ckr_draw_f(key, o * 128 + i) - 1.0) * lim);
  };
  init(kOffW1, kHid, 79, 79, 1, 1.0);  // features 0..78; the bias column 79 and padding stay 0
  init(kOffW2, kHid, kHid, kHid, 2, 1.0);
  init(kOffW3, kHid, kHid, kHid, 3, 1.0);
  init(kOffW4, kOut, kHid, kHid, 4, 0.1);
  net.grid = (uint32_t)sm_count();
  if (cudaMalloc((void **)&net.params, kNParams * 4) != cudaSuccess ||
      cudaMalloc((void **)&net.m, kNParams * 4) != cudaSuccess ||
      cudaMalloc((void **)&net.v, kNParams * 4) != cudaSuccess ||
      cudaMalloc((void **)&net.part, (size_t)net.grid * kNParams * 4) != cudaSuccess ||
      cudaMalloc((void **)&net.loss_part, net.grid * 4) != cudaSuccess ||
      cudaMalloc((void **)&net.scalars, 16) != cudaSuccess || cudaMalloc((void **)&net.img, kImgBytes) != cudaSuccess ||
      cudaMalloc((void **)&net.err, 4) != cudaSuccess) {
    destroy(net);
    return CKR_ERR_OUT_OF_MEMORY;
  }
  CKR_CUDA_TRY(cudaMemcpy(net.params, w.data(), kNParams * 4, cudaMemcpyHostToDevice));
  CKR_CUDA_TRY(cudaMemset(net.m, 0, kNParams * 4));
  CKR_CUDA_TRY(cudaMemset(net.v, 0, kNParams * 4));
  CKR_CUDA_TRY(cudaMemset(net.img, 0, kImgBytes));
  CKR_CUDA_TRY(cudaMemset(net.scalars, 0, 16));
  CKR_CUDA_TRY(cudaMemset(net.err, 0, 4));
  int dev = 0;
  CKR_CUDA_TRY(cudaGetDevice(&dev));
  for (auto [fn, smem] : {std::pair{(const void *)k_mlp_infer, sizeof(SmemInfer)},
                          std::pair{(const void *)k_mlp_infer_rec, sizeof(SmemInferRec)}}) {
    CKR_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    CKR_CUDA_TRY(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  }
  CKR_CUDA_TRY(cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemTrain)));
  int st = pack(net, nullptr);
  if (st != CKR_OK) return st;
  CKR_CUDA_TRY(cudaDeviceSynchronize());
  return CKR_OK;
}

void destroy(Net &net) {
  cudaFree(net.params);
  cudaFree(net.m);
  cudaFree(net.v);
  cudaFree(net.part);
  cudaFree(net.loss_part);
  cudaFree(net.scalars);
  cudaFree(net.img);
  cudaFree(net.err);
  net = Net();
}

int pack(Net &net, cudaStream_t stream) {
  k_mlp_adam<<<ceil_div(kNParams, 256), 256, 0, stream>>>(net.params, net.m, net.v, net.part, net.grid,
                                                           net.loss_part, net.scalars, net.img, 0, 0.f, 0.f, 0.f,
                                                           0.f, 1.f, 1.f);
  CKR_CUDA_TRY(cudaGetLastError());
  return CKR_OK;
}

int infer(const Net &net, const float4 *rec, uint32_t n, __half *probs, cudaStream_t stream) {
  if (n == 0) return CKR_OK;
  const uint32_t grid = std::min<uint32_t>(ceil_div(n, 128), (uint32_t)sm_count());
  k_mlp_infer_rec<<<grid, kRecTPB, sizeof(SmemInferRec), stream>>>(rec, n, net.img, params_of(net), probs, net.err);
  CKR_CUDA_TRY(cudaGetLastError());
  return CKR_OK;
}

int infer_paths(const Net &net, const PathRows &rows, uint32_t n_max, const uint32_t *n_dev, uint16_t *cdf16,
                float delta, cudaStream_t stream, const uint8_t *img) {
  if (n_max == 0) return CKR_OK;
  // CTAs resident per SM: shared memory (the opt-in maximum over the CTA's
  // footprint plus the 1 KB the driver reserves per CTA) or 4.
  static int per_sm = 0;
  if (!per_sm) {
    int dev = 0, smem = 0;
    CKR_CUDA_TRY(cudaGetDevice(&dev));
    CKR_CUDA_TRY(cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    per_sm = std::max(1, std::min(4, smem / (int)(sizeof(SmemInfer) + 1024)));
  }
  const uint32_t grid = std::min<uint32_t>(ceil_div(n_max, 128 * kGroups), (uint32_t)sm_count() * per_sm);
  k_mlp_infer<<<grid, kInferTPB, sizeof(SmemInfer), stream>>>(rows, n_max, n_dev, img ? img : net.img, params_of(net),
                                                              delta, cdf16, net.err);
  CKR_CUDA_TRY(cudaGetLastError());
  return CKR_OK;
}

namespace {
template <class T>
struct Same {
  using type = T;
};
// A launch that may start before the stream's previous kernel has ended; the kernel waits
// for it where it needs it (tc::wait_dependencies).
template <class... A>
cudaError_t launch_early(void (*fn)(A...), uint32_t grid, uint32_t tpb, size_t smem, cudaStream_t stream,
                         typename Same<A>::type... a) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(tpb);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fn, a...);
}
}  // namespace

int gradients(Net &net, const float4 *rec, uint32_t n_max, const uint32_t *n_dev, uint32_t n_off,
              cudaStream_t stream) {
  // One block per 128-record tile: with the grid fixed at one block per SM, the blocks
  // without a tile wrote zero partial sums (74 KB each) for k_mlp_adam to add.
  net.used = std::max<uint32_t>(1, std::min(net.grid, (uint32_t)ceil_div(n_max, 128)));
  k_mlp_wsum<<<1, 1024, 0, stream>>>(rec, n_max, n_dev, n_off, net.scalars);
  CKR_CUDA_TRY(cudaGetLastError());
  CKR_CUDA_TRY(launch_early(k_mlp_train, net.used, kTrainTPB, sizeof(SmemTrain), stream, rec, n_max, n_dev, n_off,
                            net.img, net.scalars, params_of(net), net.part, net.loss_part, net.err));
  return CKR_OK;
}

int train_step(Net &net, const float4 *rec, uint32_t n_max, const uint32_t *n_dev, uint32_t n_off,
               cudaStream_t stream) {
  if (n_max == 0) return CKR_OK;
  int st = gradients(net, rec, n_max, n_dev, n_off, stream);
  if (st != CKR_OK) return st;
  net.step += 1;
  const float c1 = 1.0f - std::pow(net.beta1, (float)net.step), c2 = 1.0f - std::pow(net.beta2, (float)net.step);
  CKR_CUDA_TRY(launch_early(k_mlp_adam, ceil_div(kNParams, 256), 256, 0, stream, net.params, net.m, net.v, net.part,
                            net.used, net.loss_part, net.scalars, net.img, 1, net.lr, net.beta1, net.beta2, net.eps, c1,
                            c2));
  return CKR_OK;
}

}  // namespace mlp
}  // namespace ckr
