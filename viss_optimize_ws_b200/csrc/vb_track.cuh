// Device pieces shared by the factored sums (vb_track.cu: stage 1,
// vb_track2.cu: stage 2).
#pragma once
#include <cuda_runtime.h>

#include "vb_common.cuh"
#include "vb_internal.h"
#include "vb_stage1.cuh"

namespace vb {

constexpr int TK_LEVELS = 3;             // pixel blocks of 64, 256, 1024
__host__ __device__ constexpr int tk_block(int level) { return 64 << (2 * level); }

// Two floats in one register pair: the packed FP32 instructions do a complex
// number's two parts in one issue slot.
using f2 = unsigned long long;
__device__ __forceinline__ f2 f2_make(float x, float y) {
  f2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 f2_split(f2 a) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
  return r;
}
__device__ __forceinline__ f2 f2_fma(f2 a, f2 b, f2 c) {
  f2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ f2 f2_add(f2 a, f2 b) {
  f2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f2 f2_mul(f2 a, f2 b) {
  f2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// One step of the transposed reduction: lanes whose bit M is clear keep the
// first half of the list, the others the second half (an odd list is padded
// with a zero).
template <int N, int M>
__device__ __forceinline__ void fold_half(float* v, bool up) {
  constexpr int H = (N + 1) / 2;
#pragma unroll
  for (int i = 0; i < H; ++i) {
    const float other = i + H < N ? v[i + H] : 0.f;
    const float keep = up ? other : v[i], send = up ? v[i] : other;
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, M);
  }
}

// cos and sin of t turns in FP64 to about 2e-9 (Taylor series on an eighth of a
// turn): the factor of a whole block's sum, so it must not carry the SFU's noise.
__device__ __forceinline__ void turn_cs(double t, double& s, double& c) {
  const double k = fma(t, 4.0, 6755399441055744.0);   // 1.5 * 2^52: rounds to an integer
  const int q = __double2loint(k);
  const double g = fma(k - 6755399441055744.0, -0.25, t);
  const double x = g * 6.283185307179586476925, x2 = x * x;
  double sp = fma(x2, 1.0 / 362880.0, -1.0 / 5040.0);
  sp = fma(sp, x2, 1.0 / 120.0);
  sp = fma(sp, x2, -1.0 / 6.0);
  sp = fma(sp * x2, x, x);
  double cp = fma(x2, -1.0 / 3628800.0, 1.0 / 40320.0);
  cp = fma(cp, x2, -1.0 / 720.0);
  cp = fma(cp, x2, 1.0 / 24.0);
  cp = fma(cp, x2, -0.5);
  cp = fma(cp, x2, 1.0);
  const double ss = (q & 1) ? cp : sp, cc = (q & 1) ? sp : cp;
  s = (q & 2) ? -ss : ss;
  c = ((q + 1) & 2) ? -cc : cc;
}

// Class of one unit endpoint (d.w = cos phi, s = sin phi of its horizon) against
// a node's cone of half-angle alpha, as exact_class in float32: every pixel
// passes when cos(axis, endpoint) >= cos(phi - alpha), every pixel fails when it
// is <= cos(phi + alpha).  The margin covers the per-pixel test's evaluation
// error (2e-6) and this test's own (below 1e-6).
__device__ __forceinline__ int endpoint_class(const TrackNode& n, const float4 d, float s) {
  constexpr float kMargin = 1.2e-5f;
  const float cd = fmaf(n.axis.x, d.x, fmaf(n.axis.y, d.y, n.axis.z * d.z));
  const float cc = d.w * n.axis.w, ss = s * n.cen.w;
  const bool vis = n.axis.w >= d.w && cd >= cc + ss + kMargin;
  const bool hid = n.axis.w >= -d.w && cd <= cc - ss - kMargin;
  return vis ? kClsVis : (hid ? kClsHid : kClsMix);
}

__device__ __forceinline__ int both_classes(int e1, int e2) {
  return (e1 == kClsHid || e2 == kClsHid) ? kClsHid : ((e1 == kClsVis && e2 == kClsVis) ? kClsVis : kClsMix);
}

// Sine of the horizon angle of a unit endpoint (NaN where the endpoint is off
// the unit sphere: no cone test then decides anything).
__device__ __forceinline__ float horizon_sine(const float4 d) {
  const double rr = (double)d.x * d.x + (double)d.y * d.y + (double)d.z * d.z;
  return fabs(rr - 1.0) <= 2e-6 && fabsf(d.w) <= 1.f ? sqrtf(fmaxf(0.f, 1.f - d.w * d.w)) : NAN;
}

}  // namespace vb
