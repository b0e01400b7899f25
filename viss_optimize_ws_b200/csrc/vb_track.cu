// Stage 1, factored over track groups: the same sum as vb_stage1.cu for the
// baselines of one satellite pair over consecutive time steps, with one sin /
// cos per (group, pixel) instead of one per (baseline, pixel).
//
// The (u, v, w) of a pair move along a smooth track, so within a group
// u_k = u_c + D_k with small D_k, and within a block of neighbouring pixels
// s_p = s_c + d_p with small d_p:
//   sum_p B_p e^{2 pi i u_k.s_p} = e^{2 pi i D_k.s_c} sum_p z_p e^{2 pi i D_k.d_p},
//   z_p = B_p e^{2 pi i u_c.s_p}     (one sin / cos per group and pixel).
// In the group's frame (e1 along the track, e2 towards its sagitta, e3 across)
// D_k is a place a on the curve b = gamma a + kappa a^2 and two small residuals
// (the positions' float rounding, mostly); e^{2 pi i D_k.d_p} is a polynomial
// in a for the curve's factor, times the residuals to first order.  The warp
// forms the polynomial's moments over the pixels once per (group, block), then
// every baseline of the group evaluates it.  A group is taken only where any
// single term is off by at most 6e-7 to 8e-7 (vb_series.h: 1e-7 for the polynomial,
// the rest for the residuals, at a block's edge and a group's end); the phase of z_p is
// rounded once here and three times in the per-term kernel, 3.7e-7 against 1.1e-6,
// so that a term is no further off than there.  Measured on skies of one source,
// largest and rms error of a term: 1.5e-6 and 3.4e-7, per-term kernel 1.5e-6 and
// 4.4e-7.  The other groups (fast tracks on coarse pixels, irregular baselines,
// skies whose pixel blocks are not compact) go to the per-term kernel through a list.
//
// Bound: FP32 issue.  Per group of K baselines and block of P pixels a warp
// executes P/32 x (phase, sin/cos, 2 J multiply-adds) + a transposed
// reduction of 2 J values + K/32 x (2 J multiply-adds and one FP64 rotation),
// where the per-term kernel needs 16 SFU cycles for each 32 terms.
//
// Which terms enter is decided exactly as in the per-term kernel: tile-cone
// classes with the upstream's float test, undecided (baseline, block) pairs by
// the conservative exact cones, and what they leave open by the per-pixel test
// (one baseline at a time, the warp's lanes on its pixels).
#include <algorithm>
#include <cmath>

#include "vb_common.cuh"
#include "vb_geom.cuh"
#include "vb_internal.h"
#include "vb_series.h"
#include "vb_stage1.cuh"
#include "vb_track.cuh"

namespace vb {

constexpr int TK_GROUP = kTrackGroup;    // slots of a group: 4 per lane
constexpr int TK_SLOTS = 4;
constexpr int TK_WARPS = 4;              // warps per CTA (independent of one another)
constexpr int TK_THREADS = 32 * TK_WARPS;
constexpr int TK_QUAD = 4;               // blocks whose moments a warp forms at a time, 8 lanes each
constexpr int TK_CHUNK = TK_QUAD * 1024; // chunks hold whole quads of the largest blocks

// Polynomial shapes: powers of a in the curve's own factor, in the residuals'
// first-order terms, and their sum (coefficients: kSeries).
template <int SET>
struct Shape {
  static constexpr int N = SET == 0 ? 8 : SET == 1 ? 12 : 16;
  static constexpr int NE = N / 2;
  static constexpr int J = N + 2 * NE;
};
constexpr int TK_SETS = 3;
constexpr int TK_JMAX = Shape<TK_SETS - 1>::J;
static_assert(Shape<0>::N == 8 && Shape<1>::N == 12 && Shape<2>::N == 16, "the shapes of kSeries");

struct TrackArgs {
  const float *B, *l, *m, *n;
  int64_t npix;
  int chunk_pix, nchunk;
  int tilecone, cull_tile, mask_visible, blockage, raw;
  const float *tcx, *tcy, *tcz, *tcosA, *tsinA;
  const TrackNode* node[TK_LEVELS];
  const unsigned* rmax;
  const TrackPlan* plan;
  const float4 *q0, *d1, *d2, *p1, *p2;   // per slot: (u, v, w, t1), unit endpoints and horizon cosines, (endpoint, horizon sine)
  const float* t2;
  const int* list;
  const int* count;                        // {groups listed, baselines left to the per-term kernel}
  int* queue;
  double2* partial;
  int n_half, nbl, steps, gpp;
  float scale[kSeriesTables][2 * TK_JMAX];  // coefficient and sign of each reduced moment
  unsigned char dest[TK_SETS][2 * TK_JMAX];
};

// ---------------------------------------------------------------------------
// Pixel blocks: centre (mean of the pixel vectors), cone, and the largest
// centre-pixel distance of the sky per level.  A value that is not finite, a
// pixel vector off the unit sphere or an absurdly large brightness anywhere
// makes the distances infinite, which keeps every group on the per-term kernel.
// Blocks of coincident pixels have no extent: the distances stay at kMinRadius or
// above (what reads them divides by them).  One CTA per 1024 pixels, 4 pixels per
// thread, so that a half-warp holds a 64-pixel block and a pair of warps a
// 256-pixel block.
// Bound: HBM (16 bytes read per pixel).
constexpr float kMinRadius = 1e-6f;   // well under the extent of any block of distinct pixels

struct BlockArgs {
  const float *B, *l, *m, *n;
  int64_t npix;
  int nsuper;
  TrackNode* node[TK_LEVELS];
  unsigned* rmax;
};

__device__ __forceinline__ double half_warp_sum(double v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__global__ void __launch_bounds__(256) k_track_blocks(const BlockArgs a) {
  __shared__ double s_sum[16][7];        // per half-warp: raw sums, unit sums, count
  __shared__ double s_min[TK_LEVELS][16];
  __shared__ float s_r[TK_LEVELS][16];
  const int hw = threadIdx.x >> 4;
  for (int sb = blockIdx.x; sb < a.nsuper; sb += gridDim.x) {
    const int64_t base = (int64_t)sb * 1024 + threadIdx.x * 4;
    float x[4], y[4], z[4];
    double ux[4], uy[4], uz[4];
    double sum[7] = {0, 0, 0, 0, 0, 0, 0};
    bool bad = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      x[k] = y[k] = z[k] = 0.f;
      ux[k] = uy[k] = uz[k] = 0.0;
      if (base + k < a.npix) {
        x[k] = a.l[base + k]; y[k] = a.m[base + k]; z[k] = a.n[base + k];
        const float b = a.B ? a.B[base + k] : 0.f;
        const double nn = (double)x[k] * x[k] + (double)y[k] * y[k] + (double)z[k] * z[k];
        bad |= !(fabs(nn - 1.0) <= 4e-6 && fabsf(b) < 1e30f);
        const double inv = rsqrt(nn);
        ux[k] = x[k] * inv; uy[k] = y[k] * inv; uz[k] = z[k] * inv;
        sum[0] += x[k]; sum[1] += y[k]; sum[2] += z[k];
        sum[3] += ux[k]; sum[4] += uy[k]; sum[5] += uz[k];
        sum[6] += 1.0;
      }
    }
#pragma unroll
    for (int c = 0; c < 7; ++c) sum[c] = half_warp_sum(sum[c]);
    __syncthreads();
    if ((threadIdx.x & 15) == 0)
      for (int c = 0; c < 7; ++c) s_sum[hw][c] = sum[c];
    __syncthreads();
    double ax[TK_LEVELS][3];
    float cc[TK_LEVELS][3];
#pragma unroll
    for (int lev = 0; lev < TK_LEVELS; ++lev) {
      const int w = 1 << (2 * lev);            // half-warps per block
      const int h0 = hw & ~(w - 1);
      double t[7] = {0, 0, 0, 0, 0, 0, 0};
      for (int h = h0; h < h0 + w; ++h)
        for (int c = 0; c < 7; ++c) t[c] += s_sum[h][c];
      const double cnt = t[6] > 0 ? t[6] : 1.0;
      const double nrm = sqrt(t[3] * t[3] + t[4] * t[4] + t[5] * t[5]);
      for (int c = 0; c < 3; ++c) {
        cc[lev][c] = (float)(t[c] / cnt);
        ax[lev][c] = t[3 + c] / nrm;
      }
      double mind = 1.0;
      float r2 = 0.f;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (base + k >= a.npix) continue;
        const double d = ax[lev][0] * ux[k] + ax[lev][1] * uy[k] + ax[lev][2] * uz[k];
        mind = d < mind ? d : (d >= mind ? mind : -1.0);   // a NaN axis makes the cone the whole sphere
        const float dx = x[k] - cc[lev][0], dy = y[k] - cc[lev][1], dz = z[k] - cc[lev][2];
        r2 = fmaxf(r2, dx * dx + dy * dy + dz * dz);
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) {
        mind = fmin(mind, __shfl_xor_sync(0xffffffffu, mind, o));
        r2 = fmaxf(r2, __shfl_xor_sync(0xffffffffu, r2, o));
      }
      if ((threadIdx.x & 15) == 0) {
        s_min[lev][hw] = mind;
        s_r[lev][hw] = sqrtf(r2) * 1.00001f;
      }
    }
    const bool any_bad = __syncthreads_or(bad ? 1 : 0);
    if ((threadIdx.x & 15) == 0) {
#pragma unroll
      for (int lev = 0; lev < TK_LEVELS; ++lev) {
        const int w = 1 << (2 * lev);
        if (hw & (w - 1)) continue;
        const int64_t blk = (int64_t)sb * (16 / w) + hw / w;
        if (blk * tk_block(lev) >= a.npix) continue;
        double mind = 1.0;
        float r = 0.f;
        for (int h = hw; h < hw + w; ++h) {
          mind = fmin(mind, s_min[lev][h]);
          r = fmaxf(r, s_r[lev][h]);
        }
        // the half-angle rounded outwards
        const double alpha = acos(fmax(-1.0, fmin(1.0, mind))) + 1e-9;
        TrackNode e;
        e.cen = make_float4(cc[lev][0], cc[lev][1], cc[lev][2], (float)sin(alpha));
        e.axis = make_float4((float)ax[lev][0], (float)ax[lev][1], (float)ax[lev][2], (float)cos(alpha));
        a.node[lev][blk] = e;
        atomicMax(&a.rmax[lev], __float_as_uint(any_bad || !(r < 16.f) ? INFINITY : fmaxf(r, kMinRadius)));
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// Plan: the shape of each group (slots per sub-group, pixel block, polynomial),
// or none.  One warp per group; O(n_half).
struct SeriesBox {
  int set;
  float x1, x2, e;
};
struct PlanArgs {
  SeriesBox box[kSeriesTables];
  const float *u, *v, *w, *x1, *y1, *z1, *in1;
  int nbl, steps, gpp, ngroups, max_level, blockage;
  const unsigned* rmax;
  TrackPlan* plan;
};

// Frame, curve and extents (half-range along the track, curve, residuals from
// the curve and across; the first two grow by the tilt that the curve's slope
// gives the axis) of one sub-group (slots [q0, q0 + ks) of the lanes).
__device__ __forceinline__ void sub_frame(const float (&p)[TK_SLOTS][3], int nv, int lane, int q0, int ks, double (&uc)[3],
                                          float (&e)[9], float& gamma, float& kappa, float (&R)[4]) {
  const int n0 = q0 * 32, n1 = min(nv, (q0 + ks) * 32);
  R[0] = R[1] = R[2] = R[3] = 0.f;
  gamma = kappa = 0.f;
  for (int c = 0; c < 9; ++c) e[c] = (c % 4 == 0) ? 1.f : 0.f;
  uc[0] = uc[1] = uc[2] = 0.0;
  if (n1 <= n0) return;
  float first[3] = {0, 0, 0}, last[3] = {0, 0, 0};
  const int ql = (n1 - 1) >> 5, ll = (n1 - 1) & 31;
#pragma unroll
  for (int q = 0; q < TK_SLOTS; ++q)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float f = __shfl_sync(0xffffffffu, p[q][c], 0), g = __shfl_sync(0xffffffffu, p[q][c], ll);
      if (q == q0) first[c] = f;
      if (q == ql) last[c] = g;
    }
  float d[3];
  for (int c = 0; c < 3; ++c) d[c] = (float)((double)last[c] - first[c]);
  float nn = d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
  if (nn > 1e-20f) {
    const float inv = __frsqrt_rn(nn);
    for (int c = 0; c < 3; ++c) e[c] = d[c] * inv;
  }
  // farthest point from the chord
  float best = -1.f, bx = 0.f, by = 0.f, bz = 0.f;
#pragma unroll
  for (int q = 0; q < TK_SLOTS; ++q) {
    if (q < q0 || q >= q0 + ks || q * 32 + lane >= n1) continue;
    const float x = (float)((double)p[q][0] - first[0]), y = (float)((double)p[q][1] - first[1]),
                z = (float)((double)p[q][2] - first[2]);
    const float t = x * e[0] + y * e[1] + z * e[2];
    const float gx = x - t * e[0], gy = y - t * e[1], gz = z - t * e[2];
    const float g2 = gx * gx + gy * gy + gz * gz;
    if (g2 > best) { best = g2; bx = gx; by = gy; bz = gz; }
  }
  const float top = warp_max(best);
  const int src = __ffs(__ballot_sync(0xffffffffu, best == top)) - 1;
  bx = __shfl_sync(0xffffffffu, bx, src & 31);
  by = __shfl_sync(0xffffffffu, by, src & 31);
  bz = __shfl_sync(0xffffffffu, bz, src & 31);
  // e2: orthonormal to e1 (any perpendicular where the points are collinear)
  if (!(top > 1e-12f * nn) || !(top > 1e-24f)) {
    const bool xs = fabsf(e[0]) < 0.6f;
    bx = xs ? 1.f : 0.f; by = xs ? 0.f : 1.f; bz = 0.f;
  }
  float t = bx * e[0] + by * e[1] + bz * e[2];
  bx -= t * e[0]; by -= t * e[1]; bz -= t * e[2];
  float inv = __frsqrt_rn(bx * bx + by * by + bz * bz);
  bx *= inv; by *= inv; bz *= inv;
  t = bx * e[0] + by * e[1] + bz * e[2];
  bx -= t * e[0]; by -= t * e[1]; bz -= t * e[2];
  inv = __frsqrt_rn(bx * bx + by * by + bz * bz);
  e[3] = bx * inv; e[4] = by * inv; e[5] = bz * inv;
  e[6] = e[1] * e[5] - e[2] * e[4];
  e[7] = e[2] * e[3] - e[0] * e[5];
  e[8] = e[0] * e[4] - e[1] * e[3];
  // coordinates in the frame
  float f[TK_SLOTS][3];
  float lo = INFINITY, hi = -INFINITY, lc = INFINITY, hc = -INFINITY;
#pragma unroll
  for (int q = 0; q < TK_SLOTS; ++q) {
    f[q][0] = f[q][1] = f[q][2] = 0.f;
    if (q < q0 || q >= q0 + ks || q * 32 + lane >= n1) continue;
    const float x = (float)((double)p[q][0] - first[0]), y = (float)((double)p[q][1] - first[1]),
                z = (float)((double)p[q][2] - first[2]);
    for (int c = 0; c < 3; ++c) f[q][c] = x * e[3 * c] + y * e[3 * c + 1] + z * e[3 * c + 2];
    lo = fminf(lo, f[q][0]); hi = fmaxf(hi, f[q][0]);
    lc = fminf(lc, f[q][2]); hc = fmaxf(hc, f[q][2]);
  }
  hi = warp_max(hi); lo = -warp_max(-lo);
  hc = warp_max(hc); lc = -warp_max(-lc);
  const float mid = 0.5f * (hi + lo), A = 0.5f * (hi - lo), midc = 0.5f * (hc + lc);
  // least squares b ~ beta + g x + k x^2, x = (a - mid) / A
  const float invA = A > 1e-12f ? 1.f / A : 0.f;
  double S[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int q = 0; q < TK_SLOTS; ++q) {
    if (q < q0 || q >= q0 + ks || q * 32 + lane >= n1) continue;
    const double x = (f[q][0] - mid) * invA, bb = f[q][1], xx = x * x;
    S[0] += 1.0; S[1] += x; S[2] += xx; S[3] += xx * x; S[4] += xx * xx;
    S[5] += bb; S[6] += x * bb; S[7] += xx * bb;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k)
    for (int o = 16; o > 0; o >>= 1) S[k] += __shfl_xor_sync(0xffffffffu, S[k], o);
  double beta = S[5] / S[0], g = 0.0, k = 0.0;
  const double m00 = S[2] * S[4] - S[3] * S[3], m01 = S[1] * S[4] - S[3] * S[2], m02 = S[1] * S[3] - S[2] * S[2];
  const double det = S[0] * m00 - S[1] * m01 + S[2] * m02;
  if (S[0] >= 4.0 && det > 1e-6 * S[0] * S[0] * S[0]) {
    beta = (S[5] * m00 - S[1] * (S[6] * S[4] - S[3] * S[7]) + S[2] * (S[6] * S[3] - S[2] * S[7])) / det;
    g = (S[0] * (S[6] * S[4] - S[7] * S[3]) - S[5] * m01 + S[2] * (S[1] * S[7] - S[2] * S[6])) / det;
    k = (S[0] * (S[2] * S[7] - S[3] * S[6]) - S[1] * (S[1] * S[7] - S[2] * S[6]) + S[5] * m02) / det;
  }
  float el = INFINITY, eh = -INFINITY;
#pragma unroll
  for (int q = 0; q < TK_SLOTS; ++q) {
    if (q < q0 || q >= q0 + ks || q * 32 + lane >= n1) continue;
    const double x = (f[q][0] - mid) * invA;
    const float r = (float)((double)f[q][1] - beta - x * (g + x * k));
    el = fminf(el, r); eh = fmaxf(eh, r);
  }
  eh = warp_max(eh); el = -warp_max(-el);
  const float mide = 0.5f * (eh + el);
  const float tilt = 1.f + fabsf((float)g) * invA;
  R[0] = A * tilt;
  R[1] = (float)fabs(k) * tilt;
  R[2] = 0.5f * (eh - el);
  R[3] = 0.5f * (hc - lc);
  gamma = (float)(g * invA);
  kappa = (float)(k * invA * invA);
  const double bc = beta + (double)mide;
  for (int c = 0; c < 3; ++c)
    uc[c] = (double)first[c] + (double)mid * e[c] + bc * e[3 + c] + (double)midc * e[6 + c];
}

__global__ void __launch_bounds__(128) k_track_plan(const PlanArgs a) {
  const int lane = threadIdx.x & 31;
  const int g = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (g >= a.ngroups) return;
  const int pair = g / a.gpp, s0 = (g - pair * a.gpp) * TK_GROUP;
  const int nv = min(TK_GROUP, a.steps - s0);
  float p[TK_SLOTS][3];
  bool fine = true;
#pragma unroll
  for (int q = 0; q < TK_SLOTS; ++q) {
    const int st = s0 + q * 32 + lane;
    p[q][0] = p[q][1] = p[q][2] = 0.f;
    if (q * 32 + lane < nv) {
      const int64_t i = (int64_t)st * 2 * a.nbl + pair;
      p[q][0] = a.u[i]; p[q][1] = a.v[i]; p[q][2] = a.w[i];
      // outside the exact phase range (or not a number): left to the per-term kernel, which flags it
      fine &= fabsf(p[q][0]) < (float)kMaxUvwF32X && fabsf(p[q][1]) < (float)kMaxUvwF32X &&
              fabsf(p[q][2]) < (float)kMaxUvwF32X;
    }
  }
  int mode = -1;
  float best = 0.f;
  double uc[3];
  float e[9], R[4], gamma, kappa;
  if (__all_sync(0xffffffffu, fine)) {
    // Issue cycles of a warp for each 32 terms, from the instruction counts of
    // k_track_sum: pixel steps, reduction, evaluation; and what the blocks on the
    // horizon cost more: a quad of each lower level, and 64-pixel parts term by
    // term for the steps that the horizon crosses there.  It sweeps `turn` radians
    // over the group (the first endpoint's motion), so that a share of the visible
    // blocks in proportion to turn + 2 r lies on it; the factor 0.28 and the line at
    // 10 were measured over nside 256 to 1024, lunar and Earth orbits, days 1 to 8
    // (0.14 to 1.1 and 7 to 15 tried: within 15 % of the best shape in each).  The
    // per-term kernel takes about 18 cycles for each 32 terms, and this one issues
    // 0.6 to 0.7 instructions a cycle.
    const float c_pix[TK_SETS] = {90.f, 130.f, 170.f}, c_red[TK_SETS] = {50.f, 70.f, 95.f}, c_eval[TK_SETS] = {125.f, 145.f, 165.f};
    float turn = 0.f;
    if (a.blockage) {
      const int64_t i0 = (int64_t)s0 * 2 * a.nbl + pair, i1 = (int64_t)(s0 + nv - 1) * 2 * a.nbl + pair;
      const float k0 = a.in1[i0], k1 = a.in1[i1];
      const float dx = a.x1[i1] * k1 - a.x1[i0] * k0, dy = a.y1[i1] * k1 - a.y1[i0] * k0, dz = a.z1[i1] * k1 - a.z1[i0] * k0;
      turn = sqrtf(dx * dx + dy * dy + dz * dz) / (float)max(nv - 1, 1);   // a step
    }
    const float r64 = __uint_as_float(a.rmax[0]);
    best = 10.f;
    for (int ls = 0; ls <= 2; ++ls) {
      const int ks = 1 << ls;
      float M[4] = {0.f, 0.f, 0.f, 0.f};
      for (int q0 = 0; q0 < TK_SLOTS; q0 += ks) {
        sub_frame(p, nv, lane, q0, ks, uc, e, gamma, kappa, R);
        for (int c = 0; c < 4; ++c) M[c] = fmaxf(M[c], R[c]);
      }
      bool fits = false;
      const float fill = (float)nv / (float)(ks * 32 * ((nv + ks * 32 - 1) / (ks * 32)));
      const float crossed = fminf(32.f * ks, 1.f + 2.f * r64 / fmaxf(turn, 1e-6f));   // steps on the horizon in a 64-pixel part
      for (int lev = 0; lev <= a.max_level; ++lev) {
        const float r = __uint_as_float(a.rmax[lev]);
        const float k = 6.2831855f * r, X1 = k * M[0], X2 = k * M[1], E = k * sqrtf(M[2] * M[2] + M[3] * M[3]);
        int tried = -1;
        for (int t = 0; t < kSeriesTables; ++t) {
          const int set = a.box[t].set;
          if (set == tried || !(X1 <= a.box[t].x1 && X2 <= a.box[t].x2 && E <= a.box[t].e)) continue;
          tried = set;   // (the tables are sorted by shape)
          fits = true;
          const float P = (float)tk_block(lev);
          float node = P * (1.f / 32.f) * c_pix[set] + c_red[set] + ks * c_eval[set];
          if (a.blockage)
            node += fminf(1.f, 0.28f * (turn * 32.f * ks + 2.f * r)) *
                    (lev * (P * (1.f / 32.f) * c_pix[set] + 4.f * (c_red[set] + c_eval[set])) + P * (1.f / 64.f) * (150.f + 70.f * crossed));
          const float cost = node / (ks * P * fill);
          if (cost < best) { best = cost; mode = set | (ls << 4) | (lev << 8) | (t << 12); }
        }
      }
      if (!fits) break;   // longer sub-groups extend further
    }
  }
  if (mode >= 0) {
    const int ks = 1 << ((mode >> 4) & 15);
    for (int q0 = 0; q0 < TK_SLOTS; q0 += ks) {
      sub_frame(p, nv, lane, q0, ks, uc, e, gamma, kappa, R);
      if (lane == 0) {
        TrackSub& s = a.plan[g].sub[q0 / ks];
        for (int c = 0; c < 3; ++c) s.uc[c] = uc[c];
        for (int c = 0; c < 9; ++c) s.e[c] = e[c];
        s.gamma = gamma;
        s.kappa = kappa;
      }
    }
  }
  if (lane == 0) {
    a.plan[g].mode = mode;
    a.plan[g].cost = best;
  }
}

// Exclusive scans over the groups in (step block, pair) order, one CTA: place of
// each factored group in their list, and baselines left to the per-term kernel
// before each group.  That list keeps the callers' order (steps, then pairs):
// with a pair's consecutive steps side by side instead, a warp's baselines span
// 32 steps of horizon motion and the per-term kernel ran up to 15 % slower.
constexpr float kTermCycles = 18.f;   // k_stage1, a warp's cycles for each 32 terms

__global__ void __launch_bounds__(1024) k_track_scan(TrackPlan* plan, int ngroups, int nbl, int gpp, int steps, int* off,
                                                     int* left, int* count, int* queue) {
  __shared__ unsigned long long s_w[32];
  __shared__ unsigned long long s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // What the factored groups are expected to save, of the whole call.  Below 8 %
  // none is factored: the baselines left fill the per-term kernel's warps less well
  // (their horizons differ more) and there are two tails; calls of 2e9 to 8e9 terms
  // with 2 to 6 % expected ran 1 to 8 % slower than without.
  float save = 0.f;
  for (int s = threadIdx.x; s < ngroups; s += 1024) {
    const int j = s / nbl;
    const TrackPlan& t = plan[(s - j * nbl) * gpp + j];
    if (t.mode >= 0) save += (kTermCycles - t.cost) / kTermCycles * (float)min(TK_GROUP, steps - j * TK_GROUP);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) save += __shfl_xor_sync(0xffffffffu, save, o);
  if (lane == 0) s_w[warp] = (unsigned long long)__float_as_uint(save);
  if (threadIdx.x == 0) s_base = 0ull;
  __syncthreads();
  save = 0.f;
  for (int w = 0; w < 32; ++w) save += __uint_as_float((unsigned)s_w[w]);
  if (!(save >= 0.08f * (float)steps * (float)nbl))
    for (int s = threadIdx.x; s < ngroups; s += 1024) plan[s].mode = -1;
  __syncthreads();
  for (int g0 = 0; g0 < ngroups; g0 += 1024) {
    const int s = g0 + threadIdx.x;
    unsigned long long v = 0ull;   // factored groups << 32 | baselines left
    if (s < ngroups) {
      const int j = s / nbl;
      v = plan[(s - j * nbl) * gpp + j].mode >= 0 ? (1ull << 32) : (unsigned long long)min(TK_GROUP, steps - j * TK_GROUP);
    }
    unsigned long long inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned long long t = __shfl_up_sync(0xffffffffu, inc, o);
      if (lane >= o) inc += t;
    }
    if (lane == 31) s_w[warp] = inc;
    __syncthreads();
    unsigned long long before = s_base;
    for (int w = 0; w < warp; ++w) before += s_w[w];
    const unsigned long long ex = before + inc - v;
    if (s < ngroups) {
      off[s] = (int)(ex >> 32);
      left[s] = (int)(ex & 0xffffffffull);
    }
    __syncthreads();
    if (threadIdx.x == 1023) s_base = before + inc;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    count[0] = (int)(s_base >> 32);
    count[1] = (int)(s_base & 0xffffffffull);
    // work queues of the per-term kernel: over every baseline, over the list
    constexpr int kNone = 1 << 30;
    queue[0] = count[0] > 0 ? kNone : 0;
    queue[1] = count[0] > 0 ? 0 : kNone;
    queue[2] = 0;   // k_track_sum
  }
}

// Lists, and the factored groups' baselines in group order (the steps of one
// pair are 2 nbl apart in the caller's arrays).
struct PackArgs {
  const float *u, *v, *w, *x1, *y1, *z1, *in1, *x2, *y2, *z2, *in2, *cp1, *cp2;
  float cosphi;
  int nbl, steps, gpp, ngroups, blockage;
  const TrackPlan* plan;
  const int *off, *left, *count;
  int *list, *direct;
  float4 *q0, *d1, *d2, *p1, *p2;
  float* t2;
};

__global__ void __launch_bounds__(128) k_track_pack(const PackArgs a) {
  const int lane = threadIdx.x & 31;
  const int g = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (g >= a.ngroups) return;
  const int pair = g / a.gpp, s0 = (g - pair * a.gpp) * TK_GROUP;
  const int nv = min(TK_GROUP, a.steps - s0);
  const bool fast = a.plan[g].mode >= 0;
  const int j = g - pair * a.gpp, s = j * a.nbl + pair;
  if (fast && lane == 0) a.list[a.off[s]] = g;
  // the left baselines of this step block: nd pairs a step, this pair's rank among them
  const int first = a.left[j * a.nbl], last = j + 1 < a.gpp ? a.left[(j + 1) * a.nbl] : a.count[1];
  const int nd = (last - first) / nv, rank = (a.left[s] - first) / nv;
  for (int q = 0; q < TK_SLOTS; ++q) {
    const int k = q * 32 + lane;
    if (k >= nv) continue;
    const int st = s0 + k;
    if (!fast) {
      a.direct[first + k * nd + rank] = st * a.nbl + pair;
      continue;
    }
    const int64_t i = (int64_t)st * 2 * a.nbl + pair;
    const int64_t o = (int64_t)g * TK_GROUP + k;
    float t1 = 0.f;
    if (a.blockage) {
      const float x1 = a.x1[i], y1 = a.y1[i], z1 = a.z1[i], i1 = a.in1[i];
      const float x2 = a.x2[i], y2 = a.y2[i], z2 = a.z2[i], i2 = a.in2[i];
      const float c1 = a.cp1 ? a.cp1[i] : a.cosphi, c2 = a.cp2 ? a.cp2[i] : a.cosphi;
      a.d1[o] = make_float4(x1 * i1, y1 * i1, z1 * i1, c1);
      a.d2[o] = make_float4(x2 * i2, y2 * i2, z2 * i2, c2);
      a.p1[o] = make_float4(x1, y1, z1, horizon_sine(a.d1[o]));
      a.p2[o] = make_float4(x2, y2, z2, horizon_sine(a.d2[o]));
      t1 = occ_threshold(i1, c1);
      a.t2[o] = occ_threshold(i2, c2);
    }
    a.q0[o] = make_float4(a.u[i], a.v[i], a.w[i], t1);
  }
}

// ---------------------------------------------------------------------------
// Classes of a lane's slots, two bits each.
__device__ __forceinline__ int cls_get(int c, int q) { return (c >> (2 * q)) & 3; }
__device__ __forceinline__ int cls_put(int c, int q, int v) { return (c & ~(3 << (2 * q))) | (v << (2 * q)); }

// Included (baseline, block) pairs of a sub-group up to which four 64-pixel parts
// of a block are summed term by term rather than through their moments.
constexpr int kFewVisible = 24;

struct TrackWarp {               // one warp's group
  double2 acc[TK_SLOTS][32];
  double dx[TK_SLOTS][32], dy[TK_SLOTS][32], dz[TK_SLOTS][32];
  float a[TK_SLOTS][32], b[TK_SLOTS][32], c[TK_SLOTS][32];
  float4 d1[TK_SLOTS][32], d2[TK_SLOTS][32];
  float s1[TK_SLOTS][32], s2[TK_SLOTS][32];
  float mom[TK_QUAD][2 * TK_JMAX];
  float scale[2 * TK_JMAX];      // of the group's table
  TrackPlan plan;
};
struct TrackSmem {
  TrackWarp w[TK_WARPS];
  unsigned char dest[TK_SETS][2 * TK_JMAX];
};

// Turn phase of a (baseline, pixel) term as angle bits, see vb_stage1.cuh; the
// products are summed before the one rounding to the 2^-23-turn grid (one FP64
// operation more a pixel and group, which all its steps share).
__device__ __forceinline__ void phase_cs(double U, double V, double W, float l, float m, float n, unsigned flip, float& s,
                                         float& c) {
  const double t = fma(U, (double)l, fma(V, (double)m, W * (double)n)) + kMagic;
  const unsigned kb = ((unsigned)__double2loint(t) & 0x7FFFFFu) ^ flip;
  __sincosf(__fmaf_rn(__uint_as_float(kb), kAngScale, -kTwoPiF), &s, &c);
}

// (l, m, n, B) of pixel p0 + j of a block of np; B = 0 past its end (and the
// position of some pixel of the sky).
__device__ __forceinline__ float4 pixel_at(const TrackArgs& a, int64_t p0, int np, int j) {
  const int64_t p = min(p0 + (j < np ? j : 0), a.npix - 1);
  return make_float4(__ldg(a.l + p), __ldg(a.m + p), __ldg(a.n + p), j < np ? __ldg(a.B + p) : 0.f);
}

// Moments of one sub-group over four neighbouring blocks (lane >> 3 is the
// lane's block, p0, np, cen its pixels and centre) into the warp's shared-memory
// slots, scaled by their coefficients.  Eight lanes a block: the transposed
// reduction of 2 J values then costs 7/8 N shuffles for four blocks instead of
// 31/32 N for each (a quarter of a 64-pixel block's time, 8 % of a 256-pixel one).
// With q = 2 kappa eta / (2 pi r) the generating function
// e^{i (a tau + a^2 q / 2)} = sum_n (i a)^n g_n / n! has
//   g_n = tau g_{n-1} - i (n - 1) q g_{n-2},
// so that the curve costs five operations a power and the moments of z g_n
// (and, for the first half of them, of z g_n eta and z g_n zeta: the residuals
// from the curve to first order) are all that the block contributes.
template <int SET>
__device__ __forceinline__ void track_moments(const TrackArgs& ta, int64_t p0, int np, int P, const TrackSub& sub, const float4 cen,
                                              float inv_r, const float* scale, const unsigned char* dest, float* mom, int lane) {
  using S = Shape<SET>;
  const double U = sub.uc[0], V = sub.uc[1], W = sub.uc[2];
  float e[9];
#pragma unroll
  for (int c = 0; c < 9; ++c) e[c] = sub.e[c] * inv_r;
#pragma unroll
  for (int c = 0; c < 3; ++c) e[c] = fmaf(sub.gamma, e[3 + c], e[c]);
  const float kq = sub.kappa * inv_r * 0.31830988618379067f;   // 2 kappa / (2 pi r)
  f2 v2[S::J];   // (re, im)
#pragma unroll
  for (int i = 0; i < S::J; ++i) v2[i] = 0ull;
  // odd pixels half a turn on with a negated brightness, as in the per-term kernel
  const unsigned flip = (lane & 1) ? 0x4B400000u : 0x4B000000u;
  const int l8 = lane & 7;
  float4 f = pixel_at(ta, p0, np, l8);
#pragma unroll 1
  for (int j0 = 0; j0 < P; j0 += 8) {
    const float4 next = pixel_at(ta, p0, np, j0 + 8 + l8);   // loaded while this step computes
    float zi, zr;
    phase_cs(U, V, W, f.x, f.y, f.z, flip, zi, zr);
    const float Bp = (lane & 1) ? -f.w : f.w;
    const float dx = f.x - cen.x, dy = f.y - cen.y, dz = f.z - cen.z;
    const float tau = fmaf(dx, e[0], fmaf(dy, e[1], dz * e[2]));
    const float eta = fmaf(dx, e[3], fmaf(dy, e[4], dz * e[5]));
    const float zet = fmaf(dx, e[6], fmaf(dy, e[7], dz * e[8]));
    const float q = kq * eta;
    const f2 eta2 = f2_make(eta, eta), zet2 = f2_make(zet, zet);
    float r0 = 0.f, i0 = 0.f, r1 = zr * Bp, i1 = zi * Bp;   // g_{n-1}, g_n
#pragma unroll
    for (int n = 0; n < S::N; ++n) {
      const f2 g = f2_make(r1, i1);
      v2[n] = f2_add(v2[n], g);
      if (n < S::NE) {
        v2[S::N + n] = f2_fma(eta2, g, v2[S::N + n]);
        v2[S::N + S::NE + n] = f2_fma(zet2, g, v2[S::N + S::NE + n]);
      }
      if (n + 1 < S::N) {
        const float nq = (float)n * q;
        const float r2 = n ? fmaf(tau, r1, nq * i0) : tau * r1;
        const float i2 = n ? fmaf(tau, i1, -nq * r0) : tau * i1;
        r0 = r1; i0 = i1;
        r1 = r2; i1 = i2;
      }
    }
    f = next;
  }
  float v[2 * S::J];
#pragma unroll
  for (int i = 0; i < S::J; ++i) {
    const float2 t = f2_split(v2[i]);
    v[2 * i] = t.x;
    v[2 * i + 1] = t.y;
  }
  constexpr int N = 2 * S::J;
  fold_half<N, 4>(v, lane & 4);
  fold_half<N / 2, 2>(v, lane & 2);
  fold_half<N / 4, 1>(v, lane & 1);
  const int base = ((lane & 4) ? N / 2 : 0) + ((lane & 2) ? N / 4 : 0) + ((lane & 1) ? N / 8 : 0);
  __syncwarp();   // the previous moments are read
#pragma unroll
  for (int k = 0; k < N / 8; ++k) mom[(lane >> 3) * 2 * TK_JMAX + dest[base + k]] = v[k] * scale[base + k];
  __syncwarp();
}

// Value of one baseline from the scaled moments: its place a on the curve and
// its residuals b (towards the sagitta) and c (across).
template <int SET>
__device__ __forceinline__ float2 track_eval(const float* mom, float a, float b, float c) {
  using S = Shape<SET>;
  const f2* m = reinterpret_cast<const f2*>(mom);
  const f2 a2 = f2_make(a, a);
  auto horner = [&](int o, int n) {
    f2 h = m[o + n - 1];
#pragma unroll
    for (int i = n - 2; i >= 0; --i) h = f2_fma(h, a2, m[o + i]);
    return h;
  };
  const f2 h0 = horner(0, S::N), hb = horner(S::N, S::NE), hc = horner(S::N + S::NE, S::NE);
  return f2_split(f2_fma(f2_make(b, b), hb, f2_fma(f2_make(c, c), hc, h0)));
}

__device__ __forceinline__ int track_tile_class(const TrackArgs& a, const float4 d1, const float4 d2, int tile) {
  const float cx = a.tcx[tile], cy = a.tcy[tile], cz = a.tcz[tile], cA = a.tcosA[tile], sA = a.tsinA[tile];
  bool vis1, hid1, vis2, hid2;
  cone_classify(cone_dot(d1.x, d1.y, d1.z, cx, cy, cz), cA, sA, d1.w, vis1, hid1);
  cone_classify(cone_dot(d2.x, d2.y, d2.z, cx, cy, cz), cA, sA, d2.w, vis2, hid2);
  return (hid1 || hid2) ? kClsHid : ((vis1 && vis2 && !a.mask_visible) ? kClsVis : kClsMix);
}

// FP64 rotation of one baseline's block sum into its total.
__device__ __forceinline__ void track_add(const TrackArgs& a, TrackWarp& w, int q, int lane, const float4 cen, int64_t o, float hr,
                                          float hi) {
  double t = fma(w.dx[q][lane], (double)cen.x, fma(w.dy[q][lane], (double)cen.y, w.dz[q][lane] * (double)cen.z));
  if (a.raw) t -= (double)a.q0[o].z;
  double es, ec;
  turn_cs(t, es, ec);
  double2 acc = w.acc[q][lane];
  acc.x = fma((double)hr, ec, fma(-(double)hi, es, acc.x));
  acc.y = fma((double)hr, es, fma((double)hi, ec, acc.y));
  w.acc[q][lane] = acc;
}

// Terms one by one for the baselines of `cls` (kClsVis: every pixel, kClsMix:
// the per-pixel occlusion test, 0: none) over a block of up to 64 pixels, two a
// lane.  The block's z_p are formed once per sub-group, then each baseline's
// terms are z_p e^{i (a tau + b eta + c zeta)} with an exact small angle.  Out of
// line: a few per cent of the terms, whose registers the moment loop does not
// have.
__device__ __forceinline__ void track_terms(const TrackArgs& a, int64_t p0, int np, int cls, const float4 cen, float inv_r,
                                         int ks, int64_t o0, int lane) {
  // (from its own declaration: through a reference the accesses would be generic)
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TrackWarp& w = reinterpret_cast<TrackSmem*>(smem_raw)->w[threadIdx.x >> 5];
  const float kr = 6.28318530717958647692f / inv_r;
  const unsigned flip = (lane & 1) ? 0x4B400000u : 0x4B000000u;
  float4 f[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) f[h] = pixel_at(a, p0, np, 32 * h + lane);
#pragma unroll 1
  for (int q0 = 0; q0 < TK_SLOTS; q0 += ks) {
    bool any = false;
    for (int q = q0; q < q0 + ks; ++q) any |= cls_get(cls, q) != kClsHid;
    if (!__any_sync(0xffffffffu, any)) continue;
    const TrackSub& sub = w.plan.sub[q0 / ks];
    float zr[2], zi[2], tau[2], eta[2], zet[2];
    const float kq = sub.kappa / kr;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      phase_cs(sub.uc[0], sub.uc[1], sub.uc[2], f[h].x, f[h].y, f[h].z, flip, zi[h], zr[h]);
      const float Bp = (lane & 1) ? -f[h].w : f[h].w;
      zr[h] *= Bp;
      zi[h] *= Bp;
      const float dx = (f[h].x - cen.x) * inv_r, dy = (f[h].y - cen.y) * inv_r, dz = (f[h].z - cen.z) * inv_r;
      tau[h] = fmaf(dx, sub.e[0], fmaf(dy, sub.e[1], dz * sub.e[2]));
      eta[h] = fmaf(dx, sub.e[3], fmaf(dy, sub.e[4], dz * sub.e[5]));
      zet[h] = fmaf(dx, sub.e[6], fmaf(dy, sub.e[7], dz * sub.e[8]));
    }
#pragma unroll 1
    for (int q = q0; q < q0 + ks; ++q) {
      const int c = cls_get(cls, q);
      unsigned mm = __ballot_sync(0xffffffffu, c != kClsHid);
      if (!mm) continue;
      const int64_t o = o0 + q * 32;
      float4 e1 = make_float4(0.f, 0.f, 0.f, 0.f), e2 = e1;
      float t1 = -INFINITY, t2 = -INFINITY;
      if (c == kClsMix) {
        e1 = a.p1[o];
        e2 = a.p2[o];
        t1 = a.q0[o].w;
        t2 = a.t2[o];
      }
      float hr = 0.f, hi = 0.f;
      while (mm) {
        const int src = __ffs(mm) - 1;
        mm &= mm - 1;
        const float ka = w.a[q][src], kc = w.c[q][src];
        const float kb = fmaf(ka, fmaf(ka, kq, sub.gamma), w.b[q][src]);   // place on the curve and its residual
        const float x1 = __shfl_sync(0xffffffffu, e1.x, src), y1 = __shfl_sync(0xffffffffu, e1.y, src), z1 = __shfl_sync(0xffffffffu, e1.z, src);
        const float x2 = __shfl_sync(0xffffffffu, e2.x, src), y2 = __shfl_sync(0xffffffffu, e2.y, src), z2 = __shfl_sync(0xffffffffu, e2.z, src);
        const float c1 = __shfl_sync(0xffffffffu, t1, src), c2 = __shfl_sync(0xffffffffu, t2, src);
        float sr = 0.f, si = 0.f;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const float g1 = f[h].x * x1 + f[h].y * y1 + f[h].z * z1;
          const float g2 = f[h].x * x2 + f[h].y * y2 + f[h].z * z2;
          const bool inc = !(g1 < c1 || g2 < c2);
          float s, k;
          __sincosf(fmaf(ka, tau[h], fmaf(kb, eta[h], kc * zet[h])), &s, &k);
          const float xr = inc ? zr[h] : 0.f, xi = inc ? zi[h] : 0.f;
          sr = fmaf(xr, k, fmaf(-xi, s, sr));
          si = fmaf(xr, s, fmaf(xi, k, si));
        }
        // (re, im) in the two halves of the warp, then five steps in all
        const bool up = lane & 16;
        float v = up ? si : sr;
        v += __shfl_xor_sync(0xffffffffu, up ? sr : si, 16);
#pragma unroll
        for (int d = 8; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
        const float re = __shfl_sync(0xffffffffu, v, 0), im = __shfl_sync(0xffffffffu, v, 16);
        if (lane == src) { hr = re; hi = im; }
      }
      if (c != kClsHid) track_add(a, w, q, lane, cen, o, hr, hi);
    }
  }
}

// One step of the walk down the pixel blocks: four neighbouring blocks of level
// lev from pixel `base` (up to `end`), cls4 the slots' classes in each (a byte a
// block; slots that other blocks decide are hidden).  Baselines still undecided
// are classified against each block's cone; the included ones take the blocks'
// moments; the undecided ones are returned for the blocks' own four parts, or at
// 64 pixels take the per-pixel test.  A few included baselines in parts of 64
// pixels are summed term by term with those (not at the group's own level, where
// a tile that the upstream's cone test calls visible takes no test).
__device__ __forceinline__ unsigned track_quad(const TrackArgs& a, TrackSmem& sm, TrackWarp& w, int lev, bool top, int set, int ks,
                                            unsigned cls4, int64_t base, int64_t end, float inv_r, int64_t o0, int lane) {
  const int P = tk_block(lev);
  unsigned open4 = 0, rest4 = 0;
  if (a.blockage) {
#pragma unroll 1
    for (int n = 0; n < TK_QUAD; ++n) {
      const int64_t p0 = base + n * P;
      int c = (cls4 >> (8 * n)) & 255;
      if (p0 >= end) c = 0;
      if (__any_sync(0xffffffffu, c != 0)) {
        const TrackNode nd = a.node[lev][p0 / P];
#pragma unroll
        for (int q = 0; q < TK_SLOTS; ++q)
          if (cls_get(c, q) == kClsMix)
            c = cls_put(c, q, both_classes(endpoint_class(nd, w.d1[q][lane], w.s1[q][lane]),
                                           endpoint_class(nd, w.d2[q][lane], w.s2[q][lane])));
      }
      cls4 = (cls4 & ~(255u << (8 * n))) | ((unsigned)c << (8 * n));
    }
    // undecided slots (class 2: the high bit of each pair)
    static_assert(kClsMix == 2 && kClsVis == 1, "class bits");
    open4 = cls4 & 0xAAAAAAAAu;
  }
  unsigned vis4 = cls4 & 0x55555555u;
  if (end < base + TK_QUAD * P && !a.blockage)
    for (int n = 0; n < TK_QUAD; ++n)
      if (base + n * P >= end) vis4 &= ~(255u << (8 * n));
  const int64_t mine = base + (lane >> 3) * P;
  const int np = (int)max((int64_t)0, min((int64_t)P, end - mine));
  const float4 cen = a.node[lev][min(mine, end - 1) / P].cen;
  for (int q0 = 0; q0 < TK_SLOTS; q0 += ks) {
    const unsigned slots = ((1u << (2 * ks)) - 1u) << (2 * q0);
    const unsigned take = vis4 & (slots * 0x01010101u);
    if (!__any_sync(0xffffffffu, take != 0)) continue;
    if (lev == 0 && !top && __reduce_add_sync(0xffffffffu, (unsigned)__popc(take)) <= kFewVisible) {
      rest4 |= take;
      continue;
    }
    const TrackSub& sub = w.plan.sub[q0 / ks];
    if (set == 0) track_moments<0>(a, mine, np, P, sub, cen, inv_r, w.scale, sm.dest[0], w.mom[0], lane);
    else if (set == 1) track_moments<1>(a, mine, np, P, sub, cen, inv_r, w.scale, sm.dest[1], w.mom[0], lane);
    else track_moments<2>(a, mine, np, P, sub, cen, inv_r, w.scale, sm.dest[2], w.mom[0], lane);
#pragma unroll 1
    for (int q = q0; q < q0 + ks; ++q) {
      const float ka = w.a[q][lane], kb = w.b[q][lane], kc = w.c[q][lane];
#pragma unroll 1
      for (int n = 0; n < TK_QUAD; ++n) {
        const bool in = (take >> (8 * n + 2 * q)) & 1u;
        if (!in) continue;
        const float2 h = set == 0   ? track_eval<0>(w.mom[n], ka, kb, kc)
                         : set == 1 ? track_eval<1>(w.mom[n], ka, kb, kc)
                                    : track_eval<2>(w.mom[n], ka, kb, kc);
        track_add(a, w, q, lane, a.node[lev][(base + n * P) / P].cen, o0 + q * 32, h.x, h.y);
      }
    }
  }
  if (lev > 0) return open4;
  rest4 |= open4;
#pragma unroll 1
  for (int n = 0; n < TK_QUAD; ++n) {
    const int c = (rest4 >> (8 * n)) & 255;
    if (!__any_sync(0xffffffffu, c != 0)) continue;
    const int64_t p0 = base + n * P;
    track_terms(a, p0, (int)min((int64_t)P, end - p0), c, a.node[0][p0 / P].cen, inv_r, ks, o0, lane);
  }
  return 0;
}

__global__ void __launch_bounds__(TK_THREADS, 3) k_track_sum(const __grid_constant__ TrackArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TrackSmem& sm = *reinterpret_cast<TrackSmem*>(smem_raw);
  const int lane = threadIdx.x & 31;
  TrackWarp& w = sm.w[threadIdx.x >> 5];
  asm volatile("griddepcontrol.launch_dependents;");   // the list kernel may take SMs that this one leaves
  const int nfast = a.count[0];
  const int n_items = nfast * a.nchunk;
  for (int i = threadIdx.x; i < TK_SETS * 2 * TK_JMAX; i += TK_THREADS) (&sm.dest[0][0])[i] = (&a.dest[0][0])[i];
  __syncthreads();

  // Work item: one group over one pixel chunk, by one warp (the warps differ in
  // how many baselines the horizon cuts in a block: a barrier would make each
  // block as slow as its slowest group).  Chunk-major, so that the warps running
  // at one time read the same pixels from L2.
  for (;;) {
    int item = 0;
    if (lane == 0) item = atomicAdd(a.queue, 1);
    item = __shfl_sync(0xffffffffu, item, 0);
    if (item >= n_items) break;
    const int chunk = item / nfast;
    const int g = a.list[item - chunk * nfast];

    // --- the group -------------------------------------------------------------
    const int mode = a.plan[g].mode, set = mode & 15, ks = 1 << ((mode >> 4) & 15), level = (mode >> 8) & 15;
    const float r = __uint_as_float(a.rmax[level]), inv_r = 1.f / r;
    const int pair = g / a.gpp, st0 = (g - pair * a.gpp) * TK_GROUP;
    const int nv = min(TK_GROUP, a.steps - st0);
    const int64_t o0 = (int64_t)g * TK_GROUP + lane;
    int act = 0;   // classes before any test
    __syncwarp();
    {
      const int* src = reinterpret_cast<const int*>(a.plan + g);
      int* dst = reinterpret_cast<int*>(&w.plan);
      for (int i = lane; i < (int)(sizeof(TrackPlan) / sizeof(int)); i += 32) dst[i] = src[i];
      for (int i = lane; i < 2 * TK_JMAX; i += 32) w.scale[i] = a.scale[mode >> 12][i];
      __syncwarp();
      const float kr = 6.28318530717958647692f * r;
      for (int q = 0; q < TK_SLOTS; ++q) {
        w.acc[q][lane] = make_double2(0.0, 0.0);
        if (q * 32 + lane >= nv) continue;
        act = cls_put(act, q, a.blockage ? kClsMix : kClsVis);
        const float4 u = a.q0[o0 + q * 32];
        const TrackSub& sub = w.plan.sub[q / ks];
        const double dx = (double)u.x - sub.uc[0], dy = (double)u.y - sub.uc[1], dz = (double)u.z - sub.uc[2];
        w.dx[q][lane] = dx; w.dy[q][lane] = dy; w.dz[q][lane] = dz;
        const float fx = (float)dx, fy = (float)dy, fz = (float)dz;
        const float ka = kr * fmaf(fx, sub.e[0], fmaf(fy, sub.e[1], fz * sub.e[2]));
        const float kb = kr * fmaf(fx, sub.e[3], fmaf(fy, sub.e[4], fz * sub.e[5]));
        w.a[q][lane] = ka;
        w.b[q][lane] = kb - ka * fmaf(ka, sub.kappa / kr, sub.gamma);
        w.c[q][lane] = kr * fmaf(fx, sub.e[6], fmaf(fy, sub.e[7], fz * sub.e[8]));
        if (a.blockage) {
          w.d1[q][lane] = a.d1[o0 + q * 32];
          w.d2[q][lane] = a.d2[o0 + q * 32];
          w.s1[q][lane] = a.p1[o0 + q * 32].w;
          w.s2[q][lane] = a.p2[o0 + q * 32].w;
        }
      }
      __syncwarp();
    }
    const int P = tk_block(level);
    const bool tc = a.tilecone && a.blockage;
    int tcls = act, tile = -1;

    const int64_t p_begin = (int64_t)chunk * a.chunk_pix;
    const int64_t p_end = min(a.npix, p_begin + a.chunk_pix);
    for (int64_t p0 = p_begin; p0 < p_end; p0 += TK_QUAD * P) {
      unsigned cls4 = (unsigned)act * 0x01010101u;
      if (tc) {   // class of the cull tile, as the upstream decides it
        cls4 = 0;
        for (int n = 0; n < TK_QUAD; ++n) {
          const int64_t pn = p0 + n * P;
          if (pn >= p_end) break;
          const int t = (int)(pn / a.cull_tile);
          if (t != tile) {
            tile = t;
            tcls = act;
#pragma unroll
            for (int q = 0; q < TK_SLOTS; ++q)
              if (cls_get(tcls, q) != kClsHid)
                tcls = cls_put(tcls, q, track_tile_class(a, w.d1[q][lane], w.d2[q][lane], t));
          }
          cls4 |= (unsigned)tcls << (8 * n);
        }
      }
      // walk down: the quad at the group's level, then the four parts of each
      // block that some baselines leave undecided (one call site: the code of a
      // quad is most of the kernel's, and shared memory must stay visible as such)
      int lev = level;
      int64_t base = p0, end = p_end;
      unsigned open2 = 0, open1 = 0;   // undecided slots of the blocks of level 2 and 1 still to walk
      int64_t base1 = p0;
      for (;;) {
        const unsigned open = track_quad(a, sm, w, lev, lev == level, set, ks, cls4, base, end, inv_r, o0, lane);
        if (lev == 2) open2 = open;
        if (lev == 1) { open1 = open; base1 = base; }
        const unsigned any1 = __reduce_or_sync(0xffffffffu, open1);
        const unsigned any2 = __reduce_or_sync(0xffffffffu, open2);
        if (any1) {
          const int n = (__ffs(any1) - 1) >> 3;
          base = base1 + n * tk_block(1);
          end = min(p_end, base + tk_block(1));
          cls4 = ((open1 >> (8 * n)) & 255u) * 0x01010101u;
          open1 &= ~(255u << (8 * n));
          lev = 0;
        } else if (any2) {
          const int n = (__ffs(any2) - 1) >> 3;
          base = p0 + n * tk_block(2);
          end = min(p_end, base + tk_block(2));
          cls4 = ((open2 >> (8 * n)) & 255u) * 0x01010101u;
          open2 &= ~(255u << (8 * n));
          lev = 1;
        } else {
          break;
        }
      }
    }
    for (int q = 0; q < TK_SLOTS; ++q) {
      const int k = q * 32 + lane;
      if (k >= nv) continue;
      const int64_t ih = (int64_t)(st0 + k) * a.nbl + pair;
      const double2 acc = w.acc[q][lane];
      a.partial[(int64_t)chunk * a.n_half + ih] = make_double2(acc.x, -acc.y);
    }
  }
}

// ---------------------------------------------------------------------------
// Coefficient and sign of each part of a moment: i^n / n! (one more i in the
// residual terms) times the table's correction.
static void series_scale(const SeriesTable& t, float* scale) {
  for (int o = 0; o < 2 * t.n; ++o) {
    const int n = o < t.n ? o : (o - t.n) % (t.n / 2);
    const int d = (n + (o < t.n ? 0 : 1)) & 3;
    double f = o < t.n ? t.main[n] : t.res[n];
    for (int k = 2; k <= n; ++k) f /= k;
    const double sre = (d == 0 || d == 1) ? f : -f;   // re -> re, im, -re, -im
    const double sim = (d == 0 || d == 3) ? f : -f;   // im -> im, -re, -im, re
    scale[2 * o] = (float)sre;
    scale[2 * o + 1] = (float)sim;
  }
}

// Where multiplication by that power of i puts the two parts.
static void series_dest(int N, unsigned char* dest) {
  for (int o = 0; o < 2 * N; ++o) {
    const int d = (o < N ? o : (o - N) % (N / 2) + 1) & 3;
    dest[2 * o] = (unsigned char)(2 * o + (d & 1));
    dest[2 * o + 1] = (unsigned char)(2 * o + 1 - (d & 1));
  }
}

// Track groups are in use for the FP32 sum with FP64 phase where the call is
// large enough that the planning launches and a second tail (40 to 60 us) do not
// count, and where groups and pixel blocks exist: 96 steps (a group of 128 mostly
// filled), 6e9 terms (3 ms on the per-term kernel), cull tiles of 64 pixels or more.
// One B200, 28 pairs, without / with: 4.4e9 terms (nside 256, 200 steps): lunar, 300 m
// 2.21 / 1.34 ms, 30 m 2.20 / 1.58, Earth orbits, 300 m 2.10 / 2.16; 8.8e9 (400 steps):
// 4.23 / 1.98, 4.17 / 2.40 and 4.03 / 3.92; nothing to factor, 8.3e9: 3.93 / 3.95.
void track_plan(Stage1Plan* p, int items_per_cta) {
  p->track = 0;
  const int steps = p->n_half / p->nbl;
  if (p->precision != VB_PREC_FP32_FP64PH || steps < 96 || (double)p->n_half * (double)p->npix < 6e9) return;
  int level = TK_LEVELS - 1;
  if (p->cull == VB_CULL_TILECONE) {
    if (p->cull_tile < tk_block(0)) return;
    while (tk_block(level) > p->cull_tile) --level;
  }
  p->trk_level = level;
  p->trk_steps = steps;
  p->trk_gpp = (int)ceil_div(steps, TK_GROUP);
  const int64_t ng = (int64_t)p->trk_gpp * p->nbl;
  if (ng * TK_GROUP > INT32_MAX) return;
  p->trk_groups = (int)ng;
  // work items (group x pixel chunk, a warp each): enough per resident warp that
  // the queue's tail stays short, chunks of 4096 pixels at least
  const int64_t warps = (int64_t)sm_count() * 12;
  int64_t nchunk = ceil_div(warps * (items_per_cta > 0 ? std::min(items_per_cta, 48) : 40), ng);
  nchunk = std::max<int64_t>(1, std::min<int64_t>(nchunk, ceil_div(p->npix, TK_CHUNK)));
  const int64_t chunk = ceil_div(ceil_div(p->npix, nchunk), TK_CHUNK) * TK_CHUNK;
  if (chunk > INT32_MAX / 2 || ng * ceil_div(p->npix, chunk) > INT32_MAX) return;
  p->trk_chunk_pix = (int)chunk;
  p->trk_nchunk = (int)ceil_div(p->npix, chunk);
  p->trk_grid = sm_count() * 3;
  p->track = 1;
}

void track_carve(const Stage1Plan& p, Carve& c, Stage1Buffers& x, bool pixels) {
  if (!p.track) return;
  if (pixels) {
    for (int lev = 0; lev < TK_LEVELS; ++lev) {
      x.trk.node[lev] = c.take<TrackNode>((size_t)ceil_div(p.npix, tk_block(lev)));
    }
    x.trk.rmax = c.take<unsigned>(TK_LEVELS);
  }
  const size_t slots = (size_t)p.trk_groups * TK_GROUP;
  x.trk.plan = c.take<TrackPlan>(p.trk_groups);
  x.trk.off = c.take<int>(p.trk_groups);
  x.trk.left = c.take<int>(p.trk_groups);
  x.trk.list = c.take<int>(p.trk_groups);
  x.trk.direct = c.take<int>(p.n_half);
  x.trk.count = c.take<int>(2);   // factored groups, baselines left
  x.trk.q0 = c.take<float4>(slots);
  if (p.blockage) {
    x.trk.d1 = c.take<float4>(slots);
    x.trk.d2 = c.take<float4>(slots);
    x.trk.p1 = c.take<float4>(slots);
    x.trk.p2 = c.take<float4>(slots);
    x.trk.t2 = c.take<float>(slots);
  }
}

int track_nodes(const float* B, const float* l, const float* m, const float* n, int64_t npix, TrackNode* const (&node)[3],
                unsigned* rmax, cudaStream_t s) {
  BlockArgs k{};
  k.B = B; k.l = l; k.m = m; k.n = n;
  k.npix = npix;
  k.nsuper = (int)ceil_div(npix, 1024);
  for (int lev = 0; lev < TK_LEVELS; ++lev) k.node[lev] = node[lev];
  k.rmax = rmax;
  VB_CUDA(cudaMemsetAsync(k.rmax, 0, TK_LEVELS * sizeof(unsigned), s));
  k_track_blocks<<<std::min(k.nsuper, sm_count() * 16), 256, 0, s>>>(k);
  VB_LAUNCH_CHECK();
  return VB_OK;
}

int track_prepare_pixels(const vb_sky* sky, const Stage1Plan& p, const Stage1Buffers& b, cudaStream_t s) {
  if (!p.track) return VB_OK;
  return track_nodes(sky->B, sky->l, sky->m, sky->n, p.npix, b.trk.node, b.trk.rmax, s);
}

// Plans the groups and builds both lists; the per-term kernel runs on
// b.trk.direct (b.trk.count[1] baselines; all of them in their own order when
// no group is factored).
int track_group(const vb_baselines* bl, const Stage1Plan& p, const Stage1Buffers& b, cudaStream_t s) {
  PlanArgs k{};
  k.u = bl->u; k.v = bl->v; k.w = bl->w;
  k.x1 = bl->x1; k.y1 = bl->y1; k.z1 = bl->z1; k.in1 = bl->invn1;
  k.nbl = p.nbl; k.steps = p.trk_steps; k.gpp = p.trk_gpp; k.ngroups = p.trk_groups; k.max_level = p.trk_level;
  k.blockage = p.blockage;
  k.rmax = b.trk.rmax;
  k.plan = b.trk.plan;
  for (int t = 0; t < kSeriesTables; ++t) k.box[t] = {kSeries[t].n / 4 - 2, kSeries[t].x1, kSeries[t].x2, kSeries[t].e};
  const int grid = (int)ceil_div(p.trk_groups, 4);
  k_track_plan<<<grid, 128, 0, s>>>(k);
  VB_LAUNCH_CHECK();
  k_track_scan<<<1, 1024, 0, s>>>(b.trk.plan, p.trk_groups, p.nbl, p.trk_gpp, p.trk_steps, b.trk.off, b.trk.left, b.trk.count,
                                   b.queue);
  VB_LAUNCH_CHECK();
  PackArgs q{};
  q.u = bl->u; q.v = bl->v; q.w = bl->w;
  q.x1 = bl->x1; q.y1 = bl->y1; q.z1 = bl->z1; q.in1 = bl->invn1;
  q.x2 = bl->x2; q.y2 = bl->y2; q.z2 = bl->z2; q.in2 = bl->invn2;
  q.cp1 = bl->cosphi1; q.cp2 = bl->cosphi2; q.cosphi = bl->cosphi;
  q.nbl = p.nbl; q.steps = p.trk_steps; q.gpp = p.trk_gpp; q.ngroups = p.trk_groups; q.blockage = p.blockage;
  q.plan = b.trk.plan; q.off = b.trk.off; q.left = b.trk.left; q.count = b.trk.count; q.list = b.trk.list; q.direct = b.trk.direct;
  q.q0 = b.trk.q0; q.d1 = b.trk.d1; q.d2 = b.trk.d2; q.p1 = b.trk.p1; q.p2 = b.trk.p2; q.t2 = b.trk.t2;
  k_track_pack<<<grid, 128, 0, s>>>(q);
  VB_LAUNCH_CHECK();
  return VB_OK;
}

int track_sum(const vb_sky* sky, const Stage1Plan& p, const Stage1Buffers& b, cudaStream_t s) {
  TrackArgs a{};
  a.B = sky->B; a.l = sky->l; a.m = sky->m; a.n = sky->n; a.npix = p.npix;
  a.chunk_pix = p.trk_chunk_pix; a.nchunk = p.trk_nchunk;
  a.tilecone = p.cull == VB_CULL_TILECONE; a.cull_tile = p.cull_tile;
  a.mask_visible = p.mask_visible; a.blockage = p.blockage; a.raw = p.phase_corrected ? 0 : 1;
  a.tcx = sky->cx; a.tcy = sky->cy; a.tcz = sky->cz; a.tcosA = sky->cosA; a.tsinA = sky->sinA;
  for (int lev = 0; lev < TK_LEVELS; ++lev) a.node[lev] = b.trk.node[lev];
  a.rmax = b.trk.rmax; a.plan = b.trk.plan;
  a.q0 = b.trk.q0; a.d1 = b.trk.d1; a.d2 = b.trk.d2; a.p1 = b.trk.p1; a.p2 = b.trk.p2; a.t2 = b.trk.t2;
  a.list = b.trk.list; a.count = b.trk.count; a.queue = b.queue + 2;
  a.partial = b.partial; a.n_half = p.n_half; a.nbl = p.nbl; a.steps = p.trk_steps; a.gpp = p.trk_gpp;
  for (int t = 0; t < kSeriesTables; ++t) series_scale(kSeries[t], a.scale[t]);
  for (int set = 0; set < TK_SETS; ++set) series_dest(8 + 4 * set, a.dest[set]);
  VB_CUDA(cudaFuncSetAttribute((const void*)k_track_sum, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TrackSmem)));
  k_track_sum<<<p.trk_grid, TK_THREADS, sizeof(TrackSmem), s>>>(a);
  VB_LAUNCH_CHECK();
  return VB_OK;
}

}  // namespace vb
