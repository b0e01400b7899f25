// Stage 2, factored over clusters of uv groups: the same image as k_recon_rec
// for the groups whose cells lie along one baseline's track in one segment, with
// one sin / cos per (cluster, pixel) instead of one per (group, pixel).
//
// The cells (a, b) that one pair visits in a segment follow a smooth curve to
// within half a cell.  For a cluster of up to 32 of them around (A, B) and a
// block of 256 pixels around s_c, with l' = l + fa n, m' = m + fb n,
//   sum_g V_g e^{2 pi i (a l' + b m')} = e^{2 pi i (A l' + B m')} P(tau, eta),
//   P = sum_g V_g e^{2 pi i D_g.s_c} e^{i (x_g tau + y_g eta)},
// where (x, y) is the cell's place in the cluster's frame and (tau, eta) the
// pixel's in the block.  e^{i (x tau + y eta)} is a polynomial of 32 terms
// (vb_series.h, any single term within 1.5e-7): a warp forms its coefficients once
// per (cluster, block), a lane per group, and every pixel evaluates it.  The
// phase of a pixel's factor is rounded once to the 2^-23-turn grid, where
// k_recon_rec rounds twice, 3.7e-7 against 7.5e-7, so that a term is no further off
// than there.  Measured with one visibility, largest and rms error of a term: 1.1e-6
// and 2.4e-7, k_recon_rec 1.2e-6 and 2.7e-7.  Clusters
// that no polynomial fits and groups outside clusters stay on k_recon_rec.
//
// Bound: FP32 issue (per cluster and 1024 pixels: 4 x (32 groups' classes, FP64
// rotation, 64 products, transposed reduction) and 32 x (phase, sin/cos, 64
// multiply-adds), against 16 SFU cycles for each 32 terms of k_recon_rec).
//
// Inclusion: groups proven visible or hidden against the block's cone are summed
// or dropped as a whole, the others take the per-pixel test, so that W counts
// the same groups.
#include <algorithm>
#include <cmath>

#include "vb_common.cuh"
#include "vb_geom.cuh"
#include "vb_internal.h"
#include "vb_segments.h"
#include "vb_series.h"
#include "vb_stage1.cuh"
#include "vb_stage2.cuh"
#include "vb_track.cuh"

namespace vb {

constexpr int G2_THREADS = 256;
constexpr int G2_PPT = 4;               // a CTA's 1024 pixels: four 256-pixel blocks, each by two warps, four pixels a lane
constexpr int G2_STAGE = 8;             // clusters per step, one a warp
constexpr int G2_LEVEL = 1;             // TrackNode level of 256 pixels
constexpr int G2_TRACKS = 4096;         // largest pairs (signed pairs) per step
constexpr int G2_MIN = 10;              // groups from which a cluster pays (about 380 / 8 + 70 cycles for each 32 pixels)

// Polynomial shapes: powers of tau for eta^0.. eta^4.
template <int SHAPE>
struct Poly {
  static constexpr int NC = 5;
  __host__ __device__ static constexpr int N(int c) { return cluster_row(SHAPE, c); }
};
constexpr int G2_SHAPES = 2, G2_J = kClusterTerms;
// Shape of each table, a bit each.
constexpr unsigned shape_bits() {
  unsigned m = 0;
  for (int t = 0; t < kClusterTables; ++t) m |= (unsigned)kClusters[t].shape << t;
  return m;
}
constexpr unsigned G2_SHAPE_BITS = shape_bits();

// --- clusters -------------------------------------------------------------------
struct ClusterArgs {
  float2 box[kClusterTables];   // largest |x tau|, |y eta| of each table
  const unsigned long long* skeys;
  const int *svals, *start, *ngroups;
  const vb_seg_params* sp;
  const int *seg_t0, *seg_tlen;
  int ntrk, nseg, n_keyed, entries;
  const unsigned* rmax;
  int* steps;                                // of each segment (segment_steps)
  int *slots, *order, *dst, *list, *count;   // count: clusters, groups left to k_recon_rec
  GroupCluster *table, *clu;                 // by entry; those in use, in a row
  vb_seg_params* spd;
};
constexpr int kClusterWords = sizeof(GroupCluster) / sizeof(int);
static_assert(kClusterWords == 16, "a lane copies one word of a cluster");

// Steps of each segment that its slots hold, one warp from the last segment back:
// slots, track orders and table entries of a segment are laid out by them, so two
// segments must not share a step.
__global__ void __launch_bounds__(32) k_cluster_steps(const ClusterArgs a) {
  const int lane = threadIdx.x;
  const int64_t steps = a.n_keyed / a.ntrk;
  int after = INT32_MAX;   // smallest t0 of the segments past this pass
  for (int top = a.nseg - 1; top >= 0; top -= 32) {
    const int seg = top - lane;
    const int t0 = seg >= 0 ? a.seg_t0[seg] : INT32_MAX;
    int low = t0;          // smallest t0 from this segment on
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, low, o);
      if (lane >= o) low = min(low, v);
    }
    const int prev = __shfl_up_sync(0xffffffffu, low, 1);
    if (seg >= 0) a.steps[seg] = segment_steps(t0, a.seg_tlen[seg], lane ? min(after, prev) : after, steps);
    after = min(after, __shfl_sync(0xffffffffu, low, 31));
  }
}

// Each group's place on its representative's track: slots[segment][track][step].
__global__ void k_cluster_mark(const ClusterArgs a) {
  const int ng = *a.ngroups;
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < ng; g += gridDim.x * blockDim.x) {
    a.dst[g] = 0;
    const int s0 = a.start[g], L = a.start[g + 1] - s0;
    const unsigned long long ck = a.skeys[s0];
    if ((unsigned)ck == 0u) continue;   // off the grid
    const int seg = (int)(ck >> 32), rep = a.svals[s0 + (L >> 1)];
    const int step = rep / a.ntrk, track = rep - step * a.ntrk;
    const int t0 = a.seg_t0[seg], tl = a.steps[seg];
    if (step < t0 || step >= t0 + tl) continue;
    a.slots[(int64_t)a.ntrk * t0 + (int64_t)track * tl + (step - t0)] = g;
  }
}

// One CTA per segment: each track's groups in step order, cut into clusters of
// at most 32 of nearly equal size.
__global__ void __launch_bounds__(1024) k_cluster_cut(const ClusterArgs a) {
  __shared__ int s_m[G2_TRACKS], s_pre[G2_TRACKS];
  const int seg = blockIdx.x, lane = threadIdx.x & 31;
  const int t0 = a.seg_t0[seg], tl = a.steps[seg];
  const int64_t base = (int64_t)a.ntrk * t0;
  for (int t = threadIdx.x >> 5; t < a.ntrk; t += 32) {
    const int64_t row = base + (int64_t)t * tl;
    int m = 0;
    for (int k = 0; k < tl; k += 32) {
      const int g = k + lane < tl ? a.slots[row + k + lane] : -1;
      const unsigned has = __ballot_sync(0xffffffffu, g >= 0);
      if (g >= 0) a.order[row + m + __popc(has & ((1u << lane) - 1u))] = g;
      m += __popc(has);
    }
    if (lane == 0) s_m[t] = m;
  }
  __syncthreads();
  if (threadIdx.x < 32) {
    int run = 0;
    for (int t = 0; t < a.ntrk; t += 32) {
      const int m = t + lane < a.ntrk ? s_m[t + lane] : 0;
      const int k = m >= G2_MIN ? (m + 31) / 32 : 0;
      int inc = k;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += v;
      }
      if (t + lane < a.ntrk) s_pre[t + lane] = run + inc - k;
      run += __shfl_sync(0xffffffffu, inc, 31);
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < a.ntrk; t += 1024) {
    const int m = s_m[t];
    if (m < G2_MIN) continue;
    const int k = (m + 31) / 32, size = (m + k - 1) / k;
    for (int c = 0; c < k; ++c) {
      const int64_t e = segment_entries(t0, seg, a.ntrk) + s_pre[t] + c;
      if (e >= a.entries) break;
      GroupCluster& q = a.table[2 * e];
      q.first = (int)(base + (int64_t)t * tl) + c * size;
      q.count = max(0, min(size, m - c * size));
      q.seg = seg;
    }
  }
}

// Frame and polynomial of each cluster, one warp each; one that no polynomial
// fits is tried as two halves (entries 2 e and 2 e + 1 of the table).
__global__ void __launch_bounds__(128) k_cluster_plan(const ClusterArgs a) {
  const int lane = threadIdx.x & 31;
  const int e = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (e >= a.entries) return;
  const GroupCluster whole = a.table[2 * e];
  if (whole.count < G2_MIN / 2) {
    if (lane < 2) a.table[2 * e + lane].set = -1;
    return;
  }
  const vb_seg_params sp = a.sp[whole.seg];
  const bool there = lane < whole.count;
  const int g = a.order[whole.first + (there ? lane : 0)];
  const unsigned long long ck = a.skeys[a.start[g]];
  const bool own = __all_sync(0xffffffffu, (int)(ck >> 32) == whole.seg) && isfinite(sp.fa) && isfinite(sp.fb);
  const int key = (int)(unsigned)(ck & 0xffffffffull) - 1;
  const int U = key / sp.RES;
  const float ua = (U - sp.half) * sp.du, ub = (key - U * sp.RES - sp.half) * sp.du;   // as k_group_records
  const double pt[3] = {(double)ua, (double)ub, (double)ua * (double)sp.fa + (double)ub * (double)sp.fb};
  const float kr = 6.2831855f * __uint_as_float(a.rmax[G2_LEVEL]);
  auto fit = [&](int l0, int l1, GroupCluster& q) {   // groups [l0, l1) of the whole
    const bool on = lane >= l0 && lane < l1;
    double f0[3], d[3], e1[3] = {1.0, 0.0, (double)sp.fa}, e2[3];
    for (int c = 0; c < 3; ++c) {
      f0[c] = __shfl_sync(0xffffffffu, pt[c], l0);
      d[c] = __shfl_sync(0xffffffffu, pt[c], l1 - 1) - f0[c];
    }
    if (d[0] * d[0] + d[1] * d[1] > 1e-12)
      for (int c = 0; c < 3; ++c) e1[c] = d[c];
    double inv = rsqrt(e1[0] * e1[0] + e1[1] * e1[1] + e1[2] * e1[2]);
    for (int c = 0; c < 3; ++c) e1[c] *= inv;
    // e2: across e1 in the plane c = a fa + b fb (normal (-fa, -fb, 1))
    const double nx = -(double)sp.fa, ny = -(double)sp.fb;
    e2[0] = ny * e1[2] - e1[1];
    e2[1] = e1[0] - nx * e1[2];
    e2[2] = nx * e1[1] - ny * e1[0];
    inv = rsqrt(e2[0] * e2[0] + e2[1] * e2[1] + e2[2] * e2[2]);
    for (int c = 0; c < 3; ++c) e2[c] *= inv;
    const float x = (float)((pt[0] - f0[0]) * e1[0] + (pt[1] - f0[1]) * e1[1] + (pt[2] - f0[2]) * e1[2]);
    const float y = (float)((pt[0] - f0[0]) * e2[0] + (pt[1] - f0[1]) * e2[1] + (pt[2] - f0[2]) * e2[2]);
    const float xh = warp_max(on ? x : -INFINITY), xl = -warp_max(on ? -x : -INFINITY);
    const float yh = warp_max(on ? y : -INFINITY), yl = -warp_max(on ? -y : -INFINITY);
    const float X1 = kr * 0.5f * (xh - xl), X2 = kr * 0.5f * (yh - yl);
    q.first = whole.first + l0;
    q.count = l1 - l0;
    q.seg = whole.seg;
    q.set = -1;
    if (!own || l1 - l0 < G2_MIN / 2) return false;
    for (int t = kClusterTables - 1; t >= 0; --t)
      if (X1 <= a.box[t].x && X2 <= a.box[t].y) q.set = t;
    if (q.set < 0) return false;
    const double mx = 0.5 * ((double)xh + xl), my = 0.5 * ((double)yh + yl);
    q.uc[0] = f0[0] + mx * e1[0] + my * e2[0];
    q.uc[1] = f0[1] + mx * e1[1] + my * e2[1];
    for (int c = 0; c < 3; ++c) { q.e1[c] = (float)e1[c]; q.e2[c] = (float)e2[c]; }
    if (on) a.dst[g] = -1;
    return true;
  };
  GroupCluster q0 = whole, q1 = whole;
  q1.set = -1;
  if (!fit(0, whole.count, q0) && whole.count >= 2 * G2_MIN) {
    const int h = (whole.count + 1) / 2;
    fit(0, h, q0);
    fit(h, whole.count, q1);
  }
  if (lane == 0) { a.table[2 * e] = q0; a.table[2 * e + 1] = q1; }
}

// One CTA: list of the clusters in use with the places of their records, and
// places of the groups left to k_recon_rec, which come first.
__global__ void __launch_bounds__(1024) k_cluster_scan(const ClusterArgs a) {
  __shared__ unsigned long long s_w[32];
  __shared__ unsigned long long s_base;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto scan = [&](unsigned long long v) {   // exclusive, running over the CTA's passes
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
    __syncthreads();
    if (threadIdx.x == 1023) s_base = before + inc;
    __syncthreads();
    return before + inc - v;
  };
  if (threadIdx.x == 0) s_base = 0ull;
  __syncthreads();
  for (int e0 = 0; e0 < 2 * a.entries; e0 += 1024) {
    const int e = e0 + threadIdx.x;
    const bool ok = e < 2 * a.entries && a.table[e].set >= 0;
    const unsigned long long ex = scan(ok ? (1ull << 32) | (unsigned)a.table[e].count : 0ull);
    if (ok) {
      a.list[(int)(ex >> 32)] = e;
      a.table[e].base = (int)(ex & 0xffffffffull);
    }
  }
  int nc = (int)(s_base >> 32);
  const int ng = *a.ngroups;
  // Fewer than a quarter of the groups: what they save does not pay for the second
  // kernel's tail (30 m, Earth orbits, nside 256 and 512: 1 to 3 % slower with them).
  if (4 * (s_base & 0xffffffffull) < (unsigned long long)ng) {
    nc = 0;
    for (int e = threadIdx.x; e < 2 * a.entries; e += 1024) a.table[e].set = -1;
    for (int g = threadIdx.x; g < ng; g += 1024) a.dst[g] = 0;
  }
  __syncthreads();
  if (threadIdx.x == 0) s_base = 0ull;
  __syncthreads();
  for (int g0 = 0; g0 < ng; g0 += 1024) {
    const int g = g0 + threadIdx.x;
    const bool left = g < ng && a.dst[g] >= 0;
    const int ex = (int)scan(left ? 1ull : 0ull);
    if (g < ng) {
      a.slots[g] = ex;   // (the slots are read)
      if (left) a.dst[g] = ex;
    }
  }
  const int nd = (int)s_base;
  __syncthreads();
  if (threadIdx.x == 0) {
    a.count[0] = nc;
    a.count[1] = nd;
  }
  // groups left in each segment: a range of the records of its own
  for (int s = threadIdx.x; s < a.nseg; s += 1024) {
    vb_seg_params q = a.sp[s];
    if (q.nuniq > 0) {
      const int g1 = q.group_start + q.nuniq;
      const int e0 = a.slots[q.group_start], e1 = g1 < ng ? a.slots[g1] : nd;
      q.group_start = e0;
      q.nuniq = e1 - e0;
    }
    a.spd[s] = q;
  }
}

__global__ void k_cluster_assign(const ClusterArgs a) {
  const int lane = threadIdx.x & 31;
  const int nc = a.count[0], nd = a.count[1];
  for (int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < nc; i += (gridDim.x * blockDim.x) >> 5) {
    const GroupCluster& q = a.table[a.list[i]];
    if (lane < q.count) a.dst[a.order[q.first + lane]] = nd + q.base + lane;
    if (lane < kClusterWords) reinterpret_cast<int*>(a.clu + i)[lane] = reinterpret_cast<const int*>(&q)[lane];
  }
}

// --- reconstruction ---------------------------------------------------------------
struct TrackReconArgs {
  const float *l, *m, *n;
  int64_t npix;
  int nblocks, rows, blockage;
  const TrackNode* node;
  const unsigned* rmax;
  const GroupCluster* clu;
  const int* count;
  const vb_seg_params* sp;
  const GroupRec* rec;
  const int* nrec;     // all groups
  int* queue;
  double* Cpart;       // [rows][npix]
  unsigned* Wpart;
  float scale[kClusterTables][2 * G2_J];
  unsigned char dest[G2_SHAPES][2 * G2_J];
};

// Coefficients of one (cluster, block): lane = group, value w = V e^{2 pi i D.s_c}
// (zero for the lanes that do not take part).
template <int SHAPE>
__device__ __forceinline__ void cluster_moments(float wr, float wi, float x, float y, const float* scale, const unsigned char* dest,
                                                float* mom, int lane) {
  using P = Poly<SHAPE>;
  float v[2 * G2_J];
  int o = 0;
#pragma unroll
  for (int c = 0; c < P::NC; ++c) {
    float pr = wr, pi = wi;
#pragma unroll
    for (int i = 0; i < P::N(c); ++i) {
      v[o] = pr;
      v[o + 1] = pi;
      pr *= x;
      pi *= x;
      o += 2;
    }
    wr *= y;
    wi *= y;
  }
  fold_half<64, 16>(v, lane & 16);
  fold_half<32, 8>(v, lane & 8);
  fold_half<16, 4>(v, lane & 4);
  fold_half<8, 2>(v, lane & 2);
  fold_half<4, 1>(v, lane & 1);
  const int base = ((lane & 16) ? 32 : 0) + ((lane & 8) ? 16 : 0) + ((lane & 4) ? 8 : 0) + ((lane & 2) ? 4 : 0) + ((lane & 1) ? 2 : 0);
#pragma unroll
  for (int k = 0; k < 2; ++k) mom[dest[base + k]] = v[k] * scale[base + k];
}

// The polynomial at a thread's four pixels (of one block: each coefficient is
// loaded once for the four, whose chains are independent).
template <int SHAPE>
__device__ __forceinline__ void cluster_eval(const float* mom, const float (&tau)[G2_PPT], const float (&eta)[G2_PPT],
                                             float2 (&out)[G2_PPT]) {
  using P = Poly<SHAPE>;
  const f2* m = reinterpret_cast<const f2*>(mom);
  f2 t2[G2_PPT], r[G2_PPT];
#pragma unroll
  for (int j = 0; j < G2_PPT; ++j) { t2[j] = f2_make(tau[j], tau[j]); r[j] = 0ull; }
  int o = G2_J;
#pragma unroll
  for (int c = P::NC - 1; c >= 0; --c) {
    o -= P::N(c);
    f2 h[G2_PPT];
    const f2 top = m[o + P::N(c) - 1];
#pragma unroll
    for (int j = 0; j < G2_PPT; ++j) h[j] = top;
#pragma unroll
    for (int i = P::N(c) - 2; i >= 0; --i) {
      const f2 k = m[o + i];
#pragma unroll
      for (int j = 0; j < G2_PPT; ++j) h[j] = f2_fma(h[j], t2[j], k);
    }
#pragma unroll
    for (int j = 0; j < G2_PPT; ++j) r[j] = c == P::NC - 1 ? h[j] : f2_fma(r[j], f2_make(eta[j], eta[j]), h[j]);
  }
#pragma unroll
  for (int j = 0; j < G2_PPT; ++j) out[j] = f2_split(r[j]);
}

struct ClusterStage {
  double A, B;
  float e1[3], e2[3];
  int rec0, set;
};

__global__ void __launch_bounds__(G2_THREADS, 2) k_recon_track(const __grid_constant__ TrackReconArgs a) {
  __shared__ __align__(16) float s_mom[G2_STAGE][G2_PPT][2 * G2_J];
  __shared__ int s_vis[G2_STAGE][G2_PPT];
  __shared__ unsigned s_mix[G2_STAGE][G2_PPT];
  __shared__ ClusterStage s_cl[G2_STAGE];
  __shared__ __align__(16) int s_clu[2][G2_STAGE][kClusterWords];   // this step's clusters and the next's
  __shared__ TrackNode s_node[G2_PPT];
  __shared__ float s_scale[kClusterTables][2 * G2_J];
  __shared__ unsigned char s_dest[G2_SHAPES][2 * G2_J];
  __shared__ int s_item;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  asm volatile("griddepcontrol.launch_dependents;");   // k_recon_rec may take SMs that this one leaves
  const int nc = a.count[0], nd = a.count[1];
  if (nc == 0) return;
  for (int i = threadIdx.x; i < kClusterTables * 2 * G2_J; i += G2_THREADS) (&s_scale[0][0])[i] = (&a.scale[0][0])[i];
  for (int i = threadIdx.x; i < G2_SHAPES * 2 * G2_J; i += G2_THREADS) (&s_dest[0][0])[i] = (&a.dest[0][0])[i];
  const float r = __uint_as_float(a.rmax[G2_LEVEL]), inv_r = 1.f / r, kr = 6.28318530717958647692f * r;
  const int per_row = (nc + a.rows - 1) / a.rows;
  const int n_items = a.rows * a.nblocks;
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = atomicAdd(a.queue, 1);
    __syncthreads();
    const int item = s_item;
    if (item >= n_items) break;
    const int row = item / a.nblocks, blk = item - row * a.nblocks;
    const int64_t pix0 = (int64_t)blk * (G2_THREADS * G2_PPT);
    const int wq = warp >> 1;                                  // this warp's 256-pixel block
    const int own = wq * 256 + (warp & 1) * 32 + lane;         // its first pixel, the others 64 apart
    float lf[G2_PPT], mf[G2_PPT], nf[G2_PPT];
    double totC[G2_PPT];
    unsigned totW[G2_PPT];
#pragma unroll
    for (int q = 0; q < G2_PPT; ++q) {
      const int64_t p = min(pix0 + own + q * 64, a.npix - 1);
      lf[q] = a.l[p]; mf[q] = a.m[p]; nf[q] = a.n[p];
      totC[q] = 0.0;
      totW[q] = 0u;
    }
    if (threadIdx.x < G2_PPT * 8) {
      const int64_t nidx = (int64_t)blk * G2_PPT + (threadIdx.x >> 3);
      if (nidx * tk_block(G2_LEVEL) < a.npix)
        reinterpret_cast<float*>(&s_node[threadIdx.x >> 3])[threadIdx.x & 7] = reinterpret_cast<const float*>(a.node + nidx)[threadIdx.x & 7];
    }
    const int c_end = min(nc, (row + 1) * per_row);
    int cs = row * per_row, buf = 0;
    if (lane < kClusterWords && cs + warp < c_end)
      s_clu[0][warp][lane] = reinterpret_cast<const int*>(a.clu + cs + warp)[lane];
    while (cs < c_end) {
      __syncthreads();   // the previous step's coefficients are read, this step's clusters are here
      // this step: up to 8 clusters of one segment
      const GroupCluster* step = reinterpret_cast<const GroupCluster*>(&s_clu[buf][0][0]);
      const int seg = step[0].seg;
      const float fa = a.sp[seg].fa, fb = a.sp[seg].fb;
      int nk = 1;
      while (nk < G2_STAGE && cs + nk < c_end && step[nk].seg == seg) ++nk;
      // the next step's clusters into the other buffer, and its records into L1
      // (they follow this step's), while this step computes
      const int next = cs + nk;
      int word = 0;
      if (lane < kClusterWords && next + warp < c_end) word = reinterpret_cast<const int*>(a.clu + next + warp)[lane];
      if (next < c_end) {
        const int rnext = nd + step[nk - 1].base + step[nk - 1].count + (int)threadIdx.x;
        if (rnext < a.nrec[0]) asm volatile("prefetch.global.L1 [%0];" ::"l"(a.rec + rnext));
      }
      if (warp < nk) {
        const GroupCluster& cl = step[warp];
        const double A = cl.uc[0], B = cl.uc[1], Cc = A * (double)fa + B * (double)fb;
        const int set = cl.set, rec0 = nd + cl.base;
        if (lane == 0) {
          ClusterStage& st = s_cl[warp];
          st.A = A; st.B = B; st.rec0 = rec0; st.set = set;
          for (int c = 0; c < 3; ++c) { st.e1[c] = cl.e1[c] * inv_r; st.e2[c] = cl.e2[c] * inv_r; }
        }
        const bool on = lane < cl.count;
        const GroupRec* g = a.rec + rec0 + (on ? lane : 0);
        const double da = g->a - A, db = g->b - B, dc = g->c - Cc;
        const float vx = g->vx, vy = g->vy;
        const float fx = (float)da, fy = (float)db, fz = (float)dc;
        const float x = kr * fmaf(fx, cl.e1[0], fmaf(fy, cl.e1[1], fz * cl.e1[2]));
        const float y = kr * fmaf(fx, cl.e2[0], fmaf(fy, cl.e2[1], fz * cl.e2[2]));
        const bool out = !on || (g->flags & 3);
        // a visibility that is not finite spreads to its own terms only: term by term
        const bool finite = fabsf(vx) < 1e30f && fabsf(vy) < 1e30f;
        float4 d1, d2;
        float s1 = 0.f, s2 = 0.f;
        if (a.blockage) {
          const float4 p1 = g->p1, p2 = g->p2;
          d1 = make_float4(p1.x * p1.w, p1.y * p1.w, p1.z * p1.w, g->cp1);
          d2 = make_float4(p2.x * p2.w, p2.y * p2.w, p2.z * p2.w, g->cp2);
          s1 = horizon_sine(d1);
          s2 = horizon_sine(d2);
        }
#pragma unroll 1
        for (int q = 0; q < G2_PPT; ++q) {
          const int64_t nidx = (int64_t)blk * G2_PPT + q;
          const bool there = nidx * tk_block(G2_LEVEL) < a.npix;
          int c = kClsHid;
          const TrackNode nd_ = s_node[q];
          if (there) {
            if (!out) {
              c = a.blockage ? both_classes(endpoint_class(nd_, d1, s1), endpoint_class(nd_, d2, s2)) : kClsVis;
              if (c == kClsVis && !finite) c = kClsMix;
            }
          }
          const unsigned vis = __ballot_sync(0xffffffffu, c == kClsVis), mix = __ballot_sync(0xffffffffu, c == kClsMix);
          if (lane == 0) { s_vis[warp][q] = __popc(vis); s_mix[warp][q] = mix; }
          if (!vis) continue;
          float wr = 0.f, wi = 0.f;
          if (c == kClsVis) {
            double es, ec;
            turn_cs(fma(da, (double)nd_.cen.x, fma(db, (double)nd_.cen.y, dc * (double)nd_.cen.z)), es, ec);
            wr = (float)fma((double)vx, ec, -(double)vy * es);
            wi = (float)fma((double)vx, es, (double)vy * ec);
          }
          const float xx = c == kClsVis ? x : 0.f, yy = c == kClsVis ? y : 0.f;
          if (!(G2_SHAPE_BITS >> set & 1)) cluster_moments<0>(wr, wi, xx, yy, s_scale[set], s_dest[0], s_mom[warp][q], lane);
          else cluster_moments<1>(wr, wi, xx, yy, s_scale[set], s_dest[1], s_mom[warp][q], lane);
        }
      }
      if (lane < kClusterWords) s_clu[buf ^ 1][warp][lane] = word;
      __syncthreads();
      if (pix0 + wq * 256 < a.npix) {
        const float4 cen = s_node[wq].cen;
        float acc[G2_PPT];
        double lp[G2_PPT], mp[G2_PPT];
#pragma unroll
        for (int q = 0; q < G2_PPT; ++q) {
          acc[q] = 0.f;
          lp[q] = fma((double)fa, (double)nf[q], (double)lf[q]);
          mp[q] = fma((double)fb, (double)nf[q], (double)mf[q]);
        }
        auto angle = [&](double t, bool odd, float& s, float& c) {
          const unsigned kb = ((unsigned)__double2loint(t) & 0x7FFFFFu) ^ (odd ? 0x4B400000u : 0x4B000000u);
          __sincosf(__fmaf_rn(__uint_as_float(kb), kAngScale, -kTwoPiF), &s, &c);
        };
#pragma unroll 1
        for (int k = 0; k < nk; ++k) {
          const ClusterStage& st = s_cl[k];
          const int nv = s_vis[k][wq];
          if (nv) {
            float tau[G2_PPT], eta[G2_PPT];
            float2 h[G2_PPT];
#pragma unroll
            for (int q = 0; q < G2_PPT; ++q) {
              const float dx = lf[q] - cen.x, dy = mf[q] - cen.y, dz = nf[q] - cen.z;
              tau[q] = fmaf(dx, st.e1[0], fmaf(dy, st.e1[1], dz * st.e1[2]));
              eta[q] = fmaf(dx, st.e2[0], fmaf(dy, st.e2[1], dz * st.e2[2]));
            }
            if (!(G2_SHAPE_BITS >> st.set & 1)) cluster_eval<0>(s_mom[k][wq], tau, eta, h);
            else cluster_eval<1>(s_mom[k][wq], tau, eta, h);
#pragma unroll
            for (int q = 0; q < G2_PPT; ++q) {
              // odd clusters half a turn on with the opposite sign (the SFU's mean error cancels)
              float s, c;
              angle(fma(st.A, lp[q], st.B * mp[q]) + kMagic, k & 1, s, c);   // one rounding to the grid
              const float v = fmaf(h[q].x, c, -h[q].y * s);
              acc[q] += (k & 1) ? -v : v;
              totW[q] += (unsigned)nv;
            }
          }
          unsigned mm = s_mix[k][wq];
          while (mm) {
            const int src = __ffs(mm) - 1;
            mm &= mm - 1;
            const GroupRec* g = a.rec + st.rec0 + src;
            const double ga = g->a, gb = g->b;
            const float vx = g->vx, vy = g->vy, cp1 = g->cp1, cp2 = g->cp2;
            const float4 p1 = g->p1, p2 = g->p2;
#pragma unroll
            for (int q = 0; q < G2_PPT; ++q) {
              const bool in = !a.blockage || (occ_dot(lf[q], mf[q], nf[q], p1.x, p1.y, p1.z, p1.w) >= cp1 &&
                                              occ_dot(lf[q], mf[q], nf[q], p2.x, p2.y, p2.z, p2.w) >= cp2);
              float s, c;
              angle(fma(ga, lp[q], fma(gb, mp[q], kMagic)), src & 1, s, c);   // a term of its own, as in k_recon_rec
              const float vv = fmaf(vx, c, -vy * s);
              if (in) {
                acc[q] += (src & 1) ? -vv : vv;
                totW[q] += 1u;
              }
            }
          }
        }
#pragma unroll
        for (int q = 0; q < G2_PPT; ++q) totC[q] += (double)acc[q];
      }
      cs = next;
      buf ^= 1;
    }
#pragma unroll
    for (int q = 0; q < G2_PPT; ++q) {
      const int64_t p = pix0 + own + q * 64;
      if (p < a.npix) {
        a.Cpart[(int64_t)row * a.npix + p] = totC[q];
        a.Wpart[(int64_t)row * a.npix + p] = a.blockage ? totW[q] : 0u;
      }
    }
  }
}

// Coefficient and sign of each part of a moment, i^(k + c) / (k! c!) times the
// table's correction, and where multiplication by that power of i puts it.
static void poly_scale(const ClusterTable& t, float* scale) {
  double col = 1.0;
  for (int c = 0, o = 0; c < 5; ++c) {
    if (c) col /= c;
    double row = 1.0;
    for (int k = 0; k < cluster_row(t.shape, c); ++k, ++o) {
      if (k) row /= k;
      const double f = t.coef[o] * col * row;
      const int d = (k + c) & 3;
      scale[2 * o] = (float)((d == 0 || d == 1) ? f : -f);
      scale[2 * o + 1] = (float)((d == 0 || d == 3) ? f : -f);
    }
  }
}

static void poly_dest(int shape, unsigned char* dest) {
  for (int c = 0, o = 0; c < 5; ++c)
    for (int k = 0; k < cluster_row(shape, c); ++k, ++o) {
      const int d = (k + c) & 1;
      dest[2 * o] = (unsigned char)(2 * o + d);
      dest[2 * o + 1] = (unsigned char)(2 * o + 1 - d);
    }
}

// Clusters are in use for the FP32 sum with FP64 phase over representatives or
// averages where the call is large enough for the planning launches and a second
// kernel's tail (3e10 (baseline, pixel) pairs, 2 ms of k_recon_rec; 8 pairs of
// satellites, nside 256, one B200, without / with clusters: 400 steps, 9e9: 0.64 / 0.74 ms;
// 1000 steps, 2e10: 1.32 / 1.35; 2000, 4e10: 2.48 / 2.30; nside 512, 400, 4e10: 1.87 /
// 1.39) and where a track can fill one (64 steps a segment on average).
void cluster_plan(Stage2Plan* p, int nbl) {
  p->trk = 0;
  const bool members = p->blockage && p->occ_mode != 2;
  if (p->precision != VB_PREC_FP32_FP64PH || members || nbl <= 0 || p->n_half_total % nbl != 0) return;
  const int64_t steps = p->n_half_total / nbl;
  const int64_t ntrk = p->mirror ? nbl : 2 * (int64_t)nbl;
  if (ntrk > G2_TRACKS || steps < 64LL * p->nseg || (double)p->n_keyed_total * (double)p->npix < 3e10) return;
  const int64_t entries = ntrk * (steps / 32 + p->nseg);
  if (entries > INT32_MAX / 64) return;
  p->trk_ntrk = (int)ntrk;
  p->trk_entries = (int)entries;
  p->trk_blocks = (int)ceil_div(p->npix, G2_THREADS * G2_PPT);
  p->trk_rows = (int)std::min<int64_t>(32, std::max<int64_t>(1, ceil_div((int64_t)sm_count() * 2 * 12, p->trk_blocks)));
  p->trk = 1;
}

void cluster_carve(const Stage2Plan& p, Carve& c, ClusterBuffers& x) {
  if (!p.trk) return;
  const size_t n = (size_t)p.n_keyed_total;
  x.count = c.take<int>(4);
  x.steps = c.take<int>(p.nseg);
  x.slots = c.take<int>(n);
  x.order = c.take<int>(n);
  x.dst = c.take<int>(n);
  x.list = c.take<int>(2 * (size_t)p.trk_entries);
  x.table = c.take<GroupCluster>(2 * (size_t)p.trk_entries);
  x.clu = c.take<GroupCluster>(2 * (size_t)p.trk_entries);
  x.spd = c.take<vb_seg_params>(p.nseg);
  x.rmax = c.take<unsigned>(TK_LEVELS);
  for (int lev = 0; lev < TK_LEVELS; ++lev) x.node[lev] = c.take<TrackNode>((size_t)ceil_div(p.npix, tk_block(lev)));
}

int cluster_group(const Stage2Plan& p, const ClusterBuffers& x, const unsigned long long* skeys,
                  const int* svals, const int* start, const int* ngroups, const vb_seg_params* sp, const int* seg_t0,
                  const int* seg_tlen, cudaStream_t s) {
  ClusterArgs a{};
  a.skeys = skeys; a.svals = svals; a.start = start; a.ngroups = ngroups; a.sp = sp;
  a.seg_t0 = seg_t0; a.seg_tlen = seg_tlen;
  a.n_keyed = p.n_keyed_total; a.ntrk = p.trk_ntrk; a.nseg = p.nseg; a.entries = p.trk_entries;
  a.rmax = x.rmax; a.steps = x.steps; a.slots = x.slots; a.order = x.order; a.dst = x.dst; a.list = x.list; a.count = x.count; a.table = x.table; a.clu = x.clu;
  a.spd = x.spd;
  for (int t = 0; t < kClusterTables; ++t) a.box[t] = make_float2(kClusters[t].x1, kClusters[t].x2);
  VB_CUDA(cudaMemsetAsync(x.slots, 0xff, (size_t)p.n_keyed_total * sizeof(int), s));
  VB_CUDA(cudaMemsetAsync(x.table, 0, 2 * (size_t)p.trk_entries * sizeof(GroupCluster), s));
  const int g = (int)std::min<int64_t>(ceil_div(p.n_keyed_total, 256), (int64_t)sm_count() * 16);
  k_cluster_steps<<<1, 32, 0, s>>>(a);
  VB_LAUNCH_CHECK();
  k_cluster_mark<<<g, 256, 0, s>>>(a);
  VB_LAUNCH_CHECK();
  k_cluster_cut<<<p.nseg, 1024, 0, s>>>(a);
  VB_LAUNCH_CHECK();
  k_cluster_plan<<<(int)ceil_div(p.trk_entries, 4), 128, 0, s>>>(a);
  VB_LAUNCH_CHECK();
  k_cluster_scan<<<1, 1024, 0, s>>>(a);
  VB_LAUNCH_CHECK();
  k_cluster_assign<<<std::min(sm_count() * 4, (int)ceil_div(p.trk_entries, 8)), 256, 0, s>>>(a);
  VB_LAUNCH_CHECK();
  return VB_OK;
}

int cluster_sum(const vb_sky* sky, const Stage2Plan& p, const ClusterBuffers& x, const vb_seg_params* sp, const GroupRec* rec,
                const int* ngroups, int* queue, double* Cpart, unsigned* Wpart, cudaStream_t s) {
  TrackReconArgs a{};
  a.l = sky->l; a.m = sky->m; a.n = sky->n; a.npix = p.npix;
  a.nblocks = p.trk_blocks; a.rows = p.trk_rows; a.blockage = p.blockage;
  a.node = x.node[G2_LEVEL]; a.rmax = x.rmax; a.clu = x.clu; a.count = x.count; a.sp = sp; a.rec = rec;
  a.nrec = ngroups;
  a.queue = queue; a.Cpart = Cpart; a.Wpart = Wpart;
  for (int t = 0; t < kClusterTables; ++t) poly_scale(kClusters[t], a.scale[t]);
  for (int shape = 0; shape < G2_SHAPES; ++shape) poly_dest(shape, a.dest[shape]);
  const int grid = (int)std::min<int64_t>((int64_t)sm_count() * 2, (int64_t)p.trk_rows * p.trk_blocks);
  k_recon_track<<<grid, G2_THREADS, 0, s>>>(a);
  VB_LAUNCH_CHECK();
  return VB_OK;
}

}  // namespace vb
