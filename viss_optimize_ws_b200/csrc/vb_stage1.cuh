// Device pieces shared by the two stage-1 kernels (vb_stage1.cu: the per-term
// sum; vb_track.cu: the factored sum over track groups).
#pragma once
#include <cuda_runtime.h>

#include "vb_common.cuh"
#include "vb_internal.h"

namespace vb {

constexpr int kTrackGroup = 128;   // steps of one pair in a track group
constexpr int kClsHid = 0, kClsVis = 1, kClsMix = 2;   // class of a (baseline, tile) pair

// F32X phase reduction: magic = 1.5 * 2^29 keeps every partial sum of the FMA
// chain in [2^29, 2^30) (|u| + |v| + |w| < 2^28); the double's ulp is then
// 2^-23 turns, so each FMA rounds to nearest on the 2^-23-turn grid the FP32
// angle is built on, and the low 23 bits of the double are the turn fraction:
// one LOP3 turns them into the exact float 2^23 + k.
constexpr double kMagic = 805306368.0;              // 1.5 * 2^29
constexpr float kTwoPiF = 6.28318530717958647692f;
constexpr float kAngScale = 6.28318530717958647692f * 1.1920928955078125e-7f;  // fl(2pi) * 2^-23
constexpr double kMaxUvwF32X = 67108864.0;         // 2^26: 3 * 2^26 < 2^28

// Per-endpoint threshold of the per-pixel occlusion test: the test
// "fl(d * invn) < cosphi" (d the FP32 dot of pixel and endpoint, rounded as
// occ_dot rounds it) holds exactly when d < t, t being the smallest float with
// fl(t * invn) >= cosphi: fl(d * invn) does not decrease as d grows (invn > 0).
// The masked path then compares d with t instead of multiplying first, with
// the same masks (two multiplies fewer per masked term: 1217.7 -> 1206.1 ms on
// the nside-1024 day, 9.66 -> 9.64 ms at nside 256).
static __device__ __noinline__ float occ_threshold(float invn, float c) {
  if (c != c || invn != invn) return -INFINITY;                  // the test never fails
  if (invn == 0.0f) return c > 0.0f ? INFINITY : -INFINITY;      // fl(d * 0) = 0 against c
  if (isinf(invn)) return 0.0f;                                  // d * inf: fails exactly for d < 0
  float t = c / invn;                                            // within a few ulps; fixed below
  for (int k = 0; k < 16 && !(t * invn >= c); ++k) t = nextafterf(t, INFINITY);
  for (int k = 0; k < 16; ++k) {
    const float p = nextafterf(t, -INFINITY);
    if (p * invn >= c) t = p; else break;
  }
  return t;
}

// --- bulk-copy staging --------------------------------------------------------
// One thread copies a stage's records (a contiguous range of the interleaved
// global array) into this CTA's own shared memory with cp.async.bulk, which
// signals an mbarrier when the bytes have landed; the other buffer is filled
// while the CTA computes on this one.  No cluster multicast: the source is
// always this GPU's own memory and the destination this CTA's shared memory.
// (Measured on one B200 against the cooperative loads it replaced, which
// staged through registers between two barriers per stage: 1231 against 1248
// ms on the nside-1024 day, 9.72 against 9.80 ms at nside 256.)
__device__ __forceinline__ unsigned smem_addr(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void bulk_stage_issue(void* dst, const void* src, unsigned bytes, unsigned long long* bar) {
  // shared memory the threads read before the preceding barrier is written by
  // the async proxy next: order the two proxies
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
// Waits for the phase `parity` of the barrier to complete, at most kBulkWaitTries
// polls; a wait that runs out sets ERR_WAIT_TIMEOUT (the outputs of the call
// are then not to be trusted) and returns.
constexpr int kBulkWaitTries = 1 << 22;
__device__ __forceinline__ void bulk_stage_wait(unsigned long long* bar, unsigned parity, unsigned* err) {
  for (int i = 0; i < kBulkWaitTries; ++i) {
    unsigned done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    if (done) return;
  }
  atomicOr(err, ERR_WAIT_TIMEOUT);
}

}  // namespace vb
