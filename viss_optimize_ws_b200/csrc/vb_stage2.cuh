// Records shared by the stage-2 kernels (vb_stage2.cu, vb_track2.cu).
#pragma once
#include <cuda_runtime.h>

#include "vb_internal.h"

namespace vb {

struct GroupRec {         // 96 bytes
  double a, b, c;         // t = a l + b m + c n  (a = ugu, b = vgu, c = ugu fa + vgu fb)
  float vx, vy;           // representative / averaged visibility
  float fa, fb;
  float cp1, cp2;         // horizon cosines of the representative endpoints
  float4 p1, p2;          // (x, y, z, invn) of the representative endpoints
  float chi, clo;         // c split into two floats (double-single phase)
  int key, flags;         // flags: bit0 = skip (key 0 / nothing to add), bit1 = non-finite V,
                          // bits 2.. = segment
};

// A cluster of up to 32 groups of one segment whose (a, b) lie along one
// baseline's track (vb_track2.cu).
struct GroupCluster {
  int first, count, seg, set;   // first entry of the track order, groups (0: none), segment, polynomial (-1: left)
  int base, pad;                // first of its records after those left to k_recon_rec
  double uc[2];                 // centre (a, b)
  float e1[3], e2[3];           // frame in (a, b, c)
};

}  // namespace vb
