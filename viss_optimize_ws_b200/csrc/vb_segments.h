// Steps of each segment that the cluster slots of stage 2 hold (vb_track2.cu).
// Plain C++, so that the CPU tests check it as well.
#pragma once
#include <cstdint>

#include "vb_host_device.h"

namespace vb {

// [t0, t0 + result) is the segment's own range of steps: cut where a later entry
// of the table begins (`next`, the smallest t0 after this entry), empty for a
// range that leaves the day.  A step belongs to the last entry that begins at or
// before it, so nothing of the segment lies past the cut; and the ranges of two
// entries never share a step, whatever the table holds: ranges that overlap, that
// run past the day, or that are out of order.
VB_HOST_DEVICE inline int segment_steps(int t0, int tlen, int64_t next, int64_t steps) {
  if (t0 < 0 || tlen <= 0 || (int64_t)t0 + tlen > steps) return 0;
  const int64_t room = next - t0;
  return room <= 0 ? 0 : (room < tlen ? (int)room : tlen);
}

// First table entry of a segment's tracks: rows for every 32 steps before it and
// one more per segment, which holds a cluster of 32 steps or fewer per row.
VB_HOST_DEVICE inline int64_t segment_entries(int t0, int seg, int64_t ntrk) { return ntrk * ((int64_t)t0 / 32 + seg); }

}  // namespace vb
