// Choosing the fastest of a few launch shapes by timing them.
#pragma once
#include <algorithm>

namespace bpf {

// The fastest of the candidates 0 .. nc - 1 into *best, the median of each
// one's times into med (infinite for one that could not be launched).
// time(k, ms) launches candidate k, puts its time into *ms and returns 0, or
// an error code.
//
// The candidates take turns, round after round, so that a drift of clocks or
// caches during the tuning reaches every one alike; medians decide, among
// those that the first round left within `near` of its best (the others are
// timed once).  A candidate that cannot be launched drops out: a GPU, or a
// part of one, that cannot hold its cluster still has the others.  Only if
// none can be launched does an error come back.
template <int kMax, int kReps, class Time>
int pick_fastest(int nc, float near, Time&& time, float (&med)[kMax], int* best) {
  const float inf = __builtin_inff();
  float t[kMax][kReps], least = inf;
  int have[kMax] = {}, rc = 0;  // times of a candidate; -1: it could not be launched
  bool in[kMax];
  for (int k = 0; k < nc; ++k) in[k] = true;
  for (int r = 0; r < kReps; ++r) {
    for (int k = 0; k < nc; ++k) {
      if (!in[k]) continue;
      const int e = time(k, &t[k][r]);
      if (e) {
        rc = e;
        in[k] = false;
        have[k] = -1;
        continue;
      }
      have[k] = r + 1;
      if (r == 0) least = std::min(least, t[k][0]);
    }
    if (r == 0)
      for (int k = 0; k < nc; ++k) in[k] = in[k] && t[k][0] <= near * least;
  }
  *best = -1;
  for (int slow = 0; slow < 2 && *best < 0; ++slow)  // one that was slow, if no other is left
    for (int k = 0; k < nc; ++k) {
      if (have[k] > 0) std::sort(t[k], t[k] + have[k]);
      med[k] = have[k] > 0 ? t[k][have[k] / 2] : inf;
      if (have[k] > 0 && (in[k] || slow) && (*best < 0 || med[k] < med[*best])) *best = k;
    }
  return *best >= 0 ? 0 : rc;
}

}  // namespace bpf
