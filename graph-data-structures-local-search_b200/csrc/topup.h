// topup.h -- completing a batch of iterations after its first launches.
#pragma once
#include <cstdint>

namespace tsb {

// The candidate pass hands single iterations to the sweeps, any number of them
// in a long batch: each time the host sees how far the search came, launches
// some sweeps and lets the pass try again.  Only rounds in a row that advance
// nothing mean that the search is stuck.
struct TopUp {
  static constexpr int kStuckRounds = 1 << 20;
  static constexpr int64_t kMaxSweeps = 4096;

  explicit TopUp(int64_t iter) : last(iter) {}
  // A round that begins at iteration `iter`; false: the search is stuck.
  bool advance(int64_t iter) {
    gained = iter - last;
    last = iter;
    stuck = gained > 0 ? 0 : stuck + 1;
    return stuck < kStuckRounds;
  }
  // Sweeps until the next try, after `sweeps` of them the last time: stops in
  // quick succession (ties everywhere) double them.
  int64_t sweeps_after(int64_t sweeps) const {
    if (gained > 4 * sweeps) return 1;
    return 2 * sweeps < kMaxSweeps ? 2 * sweeps : kMaxSweeps;
  }

  int64_t last, gained = 0;
  int stuck = 0;
};

}  // namespace tsb
