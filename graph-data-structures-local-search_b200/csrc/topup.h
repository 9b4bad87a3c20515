// topup.h -- sweeps between two tries of the candidate pass, and the rounds that
// complete a batch of iterations after its first launches.
#pragma once
#include <cstdint>

namespace tsb {

// Sweeps until the next try of the candidate pass, when the last try came after
// `sweeps` of them and `gained` iterations have been made since: stops in
// quick succession (ties everywhere) double them.
constexpr int64_t kMaxSweeps = 4096;
inline int64_t sweeps_after(int64_t sweeps, int64_t gained) {
  if (gained > 4 * sweeps) return 1;
  return 2 * sweeps < kMaxSweeps ? 2 * sweeps : kMaxSweeps;
}

// The candidate pass hands single iterations to the sweeps, any number of them
// in a long batch: each time the host sees how far the search came, launches
// some sweeps and lets the pass try again.  Only rounds in a row that advance
// nothing mean that the search is stuck.
struct TopUp {
  static constexpr int kStuckRounds = 1 << 20;

  explicit TopUp(int64_t iter) : last(iter) {}
  // A round that begins at iteration `iter`; false: the search is stuck.
  bool advance(int64_t iter) {
    gained = iter - last;
    last = iter;
    stuck = gained > 0 ? 0 : stuck + 1;
    return stuck < kStuckRounds;
  }
  int64_t sweeps_after(int64_t sweeps) const { return tsb::sweeps_after(sweeps, gained); }

  int64_t last, gained = 0;
  int stuck = 0;
};

}  // namespace tsb
