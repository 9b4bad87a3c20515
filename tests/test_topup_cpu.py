"""Completing a long batch whose iterations the candidate pass keeps handing to
the sweeps: any number of rounds that advance, an end to rounds that do not."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "graph-data-structures-local-search_b200", "csrc")

PROGRAM = r"""
#include "topup.h"
#include <cstdio>
using tsb::TopUp;
int main() {
  // a search that hands over after every five iterations of the pass: one
  // sweep each time, for as many rounds as it takes
  TopUp t(0);
  int64_t sweeps = 1;
  for (int64_t iter = 6, round = 0; round < 5000000; round++, iter += sweeps + 5) {
    if (!t.advance(iter)) return printf("stopped after %lld rounds\n", (long long)round), 1;
    sweeps = t.sweeps_after(sweeps);
    if (sweeps != 1) return printf("%lld sweeps\n", (long long)sweeps), 2;
  }
  // hand-overs at every iteration: sweeps double up to the limit
  TopUp d(0);
  sweeps = 1;
  int64_t iter = 0;
  for (int k = 0; k < 30; k++, iter += sweeps) {
    if (!d.advance(iter)) return 3;
    sweeps = d.sweeps_after(sweeps);
    const int64_t want = k < 12 ? int64_t(2) << k : tsb::kMaxSweeps;
    if (sweeps != (want < tsb::kMaxSweeps ? want : tsb::kMaxSweeps)) return 4;
  }
  // nothing advances: an end, and one iteration starts the count again
  TopUp s(7);
  for (int k = 0; k < TopUp::kStuckRounds - 1; k++)
    if (!s.advance(7)) return 5;
  if (!s.advance(8)) return 6;
  for (int k = 0; k < TopUp::kStuckRounds - 1; k++)
    if (!s.advance(8)) return 7;
  return s.advance(8) ? 8 : 0;
}
"""


def test_rounds_that_advance_never_run_out(tmp_path):
    src = tmp_path / "topup.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "topup"
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout)
