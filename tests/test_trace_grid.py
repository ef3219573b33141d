"""The division of a ray queue over a traversal launch (csrc/trace_grid.h), compiled for the host:
lanes stay without a ray only when every ray of the queue has a lane at once, and no queue is
spread over warps that are not launched or do not fit."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include <initializer_list>
#include "trace_grid.h"
int main() {
  long cases = 0, bad = 0;
  for (int sms : {1, 7, 148})
    for (int occ = 1; occ <= 16; ++occ)
      for (int per_sm = 1; per_sm <= 64; ++per_sm)
        for (bool per_thread : {false, true}) {
          const xb::TraceGrid g = xb::trace_grid(sms * per_sm, sms, occ, per_thread);
          const int resident = sms * (per_sm < occ ? per_sm : occ);   // blocks
          bad += g.blocks != (per_thread ? sms * per_sm : resident);
          bad += g.warps > 4 * g.blocks || g.warps > 4 * sms * occ;
          for (int n : {0, 1, 31, 32, 33, 4 * resident - 1, 4 * resident, 4 * resident + 1, 64 * resident + 5,
                        128 * resident - 1, 128 * resident, 128 * resident + 1, 4096 * resident + 3}) {
            const int lanes = xb::queue_lanes(n, g.warps);
            ++cases;
            bad += lanes < 1 || lanes > 32;
            bad += lanes < 32 && (long)lanes * 4 * resident < n;            // idle lanes while rays wait
            bad += lanes > 1 && (long)(lanes - 1) * 4 * resident >= n;      // spread no wider than it could be
          }
        }
  std::printf("%ld %ld\n", cases, bad);
  return 0;
}
"""


def test_no_lane_is_idle_while_rays_wait(tmp_path):
    src = tmp_path / "grid.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "grid"
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "xenon_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    cases, bad = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert cases > 10_000 and bad == 0
