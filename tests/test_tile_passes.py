"""The packed kernel names a pass with eight bits, so no class may take a query in more than 256 passes: the host
planner's rules (st_tuning.h, compiled here with the library's class shapes) over every query length."""
import os
import shutil
import subprocess

import pytest

from sabertooth_b200 import tile_classes

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r"""
#include <cstdio>
#include "st_tuning.h"
static const int kShapes[][3] = {%s};
constexpr int kN = sizeof(kShapes) / sizeof(kShapes[0]);
int st_tuning_num_classes() { return kN; }
bool st_tuning_class_team(int c) { return c == kN - 1; }
int st_tuning_class_warps(int c) { return kShapes[c][1] >= 28 ? 4 : 8; }
void st_tuning_class_shape(int c, int* G, int* R, int* C) { *G = kShapes[c][0]; *R = kShapes[c][1]; *C = kShapes[c][2]; }

static bool passes_ok(int c, unsigned m) {
  const unsigned rows = kShapes[c][0] * kShapes[c][1];
  return (m + rows - 1) / rows <= 256;
}

int main() {
  int bad = 0, forced = 0;
  const uint32_t len = 300;
  double est[kN];
  for (unsigned m = 1; m <= 10048; ++m) {
    bool any = false;
    for (int c = 0; c < kN; ++c)
      if (tune_streamed(c, m, &len, 1) < 1e300) {
        any = true;
        if (!passes_ok(c, m)) ++bad;
      }
    if (!any) ++bad;  // every length up to the shared-memory limit keeps a class
    Tuning t;
    tuning_defaults(&t);
    if (!passes_ok(tuning_pick_single(&t, m, len), m)) ++bad;
    for (int i = 0; i < kTuneMBins; ++i)
      for (int j = 0; j < kTuneNBins; ++j) t.table[i][j] = 0;  // the class of the fewest rows, forced
    const double batch = tuning_estimate(&t, m, &len, 1, est, 0xFFFFFFFFu);
    const int c = tuning_forced(&t, m, len, est);
    if (c >= 0 && !passes_ok(c, m)) ++bad;
    forced += c == 0;
    TuneCost cost[kN];
    uint8_t front[kMaxTileClasses];
    tuning_costs(&t, m, len, 1, est, batch, 148, cost);
    const int n = tuning_front(cost, front);
    if (n == 0) ++bad;
    for (int i = 0; i < n; ++i) {
      if (!passes_ok(front[i], m)) ++bad;
      // shorter paths cost more, and a limit picks the cheapest class whose path is within it
      if (i && !(cost[front[i - 1]].path < cost[front[i]].path && cost[front[i - 1]].ps > cost[front[i]].ps)) ++bad;
      if (front[tuning_under(cost, front, n, cost[front[i]].path)] != front[i]) ++bad;
      for (int k = 0; k < kN; ++k)
        if (cost[k].path <= cost[front[i]].path && cost[k].ps < cost[front[i]].ps) ++bad;
    }
    if (n && front[tuning_under(cost, front, n, 0.0)] != front[0]) ++bad;
  }
  std::printf("%%d %%d\n", bad, forced);
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_no_class_beyond_the_pass_field(tmp_path):
    shapes = tile_classes()
    assert shapes[0] == (4, 8, 4)
    src = tmp_path / "passes.cpp"
    src.write_text(PROGRAM % ", ".join("{%d, %d, %d}" % s for s in shapes))
    exe = tmp_path / "passes"
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "sabertooth_b200", "csrc"), "-o", str(exe),
                    str(src)], check=True)
    bad, forced = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert bad == 0
    assert forced == 256 * 32  # and class 0 is still taken wherever its passes can be named
