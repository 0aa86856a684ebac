"""Which action sets have tables (csrc/rank_plan.h), on the CPU.

Per action set, over speeds 0.50 to 2.50 in steps of 0.01 on a grid of unit
spacing: plans without any table, plans without those of the edge cells, and plans
of 2^7 or 2^8 slots a unit, whose tables are too large for the shared memory of
four CTAs at ten modes.  The search must find the plans that trying every phase,
slot count and merge distance in turn finds.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "e2e_gpu_dp_b200", "csrc")

DRIVER = r"""
#include <cstdio>
#include "rank_plan.h"
using namespace e2e;
int main() {
  const int sets[][2] = {{1, 8}, {1, 12}, {1, 16}, {1, 24}, {1, 32}, {2, 8}, {2, 16}};
  std::vector<float> ticks;
  for (int i = 0; i < 200; ++i) ticks.push_back(0.5f + i);
  for (auto& s : sets) {
    int none = 0, plain = 0, large = 0;
    for (int k = 50; k <= 250; ++k) {
      const float F = k / 100.0f;
      std::vector<float> speed, angle;
      for (int i = 0; i < s[0]; ++i)
        for (int j = 0; j < s[1]; ++j) {
          speed.push_back((i + 1) * (F / s[0]));
          angle.push_back((float)(2 * M_PI * j / s[1]));
        }
      RankPlan P;
      if (!make_rank_plan(200, s[0] * s[1], 1.0, speed, angle, ticks, ticks, &P)) ++none;
      else if (P.slots_log2 >= 7) ++large;
      else if (P.groups[RANK_X_EDGE] == 0) ++plain;
    }
    std::printf("%dx%d none %d plain %d large %d\n", s[0], s[1], none, plain, large);
  }
}
"""


REACH = [
    "1x8 none 0 plain 1 large 14",
    "1x12 none 0 plain 1 large 35",
    "1x16 none 4 plain 6 large 51",
    "1x24 none 4 plain 9 large 117",
    "1x32 none 14 plain 13 large 139",
    "2x8 none 1 plain 3 large 65",
    "2x16 none 9 plain 10 large 148",
]


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_action_sets_with_tables(tmp_path):
    src = tmp_path / "reach.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "reach"
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    assert [ln for ln in out if ln] == REACH

