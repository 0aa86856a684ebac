"""The width of the ranked builder's zones (csrc/rank_plan.h), on the CPU.

A sample that the reference's float chain could put on either side of a step has to
lie in the step's zone.  Velocities are packed around every step, out to several
zone widths, on grids whose coordinates make the chain's roundings large: many
cells, where the snapping coordinate of the y axis is coarser than the position it
is taken from; negative coordinates, where that of the x axis is too; and mean
velocities that the modes cancel.  Outside the zones the rank has to give the cell
and the clamps of the reference's operations (move(), src/build_model.cu:268-356).
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "e2e_gpu_dp_b200", "csrc")

DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include "rank_plan.h"
using namespace e2e;

// gsize, headings, spacing, first tick, mean velocity in cells (cancelled by the sums)
int main(int, char** argv) {
  const int g = atoi(argv[1]), na = atoi(argv[2]);
  const float dx = (float)atof(argv[3]), x0 = (float)atof(argv[4]), mean = (float)atof(argv[5]) * dx;
  std::vector<float> tk(g), sp(na, 1.0f), an(na);
  for (int i = 0; i < g; ++i) tk[i] = x0 + (float)i * dx;
  for (int a = 0; a < na; ++a) an[a] = (float)(a * (2 * M_PI) / na);
  RankPlan P;
  if (!make_rank_plan(g, na, 1.0, sp, an, tk, tk, &P)) return std::printf("no plan\n"), 1;
  const uint32_t* words = P.words.data();
  const int sh = kRankFrac - P.slots_log2;
  std::mt19937 rng(3);
  long checked = 0, zone = 0, refused = 0;
  for (int ax = 0; ax < 2; ++ax)
    for (int rep = 0; rep < 40; ++rep) {
      const int idx = rep < 8 ? (rep & 1 ? g - 1 - rep / 2 : rep / 2) : (int)(rng() % g);
      const float drift = dx * (-1.5f + 3.0f * (float)(rng() % 1000) / 1000.0f), u = mean + drift, sig = 0.15f * dx;
      RankRange r;
      if (!rank_range(words, P.slots_log2, P.groups, ax, ax ? P.sy : P.sx, P.shift, (float)P.a_min[ax],
                      (float)P.a_max[ax], u, drift, sig * sig, idx, g, &r)) { ++refused; continue; }
      const int G = P.groups[r.kind];
      const int* off = (const int*)(words + rank_off_at(P.slots_log2)) + r.kind * 2 * kRankMaxActions;
      for (int a0 = 0; a0 < na; ++a0)
        for (int h = -3; h <= 3; ++h)
          for (int k = -600; k <= 600; ++k) {
            const double tr0 = ax ? -std::sin((double)an[a0]) : std::cos((double)an[a0]);
            const double p = 0.5 * h - tr0 / dx + 0.59 * k / (1 << kRankFrac);
            const float sum = (float)((ax ? -p : p) * dx - u), v = u + sum;
            const float qf = fmaf(sum, ax ? P.sy : P.sx, r.bias);
            int q;
            std::memcpy(&q, &qf, 4);
            q = std::min(std::max(q, r.qa), r.qb);
            const uint32_t w = words[(q >> sh) + r.lut] + (uint32_t)q;
            if ((w & P.zone_mask) == 0) { ++zone; continue; }
            const int rank = (int)(w >> 16) - r.first - 1;
            for (int a = 0; a < na; ++a) {
              const float tr = ax ? std::sin(an[a]) : std::cos(an[a]);
              float n = fmaf(fmaf(sp[a], tr, v), 1.0f, ax ? tk[g - 1 - idx] : tk[idx]);
              const int clamp = n > tk[g - 1] ? 1 : n < tk[0] ? -1 : 0;
              n = std::min(std::max(n, tk[0]), tk[g - 1]);
              const float at = ax ? -(n - tk[g - 1]) : n - tk[0], rem = remainderf(at, dx);
              const int cell = (int)((at - rem) / dx) + (rem >= 0.5 * dx ? 1 : 0);
              int got = 0, gc = 0;
              for (int b = std::max(1, idx - 20); b < std::min(g, idx + 20); ++b)
                if (rank >= b * G + off[a] - r.org) got = b;
              if (r.kind & 1) {
                const int e = off[kRankMaxActions + a] - r.org;
                gc = rank < e ? -1 : rank >= (g - 1) * G + e ? 1 : 0;
              }
              if (got != cell || gc != (ax ? -clamp : clamp))
                return std::printf("axis %d cell %d heading %d v=%.9g sum=%.9g: cell %d clamp %d, reference %d %d\n", ax,
                                   idx, a, v, sum, got, gc, cell, ax ? -clamp : clamp), 1;
              ++checked;
            }
          }
    }
  std::printf("OK checked %ld zone %ld refused %ld\n", checked, zone, refused);
  return refused == 80 || checked > 100000 ? 0 : 1;
}
"""


@pytest.fixture(scope="module")
def zones(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("needs a host C++ compiler")
    d = tmp_path_factory.mktemp("zones")
    (d / "zones.cpp").write_text(DRIVER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(d / "zones.cpp"), "-o",
                    str(d / "zones")], check=True)
    return str(d / "zones")


@pytest.mark.parametrize("g,na,dx,x0", [(200, 16, 1, 0.5), (520, 16, 1, 0.5), (1000, 16, 1, 0.5), (2000, 8, 1, 0.5),
                                        (4000, 8, 1, 0.5), (900, 8, 2, 1), (1000, 8, 0.5, 0.25), (200, 16, 1, -100.5),
                                        (1000, 8, 1, -500), (300, 8, 1, -7.25), (150, 8, 1, -3.3)])
def test_samples_outside_the_zones(zones, g, na, dx, x0):
    r = subprocess.run([zones, str(g), str(na), str(dx), str(x0), "0"], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout


@pytest.mark.parametrize("mean", [20, 50, -50, 60, 120, -120, 1000, -1000])
def test_mean_velocities_that_the_modes_cancel(zones, mean):
    r = subprocess.run([zones, "200", "16", "1", "0.5", str(mean)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout
