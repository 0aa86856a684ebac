"""The ranked builder's tables (csrc/rank_plan.h) against the reference's float
chain, on the CPU.

For a velocity that the tables do not call ambiguous, the rank must give, for
every action, the landing cell and the domain clamps of the reference's own
float operations (move(), src/build_model.cu:268-356), and must lie inside the
cell's table.  Velocities are drawn from the cell's distribution and packed
around every step of every action, in single ulps, with infinities and NaN
among them; grids, time steps, spacings and action sets cover the builder's
forms, edge cells included.  Ambiguous samples take the full expression, so
they only have to be few.
"""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "e2e_gpu_dp_b200", "csrc")

DRIVER = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include "rank_plan.h"
using namespace e2e;

struct Axis { float t0, tn, D, dt; int g, y; std::vector<float> tick; };

// landing index and clamp of one axis (x: org = tick[0]; y: -(new - tick[g-1]))
static void land(const Axis& A, float F, float tr, float v, int idx, int* bin, int* clamp) {
  const float x1 = A.y ? A.tick[A.g - 1 - idx] : A.tick[idx];
  float n = fmaf(fmaf(F, tr, v), A.dt, x1);
  *clamp = (n > A.tn) ? 1 : (n < A.t0 ? -1 : 0);
  if (n > A.tn) n = A.tn;
  else if (n < A.t0) n = A.t0;
  const float a = A.y ? -(n - A.tn) : n - A.t0;
  const float rem = remainderf(a, A.D);
  int k = (int)((a - rem) / A.D);
  if (rem >= 0.5 * A.D) k += 1;
  *bin = k;
}

int main() {
  struct C { int g, na, ns; double F, dt, dx, x0; };
  const C cases[] = {{200, 16, 1, 1, 1, 1, .5}, {50, 8, 1, 1, 1, 1, .5}, {137, 12, 2, 1.5, 1, 1, .5},
                     {120, 8, 1, 1, .5, .5, .25}, {300, 16, 1, 1, 1, 1, .5}, {21, 16, 2, 1.5, 1, 1, .5},
                     {2, 8, 1, 1, 1, 1, .5}, {5, 12, 1, 1, .5, .5, .25}, {100, 8, 4, 3, 1, 1, .5},
                     {64, 16, 1, 1.3, .7, 2, 1}, {90, 2, 1, 1, 1, 1, .5}, {70, 8, 1, .6, .25, .25, 0.3},
                     {1000, 16, 1, 1, 1, 1, .5}, {33, 32, 1, 1, 1, 1, -7.3}};
  std::mt19937_64 rng(5);
  std::normal_distribution<float> gauss;
  long checked = 0, ambiguous = 0, planned = 0, gaussian = 0, gaussian_amb = 0;
  for (const C& c : cases) {
    const int na = c.na * c.ns;
    std::vector<float> tk(c.g), sp, an;
    for (int i = 0; i < c.g; ++i) tk[i] = (float)c.x0 + (float)i * (float)c.dx;
    for (int i = 0; i < c.ns; ++i)
      for (int j = 0; j < c.na; ++j) {
        sp.push_back(c.ns == 1 ? (float)c.F : (float)(i + 1) * ((float)c.F / (float)c.ns));
        an.push_back((float)(j * (2 * M_PI) / c.na));
      }
    RankPlan P;
    if (!make_rank_plan(c.g, na, (float)c.dt, sp, an, tk, tk, &P)) { std::printf("no plan: g=%d na=%d\n", c.g, na); continue; }
    ++planned;
    const uint32_t* words = P.words.data();
    const int sh = kRankFrac - P.slots_log2;
    for (int ax = 0; ax < 2; ++ax) {
      Axis A{tk[0], tk[c.g - 1], (float)c.dx, (float)c.dt, c.g, ax, tk};
      std::vector<float> tr(na);
      for (int a = 0; a < na; ++a) tr[a] = ax ? std::sin(an[a]) : std::cos(an[a]);
      const int* off0 = (const int*)(words + rank_off_at(P.slots_log2));
      for (int rep = 0; rep < 60; ++rep) {
        int idx = rep < 12 ? std::min(rep / 2, c.g - 1) : rep < 24 ? std::max(c.g - 1 - (rep - 12) / 2, 0)
                                                                : (int)(rng() % c.g);
        const float scale = (float)(c.dx / c.dt);
        const float u = scale * 0.9f * gauss(rng), sig = scale * 0.02f * (1 + rep % 25);
        RankRange r;
        if (!rank_range(words, P.slots_log2, P.groups, ax, ax ? P.sy : P.sx, P.shift, (float)P.a_min[ax],
                        (float)P.a_max[ax], u, u, sig * sig, idx, c.g, &r)) continue;
        const int G = P.groups[r.kind];
        const int* off = off0 + r.kind * 2 * kRankMaxActions;
        if (r.n < 1) { std::printf("FAIL empty range\n"); return 1; }
        std::vector<float> sums;
        for (int k = 0; k < 400; ++k) sums.push_back(sig * gauss(rng));
        const size_t ngauss = sums.size();
        const float inf = std::numeric_limits<float>::infinity();
        for (float s : {inf, -inf, std::nanf(""), 1e30f, -1e30f, 0.f, -0.f, 3e38f}) sums.push_back(s);
        for (int a = 0; a < na; ++a)
          for (int h = -2 * 6; h <= 2 * 6; ++h) {  // half-integer and integer steps around the cell
            const double disp = (ax ? -1.0 : 1.0) * (double)sp[a] * tr[a] * c.dt / c.dx;
            const double p = 0.5 * h - disp;
            float s = (float)((ax ? -p : p) * c.dx / c.dt - u);
            for (int k = 0; k < 6; ++k) s = std::nextafterf(s, -inf);
            for (int k = 0; k < 12; ++k, s = std::nextafterf(s, inf)) sums.push_back(s);
            for (double d : {3e-6, 1e-5, 3e-5, 1e-4})
              for (int sg = -1; sg <= 1; sg += 2) sums.push_back((float)(((ax ? -p : p) + sg * d) * c.dx / c.dt - u));
          }
        for (size_t k = 0; k < sums.size(); ++k) {
          const float s = sums[k], v = u + s;
          const float qf = fmaf(s, ax ? P.sy : P.sx, r.bias);
          int q;
          std::memcpy(&q, &qf, 4);
          q = std::min(std::max(q, r.qa), r.qb);
          const int at = (q >> sh) + r.lut;
          if (at < 0 || at >= RANK_KINDS * rank_lut_words(P.slots_log2)) { std::printf("FAIL lookup index\n"); return 1; }
          const uint32_t w = words[at] + (uint32_t)q;
          if (k < ngauss) ++gaussian;
          if ((w & P.zone_mask) == 0) { ++ambiguous; gaussian_amb += k < ngauss; continue; }
          const int lr = (int)(w >> 16) - r.first - 1;
          if (lr < 0 || lr >= r.n) { std::printf("FAIL rank %d of %d: g=%d na=%d s=%g\n", lr, r.n, c.g, na, s); return 1; }
          for (int a = 0; a < na; ++a) {
            int bin, cl;
            land(A, sp[a], tr[a], v, idx, &bin, &cl);
            // the cells' boundaries at or below the rank
            int got = 0;
            for (int b = std::max(1, idx - 40); b < c.g && b < idx + 40; ++b) {
              if (lr >= b * G + off[a] - r.org) got = b;
              else break;
            }
            if (idx > 40 && got == 0) { std::printf("FAIL range of the check\n"); return 1; }
            int gcl = 0;
            if (r.kind & 1) {
              const int lo = off[kRankMaxActions + a] - r.org, hi = (c.g - 1) * G + off[kRankMaxActions + a] - r.org;
              gcl = lr < lo ? -1 : lr >= hi ? 1 : 0;
              if (ax) gcl = -gcl;  // ay < 0 is y above the last tick
            }
            if (got != bin || gcl != cl) {
              std::printf("FAIL g=%d na=%d axis=%d idx=%d a=%d v=%.9g: cell %d clamp %d, reference %d %d (kind %d)\n", c.g,
                          na, ax, idx, a, v, got, gcl, bin, cl, r.kind);
              return 1;
            }
            ++checked;
          }
        }
      }
    }
  }
  std::printf("OK planned=%ld checked=%ld ambiguous=%ld gaussian=%ld listed=%ld\n", planned, checked, ambiguous, gaussian,
              gaussian_amb);
  if (planned < 13 || checked < 1000000 || gaussian_amb * 100 > gaussian) return 1;
  return 0;
}
"""


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs a host C++ compiler")
def test_ranks_give_the_reference_cells(tmp_path):
    src = tmp_path / "ranks.cpp"
    src.write_text(DRIVER)
    exe = tmp_path / "ranks"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.startswith("OK"), r.stdout
