// Breakpoint tables of the ranked builder (builder_ranks.cu): host code, plus
// the lookup that the kernel and a CPU test share.
//
// Along one axis the landing cell of a sample is floor(a + 1/2) of its snapping
// coordinate a / D = j + A_a + p: the start cell's index j, the action's own
// displacement A_a = F cos(theta_a) dt / D and the velocity's p = v dt / D (the
// y axis with its sign turned).  So action a's cells change where p passes
// b - 1/2 - j - A_a for an integer b, and a domain clamp sets in where it passes
// an integer minus j + A_a: per action a fixed fraction of a cell, the same for
// every start cell up to float rounding.  The fractions of all actions, sorted,
// split every unit of p into G groups; the rank of a velocity is the number of
// breakpoints at or below it, and a pair of ranks decides the landing cells of
// every action.
//
// p is held in fixed point: q = round(p * 2^20) + constant, as the low mantissa
// bits of one fused multiply-add.  A table with 2^slots_log2 slots a unit has at
// most one breakpoint group in a slot, so one table word gives the rank:
//   s = word + q:  rank = s >> 16,  low 16 bits = distance behind the group's zone
// The zone of a group is where float rounding could put a sample on either side
// for one of its actions (the reference's chain rounds the velocity sum, the net
// velocity, the new position and the snapping coordinate); a sample in it, low
// 16 bits below the zone width, is `ambiguous` and takes the full expression.
#pragma once

#include <math.h>
#include <stdint.h>

#include <algorithm>
#include <vector>

#if defined(__CUDACC__)
#define E2E_RANK_FN __host__ __device__ __forceinline__
#else
#define E2E_RANK_FN inline
#endif

namespace e2e {

constexpr int kRankFrac = 20;                // fixed-point bits of a unit of p
constexpr int kRankUnits = 8;                // units a table spans
constexpr uint32_t kRankBits = 0x4B000000u;  // bits of 2^23: q's exponent
constexpr float kRankMagic = 8388608.0f;     // 2^23
constexpr int kRankMaxGroups = 64;
constexpr int kRankMaxActions = 32;
constexpr double kRankMaxDrift = 8.0;        // |mean p| of a cell that takes the tables

// kinds of tables: the x and y axis, each with the cell boundaries alone
// (plain) or with the clamps' breakpoints too (cells whose samples reach the
// domain's edge)
enum : int { RANK_X = 0, RANK_X_EDGE = 1, RANK_Y = 2, RANK_Y_EDGE = 3, RANK_KINDS = 4 };

// words of the plan: lut[kind][units << slots_log2], group zone starts
// [kind][kRankMaxGroups], then per kind and action the breakpoint index of the
// cell boundary (b = j = 0) and of the clamp (a = 0)
E2E_RANK_FN int rank_lut_words(int slots_log2) { return kRankUnits << slots_log2; }
E2E_RANK_FN int rank_gq_at(int slots_log2) { return RANK_KINDS * rank_lut_words(slots_log2); }
E2E_RANK_FN int rank_off_at(int slots_log2) { return rank_gq_at(slots_log2) + RANK_KINDS * kRankMaxGroups; }
E2E_RANK_FN int rank_plan_words(int slots_log2) { return rank_off_at(slots_log2) + RANK_KINDS * 2 * kRankMaxActions; }

// A cell's table along one axis: the range of steps around its velocities and
// where they lie in fixed point.
constexpr float kRankSigmas = 4.5f;        // half range: samples beyond it take the full expression
constexpr float kRankMaxHalfRange = 2.4f;  // of a table, in cells, so that its ends stay inside
struct RankRange {
  float bias;   // q = bits of fma(velocity sum, s, bias)
  int qa, qb;   // bits of the range's ends, in the zones of its first and last step: q is clamped to them
  int lut;      // word offset of the lookup table, so that lut + (q bits >> slot shift) is the slot's word
  int first;    // table index of the range's first step: ranks first + 1 .. first + n
  int org;      // samples of action a at or beyond cell boundary b: rank - first - 1 >= b * G + off[a] - org
  int n;        // ranks in the range
  int kind;
};

// mean_v: the cell's mean velocity (added to the mode sums); centre, var: mean
// and variance of the whole velocity (they choose the range only, no result
// depends on them); idx: the cell's index on the axis.  False: left to the
// general builder (spread or drift too wide for a table, a mean velocity of more than
// 56 cells that the modes cancel, or edge cells without one).
E2E_RANK_FN bool rank_range(const uint32_t* plan, int slots_log2, const int* groups, int axis, float s, double shift,
                            float a_min, float a_max, float mean_v, float centre, float var, int idx, int g,
                            RankRange* r) {
  const float unit = (float)(1 << kRankFrac);
  const float c = centre * s * (1.0f / unit) + (float)shift;
  const float h = kRankSigmas * sqrtf(var) * fabsf(s) * (1.0f / unit) + 1e-3f;
  if (!(fabsf(c) <= (float)kRankMaxDrift) || !(h <= kRankMaxHalfRange)) return false;
  const int n0 = (int)floorf(c - 0.5f) - 3;
  // (a float of less than 2^26 is within two units of the bias: the zones have three to spare)
  const double bias = (double)kRankMagic + ((double)mean_v * ((double)s / unit) + shift - n0) * unit;
  if (!(fabs(bias) < 67108864.0)) return false;
  const float pc = c - (float)n0;  // 3.5 .. 4.5
  const int ql = (int)((pc - h) * unit), qh = (int)((pc + h) * unit);
  for (int kind = 2 * axis; kind < 2 * axis + 2; ++kind) {
    const int G = groups[kind];
    if (G == 0) return false;
    const uint32_t* gq = plan + rank_gq_at(slots_log2) + kind * kRankMaxGroups;
    const int fl = ql & ((1 << kRankFrac) - 1), fh = qh & ((1 << kRankFrac) - 1);
    int kl = 0, kh = 0;
    for (int k = 0; k < G; ++k) {
      kl += (int)gq[k] <= fl ? 1 : 0;
      kh += (int)gq[k] <= fh ? 1 : 0;
    }
    // the last step at or below the range and the first one above it
    int ua = ql >> kRankFrac, ub = qh >> kRankFrac;
    if (--kl < 0) kl = G - 1, --ua;
    if (kh == G) kh = 0, ++ub;
    const int ba = ua * G + kl, bb = ub * G + kh;
    const int qa = (ua << kRankFrac) + (int)gq[kl], qb = (ub << kRankFrac) + (int)gq[kh];
    if (!(kind & 1)) {  // do samples in the range reach the domain's clamps?
      const float at = (float)(idx + n0) - (float)shift;
      if (!(at + a_min + (float)qa / unit > 0.01f && at + a_max + (float)qb / unit < (float)(g - 1) - 0.01f)) continue;
    }
    r->bias = (float)bias;
    r->qa = (int)kRankBits + qa;
    r->qb = (int)kRankBits + qb;
    r->lut = kind * rank_lut_words(slots_log2) - (int)(kRankBits >> (kRankFrac - slots_log2));
    r->first = ba;
    r->org = ba + (idx + n0) * G;
    r->n = bb - ba;
    r->kind = kind;
    return true;
  }
  return false;
}

struct RankPlan {
  int slots_log2 = 0;
  uint32_t zone_mask = 0;  // ambiguous: (s & zone_mask) == 0
  double shift = 0;        // p' = p - n0 + shift
  float sx = 0, sy = 0;    // q = fma(velocity sum, s, offset of the cell)
  int groups[RANK_KINDS] = {0, 0, 0, 0};
  double a_min[2] = {0, 0}, a_max[2] = {0, 0};  // displacements of the actions, x and y
  double err[2] = {0, 0};  // half zone width in units of p
  std::vector<uint32_t> words;
};

namespace rank_detail {

inline double half_ulp(double v) {
  v = fabs(v);
  return v < 1e-30 ? 0.0 : ldexp(1.0, ilogb(v) - 24);
}

inline bool pow2(double v) {
  int e;
  return v > 0 && frexp(v, &e) == 0.5;
}

// The breakpoints of one kind of table, z = their places in p' for b = j = n0 = 0 and
// a shift of 0, and their groups for a shift: zones [lo, hi] in fixed point
struct Breakpoints {
  int n = 0;
  double z[2 * kRankMaxActions];
  int order[2 * kRankMaxActions];  // by place within a unit; kept from one shift to the next, which rotates it
  int group[2 * kRankMaxActions];  // of breakpoint i
  int whole[2 * kRankMaxActions];  // its units
  int64_t lo[2 * kRankMaxActions], hi[2 * kRankMaxActions];
  int groups = 0;

  void add(double at) {
    order[n] = n;
    z[n++] = at;
  }

  // zones of h on each side of a breakpoint, those within tau of each other merged
  void make_groups(double shift, int h, int64_t tau) {
    const double one = ldexp(1.0, kRankFrac);
    double in[2 * kRankMaxActions];
    for (int i = 0; i < n; ++i) {
      const double at = z[i] + shift, w = floor(at);
      whole[i] = (int)w;
      in[i] = at - w;
    }
    for (int i = 1; i < n; ++i) {
      const int k = order[i];
      int to = i;
      for (; to > 0 && in[order[to - 1]] > in[k]; --to) order[to] = order[to - 1];
      order[to] = k;
    }
    groups = 0;
    for (int i = 0; i < n; ++i) {
      const int k = order[i];
      const int64_t q = (int64_t)floor(in[k] * one), l = q - h, r = q + 1 + h;
      if (groups && l <= hi[groups - 1] + tau) {
        hi[groups - 1] = std::max(hi[groups - 1], r);
      } else {
        lo[groups] = l;
        hi[groups++] = r;
      }
      group[k] = groups - 1;
    }
  }

  // whether some neighbouring zones lie between `from` and `to` apart: else both merge the same
  bool merges_differ(int h, int64_t from, int64_t to) {
    make_groups(0.0, h, from);
    for (int k = 0; k < groups; ++k) {
      const int64_t next = k + 1 < groups ? lo[k + 1] : lo[0] + ((int64_t)1 << kRankFrac);
      if (next - hi[k] <= to + 4) return true;  // (a shift moves a place by a unit)
    }
    return false;
  }

  // every group inside a slot of its own
  bool fits(int64_t slot_w) const {
    if (groups > kRankMaxGroups) return false;
    for (int k = 0; k < groups; ++k) {
      const int64_t s = lo[k] >= 0 ? lo[k] / slot_w : -1;
      if (lo[k] < 0 || hi[k] >= ((int64_t)1 << kRankFrac) || hi[k] / slot_w != s) return false;
      if (k && lo[k - 1] / slot_w == s) return false;
    }
    return true;
  }
};

}  // namespace rank_detail

// The tables of a problem, or false when the general builder has to take it:
// spacings that are no power of two (the grid's ticks and the reference's quotient
// then round, and some cells' numbers come out one lower: a step function too, but
// not the one of these tables), breakpoints too dense for a table.
//   speed, angle: the actions (float values); xs, ys: grid ticks
inline bool make_rank_plan(int g, int na, double dt, const std::vector<float>& speed, const std::vector<float>& angle,
                           const std::vector<float>& xs, const std::vector<float>& ys, RankPlan* out) {
  using namespace rank_detail;
  if (na < 2 || na > kRankMaxActions || g < 2 || !(dt > 0) || !std::isfinite(dt)) return false;
  const double D[2] = {fabs((double)xs[1] - xs[0]), fabs((double)ys[1] - ys[0])};
  double amax = 0;
  std::vector<double> disp[2];
  for (int ax = 0; ax < 2; ++ax) {
    if (!pow2(D[ax])) return false;
    for (int a = 0; a < na; ++a) {
      const double th = angle[a], sp = speed[a];
      const double v = ax == 0 ? sp * cos(th) * dt / D[ax] : -sp * sin(th) * dt / D[ax];
      if (!std::isfinite(v) || fabs(v) > 64) return false;
      disp[ax].push_back(v);
      amax = std::max(amax, fabs(sp) * dt / D[ax]);
    }
    out->a_min[ax] = *std::min_element(disp[ax].begin(), disp[ax].end());
    out->a_max[ax] = *std::max_element(disp[ax].begin(), disp[ax].end());
  }
  // Distance between a breakpoint's place in exact arithmetic and where the
  // float chain has it, in units of p: half an ulp of the velocity sum and of
  // the net velocity (times dt), of the new position, and of the snapping
  // coordinate; the ticks' own deviation from multiples of D; and the device's
  // cosine and sine (2 ulp) against the host's.
  //
  // The snapping coordinate is the position's distance from an end of the axis
  // (org).  It is finer than a float where the position is closer to 0 than the
  // distance is long: never on an x axis of positive coordinates (org the lower
  // end); on such a y axis (org the upper end) only where the position's own half
  // ulp is at most half the distance's, so 1.5 of the largest half ulp bound both.
  for (int ax = 0; ax < 2; ++ax) {
    const std::vector<float>& t = ax == 0 ? xs : ys;
    const double t0 = t[0], tn = t[g - 1], d = D[ax];
    const double top = std::max(fabs(t0), fabs(tn)) + d;
    double dev = 0;
    for (int i = 0; i < g; ++i) {
      const double got = ax == 0 ? t[i] - t0 : tn - t[g - 1 - i];
      if (!std::isfinite(got)) return false;
      dev = std::max(dev, fabs(got - i * d));
    }
    const double org = ax == 0 ? t0 : tn, ulp = 2 * half_ulp(top);
    const bool positive = t0 >= 0 && fmod(org, ulp) == 0;
    const double snap = !positive ? half_ulp(std::max(top, tn - t0 + d)) : ax == 0 ? 0.0 : 0.5 * half_ulp(top);
    const double drift = kRankMaxDrift + kRankMaxHalfRange + 1.1;  // of a sample in a range, with its last step's unit
    double e = half_ulp(drift * d / dt) * dt + half_ulp((drift + amax) * d / dt) * dt + half_ulp(top) + snap + dev +
               5e-7 * amax * d;
    out->err[ax] = 1.05 * e / d;
  }
  const double one = ldexp(1.0, kRankFrac);
  const int64_t unit = (int64_t)1 << kRankFrac;
  const int hq[2] = {(int)ceil(std::min(out->err[0], 1.0) * one) + 3, (int)ceil(std::min(out->err[1], 1.0) * one) + 3};
  out->sx = (float)(dt / D[0] * one);
  out->sy = (float)(-dt / D[1] * one);

  // merge distance (close breakpoints of different actions share a group with a
  // wider zone), slots a unit, and the phase of the slots: the first that gives
  // every group a slot of its own with its zone inside
  // (edge cells without tables, groups[..] = 0, when only the boundaries fit).
  // The search is part of every build: up to 0.1 ms where it fails (16 headings at
  // speed 1.3 took 0.21 ms and 32 headings 0.36 when every trial made its tables).
  Breakpoints kinds[RANK_KINDS];
  for (int kind = 0; kind < RANK_KINDS; ++kind) {
    for (int a = 0; a < na; ++a) kinds[kind].add(-0.5 - disp[kind / 2][a]);
    if (kind & 1)
      for (int a = 0; a < na; ++a) kinds[kind].add(-disp[kind / 2][a]);
  }
  for (int with_edge = 1; with_edge >= 0; --with_edge) {
    // with the clamps' breakpoints the tables that hold them are the fullest: tried first
    const int tables[4] = {RANK_X_EDGE, RANK_Y_EDGE, RANK_X, RANK_Y};
    const int skip = with_edge ? 0 : 2;
    int64_t tau_before = -1;
    for (int tau : {0, 64, 256, 1024}) {
      bool differs = tau_before < 0;
      for (int t = skip; t < 4 && !differs; ++t) differs = kinds[tables[t]].merges_differ(hq[tables[t] / 2], tau_before, tau);
      tau_before = tau;
      if (!differs) continue;
      for (int sl = 5; sl <= 8; ++sl) {
        for (int ph = 0; ph < 8; ++ph) {
          const double shift = (ph + 0.5) / (8.0 * (1 << sl));
          const int64_t slot_w = unit >> sl;
          int64_t widest = 1;
          bool ok = true;
          for (int t = skip; t < 4 && ok; ++t) {
            Breakpoints& b = kinds[tables[t]];
            b.make_groups(shift, hq[tables[t] / 2], tau);
            ok = b.fits(slot_w);
            for (int k = 0; k < b.groups && ok; ++k) widest = std::max(widest, b.hi[k] - b.lo[k] + 1);
          }
          if (!ok) continue;
          int64_t W = 1;
          while (W < widest) W *= 2;
          if (W > slot_w / 4) continue;
          out->words.assign((size_t)rank_plan_words(sl), 0u);
          uint32_t* const words = out->words.data();
          for (int kind = 0; kind < RANK_KINDS; ++kind) {
            const Breakpoints& b = kinds[kind];
            const bool have = with_edge || !(kind & 1);
            const int G = out->groups[kind] = have ? b.groups : 0, per = 1 << sl;
            int* off = reinterpret_cast<int*>(words + rank_off_at(sl) + kind * 2 * kRankMaxActions);
            for (int i = 0; i < b.n && have; ++i)  // breakpoint i: cell boundaries, then clamps, of action i % na
              off[(i / na) * kRankMaxActions + i % na] = b.whole[i] * G + b.group[i];
            for (int k = 0; k < G; ++k) words[rank_gq_at(sl) + kind * kRankMaxGroups + k] = (uint32_t)b.lo[k];
            for (int u = 0; u < kRankUnits; ++u) {
              int k = 0;
              for (int s = 0; s < per; ++s) {
                const int64_t start = (int64_t)u * unit + s * slot_w;
                uint32_t w = (uint32_t)(u * G + k) << 16;
                if (k < G && b.lo[k] / slot_w == s) {
                  w += 0x10000u - (uint32_t)(b.lo[k] - s * slot_w);
                  ++k;
                } else {
                  w += (uint32_t)W;
                }
                words[(size_t)kind * rank_lut_words(sl) + u * per + s] = w - (kRankBits + (uint32_t)start);
              }
            }
          }
          out->slots_log2 = sl;
          out->zone_mask = 0xffffu & ~((uint32_t)W - 1u);
          out->shift = shift;
          return true;
        }
      }
    }
  }
  return false;
}

}  // namespace e2e
