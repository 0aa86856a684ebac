// K1 by velocity ranks: the Monte-Carlo transition builder for grids whose
// spacing is a power of two, up to ten modes and 2 to 32 actions; groups of
// cells it cannot take (velocities spread too widely for a table, rows with
// samples outside their 8x8 window) are marked and left to k_build_listed.
//
// transition_calc (src/build_model.cu:483-559) moves every sample of every
// action.  But along one axis the landing cell is a step function of the
// velocity alone, and the steps of all actions lie at the same few places of
// every cell (rank_plan.h).  So a velocity is ranked once among the steps of all
// actions, one table lookup per axis, a cell's samples are counted by their
// pair of ranks, and prefix sums over that small table give each action's cell
// counts as differences of four entries:
//   per (cell, realisation): the mode sum (20 fused multiply-adds, packed two
//     realisations at a time) and about 17 more instructions, for all actions
//     together, against 11-14 per action of the counting loops;
//   per (cell, action): at most 81 table reads.
// A sample within the zone of a step (where the reference's float rounding
// decides) or outside the table's range, about 1 in 2000 (1 in 1000 on a thousand cells a side), goes to the cell's
// list and takes the reference's full expression for each action.  Counts are
// the reference's exactly; rewards are folded from the counts as in
// k_build_tiles.
//
// Measured on B200 (whole call, counting loops -> ranks): 200x200x120, 16
// actions, 5000 realisations 330.6 -> 61.5 ms; 300x300x40, 2000 realisations
// 102.3 -> 23.6 ms; 137x137x53, 24 actions, 777 realisations 29.7 -> 8.7 ms.
// Of the 13.8 ms of 200x200x30 the counting takes about 10 ms (the shared-memory
// pipe at 60 % of its peak, issue slots at 62 %), staging 0.9,
// the prefix sums 0.5, the rows 2.4.  Four or five CTAs of 4 warps an SM: one
// CTA's staging and rows run beside the others' counting (two of 8 warps: 16.8
// ms, four of 4: 14.3); the table reads of a lane's four samples before their
// increments: 15.5 -> 14.3 ms.
//
// A CTA (4 warps) takes a run of cells of one layer, 128 rows where the action
// count allows it.  A warp holds the coefficients of 128 realisations (4 a
// lane) in registers and walks a subset of the cells, whose modes it reads as
// broadcasts; the tables of the cells are shared by the CTA's warps (atomic
// increments, no order needed).
#include <algorithm>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "kernels.h"
#include "rank_plan.h"
#include "tile_order.h"

namespace e2e {

namespace {

constexpr int kThreads = 128;     // 4 or 5 CTAs an SM: one CTA's set-up and rows overlap the others' counting
constexpr int kWarps = kThreads / 32;
constexpr int kWin = 8;           // window side, as k_build_tiles
constexpr int kListPool = 384;    // samples on the lists of a CTA's cells
constexpr int kObsR = 10;         // obstacle bitmap radius around a cell
constexpr int kObsRows = 2 * kObsR + 1;
constexpr int kMaxCells = 32;     // cells of a CTA
constexpr int kMaxTiles = 4;      // emission tiles of a CTA, one a warp
constexpr int kRewardR = 6;       // reach of k_rank_rewards' tables around a cell

// A cell of the CTA and its table
struct __align__(16) CellTab {
  float bx, bx2, by, by2;  // fixed-point offset of a velocity sum, x and y, each twice
  int qax, qbx, qay, qby;  // the ranges' ends (bits): the zones of their first and last step
  uint32_t lx, ly;         // shared address of slot 0 of the axis' lookup table, less q's constant bits
  uint32_t mul;            // counter index = rank_x + rank_y * stride + cst: 1 | stride << 8;
  uint32_t cst;            //   mul is 0 while the cell is not counted
  int bax, bay;            // step index of the range's lower end, in table units
  int orgx, orgy;          // step index of cell boundary b: b * G + off[action] - org
  int nx, ny;              // ranks in the table
  int stride, base;        // row stride and first word of the prefix sums (ny + 1 x nx + 1)
  int kx, ky;              // table kinds
  float u1, v1;
  int i1, j1;
  int state;               // 0 counted, 1 nothing to count (terminal or obstacle cell, beyond the
                           // layer), 2 left to the general builder
  int pad;
};

// a word of the lookup tables, which nothing writes while samples are counted:
// not volatile, so that the loads of several samples are in flight together
__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
  uint32_t v;
  asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}

__device__ __forceinline__ void reds_inc(uint32_t addr) {
  asm volatile("red.shared.add.u32 [%0], 1;" ::"r"(addr) : "memory");
}

// The counts of 4 realisations a lane (rows r0 .. r0 + 3 of the coefficients)
// over the cells [c_lo, c_hi).  Sums: extract_velocity's (src/build_model.cu:
// 389-401), for each realisation and component a chain of fused multiply-adds in
// mode order.  A sample in a step's zone, or clamped into the zone at its
// range's end (NaN and overflow too: their bits lie beyond an end), counts in the
// pool's word 0 and goes to the cell's list.
template <int NM, bool FULL>
__device__ __forceinline__ void count_block(const RankArgs& K, const float* yt, int r0, int nrz, const float4* md,
                                            const CellTab* cells, int c_lo, int c_hi, uint32_t pool, int* lcnt,
                                            float2* list, int lcap) {
  float2 y01[NM], y23[NM];
#pragma unroll
  for (int k = 0; k < NM; ++k) {
    const float4 y = __ldg(reinterpret_cast<const float4*>(yt + (int64_t)k * K.nrp + r0));
    y01[k] = make_float2(y.x, y.y);
    y23[k] = make_float2(y.z, y.w);
  }
  const int sh = kRankFrac - K.slots_log2;
  const uint32_t zm = K.zone_mask;
  const float2 fx = make_float2(K.sx, K.sx), fy = make_float2(K.sy, K.sy);
  for (int c = c_lo; c < c_hi; ++c) {
    const CellTab* ct = cells + c;
    const uint4 h2 = *reinterpret_cast<const uint4*>(&ct->lx);
    if (h2.z == 0u) continue;
    const float4 h0 = *reinterpret_cast<const float4*>(ct);
    const int4 h1 = *reinterpret_cast<const int4*>(&ct->qax);
    float2 sx01, sx23, sy01, sy23;
    {
      const float4 m = md[c * NM];
      const float2 mu = make_float2(m.x, m.y), mv = make_float2(m.z, m.w);
      sx01 = __fmul2_rn(mu, y01[0]);  // fma(m, y, 0) but for the sign of a zero, which no result depends on
      sx23 = __fmul2_rn(mu, y23[0]);
      sy01 = __fmul2_rn(mv, y01[0]);
      sy23 = __fmul2_rn(mv, y23[0]);
    }
#pragma unroll
    for (int k = 1; k < NM; ++k) {
      const float4 m = md[c * NM + k];
      const float2 mu = make_float2(m.x, m.y), mv = make_float2(m.z, m.w);
      sx01 = __ffma2_rn(mu, y01[k], sx01);
      sx23 = __ffma2_rn(mu, y23[k], sx23);
      sy01 = __ffma2_rn(mv, y01[k], sy01);
      sy23 = __ffma2_rn(mv, y23[k], sy23);
    }
    const float2 bx = make_float2(h0.x, h0.y), by = make_float2(h0.z, h0.w);
    const float2 qx01 = __ffma2_rn(sx01, fx, bx), qx23 = __ffma2_rn(sx23, fx, bx);
    const float2 qy01 = __ffma2_rn(sy01, fy, by), qy23 = __ffma2_rn(sy23, fy, by);
    const float qx[4] = {qx01.x, qx01.y, qx23.x, qx23.y}, qy[4] = {qy01.x, qy01.y, qy23.x, qy23.y};
    uint32_t s[4], t[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s[i] = (uint32_t)min(max(__float_as_int(qx[i]), h1.x), h1.y);
      t[i] = (uint32_t)min(max(__float_as_int(qy[i]), h1.z), h1.w);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s[i] += lds_u32(h2.x + ((s[i] >> sh) << 2));
      t[i] += lds_u32(h2.y + ((t[i] >> sh) << 2));
    }
    bool listed[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t at = __dp2a_lo(__byte_perm(s[i], t[i], 0x7632), h2.z, h2.w);
      listed[i] = (s[i] & zm) == 0u || (t[i] & zm) == 0u;
      if (!FULL && r0 + i >= nrz) {
        listed[i] = false;
        at = 0u;
      }
      if (listed[i]) at = 0u;
      reds_inc(pool + (at << 2));
    }
    if (listed[0] || listed[1] || listed[2] || listed[3]) {
      const float sx[4] = {sx01.x, sx01.y, sx23.x, sx23.y}, sy[4] = {sy01.x, sy01.y, sy23.x, sy23.y};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (listed[i]) {
          const int at = atomicAdd(lcnt + c, 1);
          if (at < lcap) list[c * lcap + at] = make_float2(ct->u1 + sx[i], ct->v1 + sy[i]);
        }
      }
    }
  }
}

// the reference's obstacle override of (i1, j1) -> (i1 + di, j1 + dj)
// (goes_through_obstacle, src/build_model.cu:444-477) from the cell's obstacle
// bits: the same within_band tests, for the obstacle cells of the box only
__device__ __forceinline__ bool passes_obstacle(const DevProblem& P, const int32_t* mask, int T, const uint32_t* rows,
                                                int i1, int j1, int di, int dj) {
  if (abs(di) > kObsR || abs(dj) > kObsR) return through_obstacle(P, mask, T, i1, j1, i1 + di, j1 + dj);
  const int a0 = min(di, 0), a1 = max(di, 0), b0 = min(dj, 0), b1 = max(dj, 0);
  const uint32_t cols = ((2u << (b1 - b0)) - 1u) << (b0 + kObsR);
  for (int a = a0; a <= a1; ++a) {
    uint32_t m = rows[a + kObsR] & cols;
    if (!m) continue;
    if (di == 0 || dj == 0) return true;  // within_band of an axis-parallel way
    do {
      const int b = __ffs(m) - 1 - kObsR;
      if (within_band(P, i1 + a, j1 + b, i1, j1, i1 + di, j1 + dj)) return true;
      m &= m - 1;
    } while (m);
  }
  return false;
}

__device__ __forceinline__ void land_any(const DevProblem& P, float F, float cs, float sn, float vx, float vy, float x,
                                         float y, int& i2, int& j2) {
  if (P.unit_step) land_unit(P, F, cs, sn, vx, vy, x, y, i2, j2);
  else land_general(P, F, cs, sn, vx, vy, x, y, i2, j2);
}

// obstacle bits of the rows around the CTA's cells c0 .. c0 + n - 1 of layer T
__device__ __forceinline__ void stage_obstacles(const RankArgs& K, int T, int g, int nc, int c0, int n, int i0, int j0,
                                                uint32_t* orow) {
  for (int e = threadIdx.x; e < n * kObsRows; e += kThreads) {
    const int c = e / kObsRows, a = e - c * kObsRows - kObsR;
    uint32_t bits = 0;
    if (c0 + c < nc) {
      int i = i0 + a, j = j0 + c;
      for (; j >= g; j -= g) ++i;
      if (i >= 0 && i < g) {
        const uint32_t* row = K.obits + ((int64_t)T * g + i) * K.owords;
        const int b = j - kObsR, w = b >> 5;
        const uint32_t lo = w >= 0 ? __ldg(row + w) : 0u, hi = w + 1 < K.owords ? __ldg(row + w + 1) : 0u;
        bits = __funnelshift_r(lo, hi, b & 31) & ((1u << kObsRows) - 1u);
        if (a == 0) bits &= ~(1u << kObsR);  // the cell itself does not count
      }
    }
    orow[e] = bits;
  }
}

// reward of a sample of `cell` (speed F) that lands in (i2, j2) after k domain
// clamps, no obstacle on its way: move() and transition_calc
// (src/build_model.cu:291-354, :533), the additions in their order
__device__ __forceinline__ float landing_reward(const BuildArgs& A, int T, bool late, bool rad, float F, int cell, int i2,
                                                int j2, int k) {
  const DevProblem& P = A.P;
  const int64_t nc = (int64_t)P.g * P.g;
  float r = 0.f;
  for (; k > 0; --k) r += P.r_out;
  if (i2 == 0 || i2 == P.g - 1 || j2 == 0 || j2 == P.g - 1) r += P.r_out;
  if (is_terminal(P, i2, j2)) {
    r += P.r_term;
  } else {
    if (late) r += 0.05 * P.r_out;
  }
  float rad1 = 0.f, rad2 = 0.f;
  if (rad) {
    rad1 = __ldg(A.F.s + (int64_t)T * nc + cell);
    rad2 = __ldg(A.F.s + (int64_t)(T + 1) * nc + (int64_t)i2 * P.g + j2);
  }
  const float r_step = step_reward(P, F, rad1, rad2);
  return r + r_step;
}

struct Smem {
  uint32_t* lut;     // the plan's words
  float* tab;        // 32 x 8 landing rewards
  float4* md;        // cells x NM modes: (ui, ui, vi, vi)
  CellTab* cells;
  uint32_t* orow;    // cells x kObsRows obstacle bits
  int* lcnt;         // cells: samples on the list
  float2* list;      // kListPool
  uint16_t* wcol;    // warps x 64 bins x 32 rows: counts of the rows a warp finishes
  uint32_t* pool;    // rank tables
};

__host__ __device__ inline size_t smem_fixed_bytes(int slots_log2, int nm, int ct) {
  size_t b = sizeof(uint32_t) * (size_t)rank_plan_words(slots_log2);
  b += sizeof(float) * 32 * 8;
  b += sizeof(float4) * (size_t)ct * nm;
  b += sizeof(CellTab) * (size_t)ct;
  b += sizeof(uint32_t) * (size_t)((ct * kObsRows + 3) & ~3);
  b += sizeof(int) * kMaxCells;
  b += sizeof(float2) * kListPool;
  b += sizeof(uint16_t) * (size_t)kWarps * 64 * 32;
  return b;
}

// the rows of one emission tile (32 / P cells x P action lanes of a warp):
// window counts from the prefix sums and the lists, rewards, emission
template <typename Dummy = void>
__device__ __forceinline__ void finish_tile(const BuildArgs& A, const RankArgs& K, const Smem& S, int T, int64_t c0,
                                            int tile, int lcap) {
  const DevProblem& P = A.P;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = P.g;
  const int64_t nc = (int64_t)g * g;
  const int cpw_log2 = 5 - A.lanes_log2;
  const int cl = (tile << cpw_log2) + (lane >> A.lanes_log2);
  const int a = lane & ((1 << A.lanes_log2) - 1);
  const int64_t cell = c0 + cl;
  const int64_t et = (c0 >> cpw_log2) + tile;  // emission tile within the layer
  if (c0 + ((int64_t)tile << cpw_log2) >= nc) return;  // beyond the layer (whole warp)
  const CellTab& ct = S.cells[cl];
  const bool valid = cell < nc && a < P.na;
  uint16_t* const wcol = S.wcol + warp * 64 * 32 + lane;
  const int i1 = valid ? ct.i1 : 0, j1 = valid ? ct.j1 : 0;
  const int aa = a < P.na ? a : 0;
  const float F = P.ac_speed[aa], cs = P.ac_cos[aa], sn = P.ac_sin[aa];
  const float x1 = P.xs[j1], y1 = P.ys[g - 1 - i1];
  const bool late = T > P.nt - 20;
  const bool rad = P.reward_type == 2 || P.reward_type == 3;
  const int W = g < kWin ? g : kWin;
  bool window = valid && ct.state != 1;
  bool ok = !(valid && ct.state >= 2);
  const int nlist = window ? S.lcnt[cl] : 0;
  ok = ok && nlist <= lcap;
  int wi0 = 0, wj0 = 0, n_cl = 0;
  uint64_t nz = 0, ovr = 0;
  if (window && ok) {
    int ci, cj;  // the window around the mean flow's landing, as k_build_tiles
    land_any(P, F, cs, sn, ct.u1, ct.v1, x1, y1, ci, cj);
    wi0 = min(max(ci - (kWin / 2 - 1), i1 - P.del), i1 + P.del - W + 1);
    wj0 = min(max(cj - (kWin / 2 - 1), j1 - P.del), j1 + P.del - W + 1);
    wi0 = min(max(wi0, 0), g - W);
    wj0 = min(max(wj0, 0), g - W);
    const int* offs = reinterpret_cast<const int*>(S.lut + rank_off_at(K.slots_log2));
    const int Gx = K.groups[ct.kx], Gy = K.groups[ct.ky];
    const int nx = ct.nx, ny = ct.ny, stride = ct.stride;
    const uint32_t* sat = S.pool + ct.base;
    const int tx = wj0 * Gx + offs[ct.kx * 2 * kRankMaxActions + aa] - ct.orgx;
    const int ty = wi0 * Gy + offs[ct.ky * 2 * kRankMaxActions + aa] - ct.orgy;
    // ranks below window column lj; a clamped sample lands in the edge cell, so
    // the grid's first and last cell have no outer boundary
    int cx[kWin + 1];
#pragma unroll
    for (int lj = 0; lj <= kWin; ++lj) {
      int t = min(max(tx + lj * Gx, 0), nx);
      if (wj0 + lj <= 0) t = 0;
      if (wj0 + lj >= g) t = nx;
      if (lj > W) t = cx[lj > 0 ? lj - 1 : 0];
      cx[lj] = t;
    }
    auto row_of = [&](int li) -> int {
      int t = min(max(ty + li * Gy, 0), ny);
      if (wi0 + li <= 0) t = 0;
      if (wi0 + li >= g) t = ny;
      return t;
    };
    uint32_t inside = 0;
    int r0 = row_of(0);
    for (int li = 0; li < W; ++li) {
      const int r1 = row_of(li + 1);
      if (r1 > r0) {
        const uint32_t* p0 = sat + r0 * stride;
        const uint32_t* p1 = sat + r1 * stride;
        uint32_t left = p1[cx[0]] - p0[cx[0]];
#pragma unroll
        for (int lj = 0; lj < kWin; ++lj) {
          if (cx[lj + 1] > cx[lj]) {
            const uint32_t right = p1[cx[lj + 1]] - p0[cx[lj + 1]];
            const uint32_t n = right - left;
            left = right;
            if (n) {
              const int b = li * kWin + lj;
              wcol[b * 32] = (uint16_t)n;
              nz |= 1ull << b;
              inside += n;
            }
          }
        }
      }
      r0 = r1;
    }
    ok = inside == (uint32_t)(P.nrzns - nlist);  // else samples outside the window
    // the listed samples, by the full expression
    bool clamped = false;
    for (int e = 0; e < nlist && ok; ++e) {
      const float2 v = S.list[cl * lcap + e];
      int i2, j2;
      land_any(P, F, cs, sn, v.x, v.y, x1, y1, i2, j2);
      const int li = i2 - wi0, lj = j2 - wj0;
      ok = (unsigned)li < (unsigned)W && (unsigned)lj < (unsigned)W;
      if (ok) {
        const int b = li * kWin + lj;
        const uint64_t bit = 1ull << b;
        wcol[b * 32] = (uint16_t)((nz & bit) ? wcol[b * 32] + 1 : 1);
        nz |= bit;
        clamped = clamped || i2 == 0 || j2 == 0 || i2 == g - 1 || j2 == g - 1;
      }
    }
    if (ok) {
      for (uint64_t m = nz; m; m &= m - 1) {
        const int b = __ffsll((long long)m) - 1;
        const int i2 = wi0 + (b >> 3), j2 = wj0 + (b & 7);
        // k_rank_rewards: landings within its tables, none that the general
        // builder takes out of the samples' order
        if (K.seq_rewards) {
          const int reach = min(P.del, kRewardR);
          ok = ok && abs(i2 - i1) <= reach && abs(j2 - j1) <= reach;
        }
        if (passes_obstacle(P, A.F.mask, T, S.orow + cl * kObsRows, i1, j1, i2 - i1, j2 - j1)) ovr |= 1ull << b;
      }
      // domain clamps of the samples in bins that no obstacle overrides: each adds
      // one r_outbound (move(), src/build_model.cu:291-310)
      if (clamped) {
        for (int e = 0; e < nlist; ++e) {
          const float2 v = S.list[cl * lcap + e];
          int i2, j2;
          land_any(P, F, cs, sn, v.x, v.y, x1, y1, i2, j2);
          const int b = (i2 - wi0) * kWin + j2 - wj0;
          if ((ovr >> b) & 1ull) continue;
          float xn, yn;
          advect(P, F, cs, sn, v.x, v.y, x1, y1, xn, yn);
          n_cl += (xn > P.xsn || xn < P.xs0) ? 1 : 0;
          n_cl += (yn > P.ysn || yn < P.ys0) ? 1 : 0;
        }
      }
      auto rect = [&](int ra, int rb, int ca, int cb) -> int {
        if (rb <= ra || cb <= ca) return 0;
        return (int)(sat[rb * stride + cb] - sat[ra * stride + cb] - sat[rb * stride + ca] + sat[ra * stride + ca]);
      };
      if (ct.kx & 1) {
        const int te = offs[ct.kx * 2 * kRankMaxActions + kRankMaxActions + aa] - ct.orgx;
        for (int side = 0; side < 2; ++side) {
          const int lj = side ? g - 1 - wj0 : -wj0;
          if (lj < 0 || lj >= W) continue;
          const int t = min(max(te + (side ? g - 1 : 0) * Gx, 0), nx);
          const int ca = side ? t : 0, cb = side ? nx : t;
          for (int li = 0; li < W; ++li)
            if (!((ovr >> (li * kWin + lj)) & 1ull)) n_cl += rect(row_of(li), row_of(li + 1), ca, cb);
        }
      }
      if (ct.ky & 1) {
        const int te = offs[ct.ky * 2 * kRankMaxActions + kRankMaxActions + aa] - ct.orgy;
        for (int side = 0; side < 2; ++side) {
          const int li = side ? g - 1 - wi0 : -wi0;
          if (li < 0 || li >= W) continue;
          const int t = min(max(te + (side ? g - 1 : 0) * Gy, 0), ny);
          const int ra = side ? t : 0, rb = side ? ny : t;
#pragma unroll
          for (int lj = 0; lj < kWin; ++lj)
            if (!((ovr >> (li * kWin + lj)) & 1ull)) n_cl += rect(ra, rb, cx[lj], cx[lj + 1]);
        }
      }
    }
  }
  if (__any_sync(0xffffffffu, !ok)) {  // the tile goes to the general builder
    const bool inner = !__any_sync(0xffffffffu, valid && in_edge_band(i1, j1, g));
    if (lane == 0) {
      uint8_t* const left = A.defer + T * defer_bytes(K.etiles_per_layer);
      left[kDeferCounts + et] = inner ? TILE_INNER : TILE_EDGE;
      atomicAdd(reinterpret_cast<unsigned int*>(left) + inner, 1u);
      atomicAdd(A.counters + CTR_DEFERRED, 1ull);
    }
    return;
  }
  float sumR = 0.f;
  uint32_t n_drop = 0, n_misbin = 0;
  if (window) {
    // the rewards folded from the counts, as k_build_tiles' fold_window
    const float rad1 = rad ? __ldg(A.F.s + (int64_t)T * nc + cell) : 0.f;
    for (uint64_t m = nz; m; m &= m - 1) {
      const int b = __ffsll((long long)m) - 1;
      const uint32_t c = wcol[b * 32];
      const int i2 = wi0 + (b >> 3), j2 = wj0 + (b & 7);
      float r;
      if ((ovr >> b) & 1ull) {
        r = P.r_out;
      } else {
        const int k = (i2 == 0 || i2 == g - 1 || j2 == 0 || j2 == g - 1) ? 1 : 0;
        const bool tm = is_terminal(P, i2, j2);
        if (!rad) {
          r = S.tab[aa * 8 + (tm ? 4 : 0) + k];
        } else {
          const float rad2 = __ldg(A.F.s + (int64_t)(T + 1) * nc + (int64_t)i2 * g + j2);
          r = k ? P.r_out : 0.f;
          if (tm) r += P.r_term;
          else if (late) r += 0.05 * P.r_out;
          r += step_reward(P, F, rad1, rad2);
        }
      }
      sumR = __fmaf_rn((float)c, r, sumR);
      if (abs(i2 - i1) > P.del || abs(j2 - j1) > P.del) {  // the reference counts its reward only
        n_drop += c;
        if (i2 - i1 + P.del < P.m && j2 - j1 + P.del < P.m) n_misbin += c;
        nz &= ~(1ull << b);
      }
    }
    sumR = __fmaf_rn((float)n_cl, P.r_out, sumR);
    if (n_drop) atomicAdd(A.counters + CTR_DROPPED, (unsigned long long)n_drop);
    if (n_misbin) atomicAdd(A.counters + CTR_MISBIN, (unsigned long long)n_misbin);
  } else if (valid && !is_terminal(P, i1, j1)) {
    sumR = K.stay_sum;  // obstacle cell: no move, r_outbound per sample (:542-544)
  }
  const int nnz = !valid ? 0 : (window ? __popcll(nz) : 1);
  int incl = nnz;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int t2 = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t2;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  unsigned long long wbase = 0;
  if (lane == 0) {
    wbase = atomicAdd(A.counters + CTR_STAGE, (unsigned long long)total);
    const int64_t wt = (int64_t)T * K.etiles_per_layer + et;
    A.tile_base[wt] = (int64_t)wbase;
    A.tile_len[wt] = total;
  }
  wbase = __shfl_sync(0xffffffffu, wbase, 0);
  if (!valid) return;
  const int64_t grow = ((int64_t)T * nc + cell) * P.na + a;
  A.row_off[grow] = (uint32_t)(incl - nnz);
  A.R[grow] = sumR / P.nrzns;  // compute_mean, src/build_model.cu:567
  if (A.sumR) A.sumR[grow] = sumR;
  unsigned long long off = wbase + (unsigned long long)(incl - nnz);
  if (off + (unsigned long long)nnz > (unsigned long long)A.stage_cap) return;  // host re-runs
  const int32_t next = (int32_t)((int64_t)(T + 1) * nc);
  auto put = [&](int32_t col, uint32_t n) {
    A.stage_col[off] = col;
    if (K.count_bits == 16) reinterpret_cast<uint16_t*>(A.stage_cnt)[off] = (uint16_t)n;
    else reinterpret_cast<uint32_t*>(A.stage_cnt)[off] = n;
    ++off;
  };
  if (!window) {
    put(next + (int32_t)cell, (uint32_t)P.nrzns);
  } else {
    for (uint64_t m = nz; m; m &= m - 1) {
      const int b = __ffsll((long long)m) - 1;
      put(next + (wi0 + (b >> 3)) * g + wj0 + (b & 7), wcol[b * 32]);
    }
  }
}

// the range of one axis' table: a thread per (cell, axis)
template <int NM>
__device__ __forceinline__ void cell_axis(const RankArgs& K, const uint32_t* plan, CellTab& ct, const float4* md, int axis,
                                          int g, const float* stat) {
  const float mean_v = axis ? ct.v1 : ct.u1;
  float centre = mean_v, var = 0.f;
#pragma unroll
  for (int k = 0; k < NM; ++k) {
    const float w = axis ? md[k].z : md[k].x;
    const float2 st = __ldg(reinterpret_cast<const float2*>(stat) + k);
    centre = fmaf(w, st.x, centre);
    var = fmaf(w * w, st.y, var);
  }
  RankRange r;
  if (!rank_range(plan, K.slots_log2, K.groups, axis, axis ? K.sy : K.sx, K.shift, K.a_min[axis], K.a_max[axis], mean_v,
                  centre, var, axis ? ct.i1 : ct.j1, g, &r)) {
    ct.state = 2;  // (both axes' threads write 2)
    return;
  }
  const uint32_t lut = (uint32_t)__cvta_generic_to_shared(plan) + ((uint32_t)r.lut << 2);
  if (axis == 0) {
    ct.bx = ct.bx2 = r.bias;
    ct.qax = r.qa;
    ct.qbx = r.qb;
    ct.lx = lut;
    ct.bax = r.first;
    ct.orgx = r.org;
    ct.nx = r.n;
    ct.kx = r.kind;
  } else {
    ct.by = ct.by2 = r.bias;
    ct.qay = r.qa;
    ct.qby = r.qb;
    ct.ly = lut;
    ct.bay = r.first;
    ct.orgy = r.org;
    ct.ny = r.n;
    ct.ky = r.kind;
  }
}

template <int NM>
__global__ void __launch_bounds__(kThreads, 5) k_build_ranks(BuildArgs A, RankArgs K) {
  extern __shared__ __align__(16) unsigned char smem[];
  const DevProblem& P = A.P;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = P.g, nrz = P.nrzns, ct_log2 = K.cells_log2, CT = 1 << ct_log2;
  const int nc = g * g;  // (states fit 31 bits: validate_problem)
  const int lcap = kListPool >> ct_log2;
  const int cpw_log2 = 5 - A.lanes_log2;
  const int ntiles = CT >> cpw_log2;
  Smem S;
  {
    unsigned char* p = smem;
    auto take = [&](size_t b) {
      unsigned char* q = p;
      p += b;
      return q;
    };
    S.md = reinterpret_cast<float4*>(take(sizeof(float4) * CT * NM));
    S.cells = reinterpret_cast<CellTab*>(take(sizeof(CellTab) * CT));
    S.lut = reinterpret_cast<uint32_t*>(take(sizeof(uint32_t) * rank_plan_words(K.slots_log2)));
    S.tab = reinterpret_cast<float*>(take(sizeof(float) * 32 * 8));
    S.orow = reinterpret_cast<uint32_t*>(take(sizeof(uint32_t) * ((CT * kObsRows + 3) & ~3)));
    S.lcnt = reinterpret_cast<int*>(take(sizeof(int) * kMaxCells));
    S.list = reinterpret_cast<float2*>(take(sizeof(float2) * kListPool));
    S.wcol = reinterpret_cast<uint16_t*>(take(sizeof(uint16_t) * kWarps * 64 * 32));
    S.pool = reinterpret_cast<uint32_t*>(p);
  }
  // the tiles in rounds whose tables fit the pool together (one round, but for
  // cells with wide tables): a tile's round, and the words a round uses
  __shared__ int tile_round[kMaxTiles], round_words[kMaxTiles], rounds;
  for (int i = tid; i < rank_plan_words(K.slots_log2); i += kThreads) S.lut[i] = __ldg(K.plan + i);
  const int tasks_per_layer = (nc + CT - 1) >> ct_log2;
  int tab_late = -1;
  int T = K.t0, chunk = (int)blockIdx.x;
  for (;; chunk += (int)gridDim.x) {
    while (chunk >= tasks_per_layer) {
      chunk -= tasks_per_layer;
      ++T;
    }
    if (T >= K.t1) break;
    const int c0 = chunk << ct_log2;
    __syncthreads();  // the previous task's tables are consumed
    // ---- stage the cells -------------------------------------------------------
    const bool late = T > P.nt - 20;
    if (tab_late != (late ? 1 : 0)) {
      tab_late = late ? 1 : 0;
      if (tid < P.na) {
        // landing rewards after k r_outbound additions, then terminal or late, then
        // the step reward: move() + transition_calc (:343-354, :533)
        const float r_step = step_reward(P, P.ac_speed[tid], 0.f, 0.f);
        float tk = 0;
        for (int k = 0; k < 4; ++k) {
          float r = tk;
          if (late) r += 0.05 * P.r_out;
          r += r_step;
          S.tab[tid * 8 + k] = r;
          float rt = tk;
          rt += P.r_term;
          rt += r_step;
          S.tab[tid * 8 + 4 + k] = rt;
          tk += P.r_out;
        }
      }
    }
    for (int e = tid; e < (NM << ct_log2); e += kThreads) {
      const int k = e >> ct_log2, c = e & (CT - 1);
      float ui = 0.f, vi = 0.f;
      if (k < P.nm && c0 + c < nc) {
        ui = __ldg(A.F.ui + ((int64_t)T * P.nm + k) * nc + c0 + c);
        vi = __ldg(A.F.vi + ((int64_t)T * P.nm + k) * nc + c0 + c);
      }
      S.md[c * NM + k] = make_float4(ui, ui, vi, vi);
    }
    const int i0 = c0 / g, j0 = c0 - i0 * g;
    stage_obstacles(K, T, g, nc, c0, CT, i0, j0, S.orow);
    if (tid < CT) {
      CellTab& ct = S.cells[tid];
      int state = 1, i = i0, j = j0 + tid;
      for (; j >= g; j -= g) ++i;
      ct.i1 = i;
      ct.j1 = j;
      ct.mul = 0u;
      S.lcnt[tid] = 0;
      if (c0 + tid < nc) {
        ct.u1 = __ldg(A.F.u + (int64_t)T * nc + c0 + tid);
        ct.v1 = __ldg(A.F.v + (int64_t)T * nc + c0 + tid);
        if (!is_terminal(P, i, j) && __ldg(A.F.mask + (int64_t)T * nc + c0 + tid) != 1) state = 0;
      }
      ct.state = state;
    }
    __syncthreads();
    // ---- ranges and table space ----------------------------------------------
    if (tid < 2 * CT) {
      CellTab& ct = S.cells[tid >> 1];
      if (ct.state != 1) cell_axis<NM>(K, S.lut, ct, S.md + (tid >> 1) * NM, tid & 1, g, K.ystat + (int64_t)T * 2 * NM);
    }
    __syncthreads();
    if (warp == 0) {
      int words = 0, stride = 0, state = 1;
      CellTab* ct = S.cells + (lane < CT ? lane : 0);
      if (lane < CT) {
        state = ct->state;
        if (state == 0) {
          stride = (ct->nx + 1) | 1;
          words = (ct->ny + 1) * stride;
          if (stride > 255) state = 2;
        }
      }
      int end = words;  // inclusive prefix sum over the cells
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, end, o);
        if (lane >= o) end += v;
      }
      const unsigned out = __ballot_sync(0xffffffffu, state == 2);
      const int first = lane & ~((1 << cpw_log2) - 1), last = first + (1 << cpw_log2) - 1;  // the tile's lanes
      const unsigned mates = (cpw_log2 == 5 ? ~0u : (1u << (1 << cpw_log2)) - 1u) << first;
      const int before = __shfl_sync(0xffffffffu, end - words, first);
      const int need = __shfl_sync(0xffffffffu, end, last & 31) - before;
      // a cell beside one that is left to the general builder is not counted
      // either, nor is a tile larger than the pool (word 0 is the listed samples')
      bool skip = (out & mates) != 0 || need > K.pool_words - 4;
      int round = 0, used = 4, base = 0;
      for (int t = 0; t < ntiles; ++t) {
        const int n = __shfl_sync(0xffffffffu, need, t << cpw_log2);
        const bool sk = __shfl_sync(0xffffffffu, skip, t << cpw_log2);
        if (sk) {
          if (lane == 0) tile_round[t] = 0;
          continue;
        }
        if (used + n > K.pool_words) {
          if (lane == 0) round_words[round] = used;
          ++round;
          used = 4;
        }
        if ((lane >> cpw_log2) == t) base = used + (end - words - before);
        used += n;
        if (lane == 0) tile_round[t] = round;
      }
      if (lane == 0) {
        round_words[round] = used;
        rounds = round + 1;
      }
      if (lane < CT && state != 1) {
        ct->state = skip ? 2 : 0;
        ct->stride = stride;
        ct->base = base;
        ct->cst = (uint32_t)(base - ct->bax - ct->bay * stride);
      }
    }
    __syncthreads();
    for (int round = 0; round < rounds; ++round) {
      // ---- clear the tables ------------------------------------------------------
      {
        const int n4 = (round_words[round] + 3) >> 2;
        for (int i = tid; i < n4; i += kThreads) reinterpret_cast<uint4*>(S.pool)[i] = make_uint4(0u, 0u, 0u, 0u);
        if (tid < CT) {
          CellTab& ct = S.cells[tid];
          ct.mul = ct.state == 0 && tile_round[tid >> cpw_log2] == round ? ((uint32_t)ct.stride << 8) | 1u : 0u;
        }
      }
      __syncthreads();
      // ---- count the realisations ------------------------------------------------
      {
        const float* yt = K.yt + (int64_t)T * NM * K.nrp;
        const uint32_t pool = (uint32_t)__cvta_generic_to_shared(S.pool);
        const int per = CT >> K.nsub_log2;
        for (int it = warp; it < (K.nblocks << K.nsub_log2); it += kWarps) {
          const int blk = it >> K.nsub_log2, lo = (it & ((1 << K.nsub_log2) - 1)) * per;
          const int r0 = blk * 128 + 4 * lane;
          if (blk * 128 + 128 <= nrz)
            count_block<NM, true>(K, yt, r0, nrz, S.md, S.cells, lo, lo + per, pool, S.lcnt, S.list, lcap);
          else
            count_block<NM, false>(K, yt, r0, nrz, S.md, S.cells, lo, lo + per, pool, S.lcnt, S.list, lcap);
        }
      }
      __syncthreads();
      // ---- prefix sums of the tables: along x, then along y -------------------------
      for (int c = warp; c < CT; c += kWarps) {
        const CellTab& ct = S.cells[c];
        if (ct.mul == 0u) continue;
        uint32_t* t = S.pool + ct.base;
        for (int y = 1 + lane; y <= ct.ny; y += 32) {
          uint32_t* p = t + y * ct.stride + 1;
          uint32_t run = 0;
#pragma unroll 4
          for (int x = 0; x < ct.nx; ++x) {
            run += p[x];
            p[x] = run;
          }
        }
        __syncwarp();
        for (int x = 1 + lane; x <= ct.nx; x += 32) {
          uint32_t* p = t + ct.stride + x;
          uint32_t run = 0;
#pragma unroll 4
          for (int y = 0; y < ct.ny; ++y) {
            run += *p;
            *p = run;
            p += ct.stride;
          }
        }
      }
      __syncthreads();
      // ---- the rows ------------------------------------------------------------------
      if (warp < ntiles && tile_round[warp] == round) finish_tile(A, K, S, T, c0, warp, lcap);
      if (round + 1 < rounds) __syncthreads();
    }
  }
}

// Reward sums of the window rows in the order of their samples (K.seq_rewards):
// for spacings other than one the general builder adds a row's rewards sample by
// sample, which for rewards that are no small integers is not the sum of count x
// reward.  Same tasks as k_build_ranks, after it: per chunk of realisations the
// velocities of the CTA's cells, then a lane per row walks them: landing (the
// packed snapping chain of k_build_tiles, its rounding constants scaled by the
// spacing, a power of two, so it rounds as the reference's remainderf snapping),
// reward by the landing's place (and number of clamps) in the cell's table, one
// addition.  Bound by issue: 35 instructions a sample and row of 32 lanes, half of
// them the walk itself.  120x120x40, 8 actions, 500 realisations, radiation
// reward: 58.5 ms a call with the general builder (remainderf twice a sample and
// the full expression again), 5.7 ms now (this kernel 3.3, k_build_ranks 1.4;
// without tables for clamped samples 10.2).
constexpr int kRewardSide = 2 * kRewardR + 1;
constexpr int kRewardPlaces = kRewardSide * kRewardSide;
constexpr int kRewardTable = 3 * kRewardPlaces;  // after 0, 1, 2 domain clamps
constexpr int kRewardChunk = 64;
constexpr int kVelStride = kRewardChunk + 2;
constexpr uint32_t kNoReward = 0xffffffffu;  // table place not taken yet (no reward has these bits)

// Reward of the landing at place `at` around cell (i1, j1) after k clamps (each adds
// r_outbound first, unless an obstacle on the way overrides the reward).  Out of
// line: taken once per place and cell, and inlined into the sample loop it costs
// the loop its registers.
__device__ __noinline__ float reward_at(const BuildArgs& A, int T, float F, const uint32_t* obs, int i1, int j1,
                                        uint32_t at, int k) {
  const DevProblem& P = A.P;
  const int i2 = i1 + (int)(at / kRewardSide) - kRewardR, j2 = j1 + (int)(at % kRewardSide) - kRewardR;
  if (i2 < 0 || i2 >= P.g || j2 < 0 || j2 >= P.g) return 0.f;  // (a row that is left to the general builder)
  if (passes_obstacle(P, A.F.mask, T, obs, i1, j1, i2 - i1, j2 - j1)) return P.r_out;
  return landing_reward(A, T, T > P.nt - 20, P.reward_type == 2 || P.reward_type == 3, F, i1 * P.g + j1, i2, j2, k);
}

template <int NM>
__global__ void __launch_bounds__(kThreads, 6) k_rank_rewards(const __grid_constant__ BuildArgs A,
                                                              const __grid_constant__ RankArgs K) {
  extern __shared__ __align__(16) unsigned char smem[];
  const DevProblem& P = A.P;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = P.g, nrz = P.nrzns, CT = 1 << K.cells_log2, nc = g * g;
  const int cpw_log2 = 5 - A.lanes_log2;
  float2* const vel = reinterpret_cast<float2*>(smem);               // CT x kVelStride
  float2* const md = vel + CT * kVelStride;                          // CT x NM: (ui, vi)
  float2* const uv = md + CT * NM;                                   // CT
  float* const rew = reinterpret_cast<float*>(uv + CT);              // CT x speeds x kRewardTable
  uint32_t* const orow = reinterpret_cast<uint32_t*>(rew + CT * K.nspeeds * kRewardTable);
  const int tasks_per_layer = (nc + CT - 1) >> K.cells_log2;
  int T = K.t0, chunk = (int)blockIdx.x;
  for (;; chunk += (int)gridDim.x) {
    while (chunk >= tasks_per_layer) {
      chunk -= tasks_per_layer;
      ++T;
    }
    if (T >= K.t1) break;
    const int c0 = chunk << K.cells_log2, i0 = c0 / g, j0 = c0 - i0 * g;
    __syncthreads();
    for (int e = tid; e < CT * NM; e += kThreads) {
      const int k = e >> K.cells_log2, c = e & (CT - 1);
      float2 m = make_float2(0.f, 0.f);
      if (k < P.nm && c0 + c < nc) {
        m.x = __ldg(A.F.ui + ((int64_t)T * P.nm + k) * nc + c0 + c);
        m.y = __ldg(A.F.vi + ((int64_t)T * P.nm + k) * nc + c0 + c);
      }
      md[c * NM + k] = m;
    }
    if (tid < CT && c0 + tid < nc)
      uv[tid] = make_float2(__ldg(A.F.u + (int64_t)T * nc + c0 + tid), __ldg(A.F.v + (int64_t)T * nc + c0 + tid));
    stage_obstacles(K, T, g, nc, c0, CT, i0, j0, orow);
    __syncthreads();
    // ---- rewards of unclamped landings around a cell -----------------------------
    // A warp's own cells: the box that nearly every sample lands in is taken at
    // once (lanes over its places), other places at their first use.
    const int per_cell = K.nspeeds * kRewardTable;
    for (int q = 0; q < (1 << cpw_log2); ++q) {
      const int c = (warp << cpw_log2) + q;
      if (c >= CT || c0 + c >= nc) break;  // whole warps
      float* const t = rew + c * per_cell;
      for (int e = lane; e < per_cell; e += 32) t[e] = __uint_as_float(kNoReward);
      int i1 = i0, j1 = j0 + c;
      for (; j1 >= g; j1 -= g) ++i1;
      int lo[2], hi[2];
#pragma unroll
      for (int ax = 0; ax < 2; ++ax) {
        float m = ax ? uv[c].y : uv[c].x, var = 0.f;
#pragma unroll
        for (int k = 0; k < NM; ++k) {
          const float w = ax ? md[c * NM + k].y : md[c * NM + k].x;
          const float2 st = __ldg(reinterpret_cast<const float2*>(K.ystat + (int64_t)T * 2 * NM) + k);
          m = fmaf(w, st.x, m);
          var = fmaf(w * w, st.y, var);
        }
        const float s = (ax ? K.sy : K.sx) * (1.0f / (1 << kRankFrac)), h = 3.0f * sqrtf(var) * fabsf(s);
        lo[ax] = (int)floorf(fminf(fmaxf(K.a_min[ax] + m * s - h + 0.5f, -(float)kRewardR), (float)kRewardR));
        hi[ax] = (int)floorf(fminf(fmaxf(K.a_max[ax] + m * s + h + 0.5f, -(float)kRewardR), (float)kRewardR));
      }
      const int w = hi[0] - lo[0] + 1, places = w * (hi[1] - lo[1] + 1);
      __syncwarp();
      for (int e = lane; e < places * K.nspeeds; e += 32) {
        const int f = e / places, o = e - f * places, di = lo[1] + o / w, dj = lo[0] + o % w;
        const uint32_t at = (uint32_t)((di + kRewardR) * kRewardSide + dj + kRewardR);
        t[f * kRewardTable + at] = reward_at(A, T, P.ac_speed[f * K.nangles], orow + c * kObsRows, i1, j1, at, 0);
      }
    }
    // ---- this lane's row --------------------------------------------------------
    const int tile = warp, cl = (tile << cpw_log2) + (lane >> A.lanes_log2);
    const int a = lane & ((1 << A.lanes_log2) - 1), aa = a < P.na ? a : 0;
    const int cell = c0 + cl;
    int i1 = i0, j1 = j0 + (cl < CT ? cl : 0);
    for (; j1 >= g; j1 -= g) ++i1;
    bool row = cl < CT && cell < nc && a < P.na;
    row = row && !is_terminal(P, i1, j1) && __ldg(A.F.mask + (int64_t)T * nc + cell) != 1;
    const float F = P.ac_speed[aa];
    const float2 FF = make_float2(F, F), csn = make_float2(P.ac_cos[aa], P.ac_sin[aa]), dt2 = make_float2(P.dt, P.dt);
    const float2 xy1 = make_float2(P.xs[row ? j1 : 0], P.ys[row ? g - 1 - i1 : 0]);
    const float2 sgn = make_float2(1.0f, -1.0f), org = make_float2(-P.xs0, P.ysn);
    const float2 half = make_float2(0.5f * P.Dj, 0.5f * P.Di);
    const float2 big = make_float2(12582912.0f * P.Dj, 12582912.0f * P.Di);  // 1.5 * 2^23 cells
    const float2 magic = make_float2(big.x - (float)(j1 - kRewardR) * P.Dj, big.y - (float)(i1 - kRewardR) * P.Di);
    const uint32_t mx = __float_as_uint(big.x), my = __float_as_uint(big.y);
    float* const rt = rew + (row ? cl * per_cell + (aa / K.nangles) * kRewardTable : 0);
    const uint32_t rt_addr = (uint32_t)__cvta_generic_to_shared(rt);
    // cells whose samples can reach the domain's clamps (a landing beyond the
    // tables' reach is not this kernel's)
    const bool edge = __any_sync(0xffffffffu, row && (i1 <= kRewardR + 1 || j1 <= kRewardR + 1 || i1 >= g - 2 - kRewardR ||
                                                      j1 >= g - 2 - kRewardR));
    float sum = 0.f;
    auto place = [&](float2 d) -> uint32_t {
      const float2 t = __fadd2_rd(__fadd2_rd(d, half), magic);
      const uint32_t at = (__float_as_uint(t.y) - my) * (uint32_t)kRewardSide + (__float_as_uint(t.x) - mx);
      return min(at, (uint32_t)(kRewardPlaces - 1));  // (rows that are left to the general builder land anywhere)
    };
    const uint32_t* const obs = orow + cl * kObsRows;
    // the rewards of up to four landings (at: clamps * kRewardPlaces + place), in
    // order, onto the sum
    auto take = [&](const uint32_t (&at)[4], int n) {
      float r[4];
      bool all = true;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        asm volatile("ld.shared.f32 %0, [%1];" : "=f"(r[i]) : "r"(rt_addr + (at[i] << 2)) : "memory");
        all = all && __float_as_uint(r[i]) != kNoReward;
      }
      if (!all) {
        for (int i = 0; i < 4; ++i) {
          if (__float_as_uint(r[i]) != kNoReward) continue;
          r[i] = reward_at(A, T, F, obs, i1, j1, at[i] % kRewardPlaces, (int)(at[i] / kRewardPlaces));
          rt[at[i]] = r[i];  // (lanes that meet here write the same value)
        }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (i < n) sum += r[i];
    };
    const float* yt = K.yt + (int64_t)T * NM * K.nrp;
    for (int base = 0; base < nrz; base += kRewardChunk) {
      const int clen = min(kRewardChunk, nrz - base);
      __syncthreads();  // tables in place; the chunk before is consumed
      {
        const int q = tid & (kRewardChunk - 1);
        float y[NM];
#pragma unroll
        for (int k = 0; k < NM; ++k) y[k] = __ldg(yt + (int64_t)k * K.nrp + base + q);  // (rows are padded)
        for (int c = tid / kRewardChunk; c < CT; c += kThreads / kRewardChunk) {
          float2 s = md[c * NM];
          s = make_float2(s.x * y[0], s.y * y[0]);
#pragma unroll
          for (int k = 1; k < NM; ++k) s = __ffma2_rn(md[c * NM + k], make_float2(y[k], y[k]), s);
          vel[c * kVelStride + q] = make_float2(uv[c].x + s.x, uv[c].y + s.y);
        }
      }
      __syncthreads();
      if (row) {
        const float2* v = vel + cl * kVelStride;
        for (int q = 0; q < clen; q += 4) {  // (a velocity row holds two more than a chunk, and clen's rest is not added)
          const float4 w0 = *reinterpret_cast<const float4*>(v + q), w1 = *reinterpret_cast<const float4*>(v + q + 2);
          const float2 vv[4] = {make_float2(w0.x, w0.y), make_float2(w0.z, w0.w), make_float2(w1.x, w1.y),
                                make_float2(w1.z, w1.w)};
          uint32_t at[4];
          if (!edge) {
#pragma unroll
            for (int i = 0; i < 4; ++i) at[i] = place(__ffma2_rn(advect2(FF, csn, vv[i], dt2, xy1), sgn, org));
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float2 xy = advect2(FF, csn, vv[i], dt2, xy1);
              const float2 d = __ffma2_rn(xy, sgn, org);
              at[i] = place(make_float2(fminf(fmaxf(d.x, 0.0f), P.axmax), fminf(fmaxf(d.y, 0.0f), P.aymax)));
              at[i] += (xy.x > P.xsn || xy.x < P.xs0) ? kRewardPlaces : 0;
              at[i] += (xy.y > P.ysn || xy.y < P.ys0) ? kRewardPlaces : 0;
            }
          }
          take(at, clen - q);
        }
      }
    }
    if (row) {
      const int64_t grow = ((int64_t)T * nc + cell) * P.na + a;
      A.R[grow] = sum / P.nrzns;
      if (A.sumR) A.sumR[grow] = sum;
    }
  }
}

// Per layer [t0, t1): the coefficients mode-major with rows padded to nrp (so a
// lane reads four realisations at once), their mean and variance per mode (the
// tables' ranges), and a bit per cell for the obstacles at T or T + 1.
// blockIdx.y == 0: coefficients; others: 32 grid rows each.
template <int NM>
__global__ void __launch_bounds__(1024) k_rank_prepare(DevProblem P, DevFields F, RankArgs K, float* yt, float* ystat,
                                                       uint32_t* obits) {
  const int T = K.t0 + blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (blockIdx.y == 0) {
    __shared__ float red[32][2 * NM];
    const float* y = F.Y + (int64_t)T * P.nrzns * P.nm;
    float* o = yt + (int64_t)T * NM * K.nrp;
    float s[NM], q[NM];
#pragma unroll
    for (int k = 0; k < NM; ++k) s[k] = q[k] = 0.f;
    for (int r = tid; r < K.nrp; r += 1024) {
#pragma unroll
      for (int k = 0; k < NM; ++k) {
        const float v = (r < P.nrzns && k < P.nm) ? __ldg(y + (int64_t)r * P.nm + k) : 0.f;
        o[(int64_t)k * K.nrp + r] = v;
        s[k] += v;
        q[k] = fmaf(v, v, q[k]);
      }
    }
#pragma unroll
    for (int k = 0; k < NM; ++k) {
      for (int w = 16; w > 0; w >>= 1) {
        s[k] += __shfl_xor_sync(0xffffffffu, s[k], w);
        q[k] += __shfl_xor_sync(0xffffffffu, q[k], w);
      }
      if (lane == 0) {
        red[warp][2 * k] = s[k];
        red[warp][2 * k + 1] = q[k];
      }
    }
    __syncthreads();
    if (tid < NM) {
      float a = 0.f, b = 0.f;
      for (int w = 0; w < 32; ++w) {
        a += red[w][2 * tid];
        b += red[w][2 * tid + 1];
      }
      const float m = a / (float)P.nrzns;
      ystat[(int64_t)T * 2 * NM + 2 * tid] = m;
      ystat[(int64_t)T * 2 * NM + 2 * tid + 1] = fmaxf(b / (float)P.nrzns - m * m, 0.f);
    }
    return;
  }
  const int i = ((int)blockIdx.y - 1) * 32 + warp;
  if (i >= P.g) return;
  const int64_t nc = (int64_t)P.g * P.g;
  const int32_t* m0 = F.mask + (int64_t)T * nc + (int64_t)i * P.g;
  for (int w = 0; w < K.owords; ++w) {
    const int j = w * 32 + lane;
    const bool ob = j < P.g && (__ldg(m0 + j) == 1 || __ldg(m0 + nc + j) == 1);
    const uint32_t bits = __ballot_sync(0xffffffffu, ob);
    if (lane == 0) obits[((int64_t)T * P.g + i) * K.owords + w] = bits;
  }
}

std::mutex g_cap_mu;
bool g_cap_set[64][8] = {};

// f(integral constant of the padded mode count)
template <typename F>
cudaError_t dispatch_nm(int nmp, F&& f) {
  switch (nmp) {
    case 2: return f(std::integral_constant<int, 2>{});
    case 4: return f(std::integral_constant<int, 4>{});
    case 6: return f(std::integral_constant<int, 6>{});
    case 8: return f(std::integral_constant<int, 8>{});
    case 10: return f(std::integral_constant<int, 10>{});
  }
  return cudaErrorInvalidValue;
}

// Shared memory of a CTA where four or five of them share an SM.  Five wherever
// the pool then still holds the widest tables of a tile of inner cells (ranges
// of 2 x kRankMaxHalfRange cells), else its cells would go to the general
// builder: 200x200x30, 10 modes, 5000 realisations 14.5 -> 13.8 ms; 8 modes, 2000
// 7.54 -> 7.30, 1000 5.73 -> 5.77; 8 actions, 4 modes, 1280 3.83 -> 3.56; six
// CTAs 14.0, 7.70, 6.30, 3.50.
constexpr size_t kSmem4 = 55 * 1024, kSmem5 = 44 * 1024;

// k_rank_rewards: two CTAs an SM at least.  (Few actions a cell, or several speeds,
// make the tables of the 32 or 16 cells of a CTA need
// more than 48 KB: with the general builder 90x90x40, 300 realisations, 4 actions
// took 14.8 ms, here 1.9; 2 speeds x 4 headings 21.4 -> 2.2; 4 x 4 33.1 -> 3.7.)
constexpr size_t kRewardSmem = 110 * 1024;

size_t reward_smem_bytes(const RankArgs& K, int nmp) {
  const size_t ct = (size_t)1 << K.cells_log2;
  return ct * (sizeof(float2) * (kVelStride + nmp + 1) + sizeof(float) * K.nspeeds * kRewardTable +
               sizeof(uint32_t) * kObsRows);
}

}  // namespace

int rank_padded_modes(int nm) { return nm <= 2 ? 2 : (nm + 1) & ~1; }

bool rank_shape(int nm, int slots_log2, int lanes_log2, int nrzns, RankArgs* K) {
  if (nm > 10) return false;
  const int nmp = rank_padded_modes(nm);
  K->slots_log2 = slots_log2;
  // kMaxTiles emission tiles of 32 / P cells (P action lanes)
  K->cells_log2 = std::min(5, 7 - lanes_log2);
  const int cells = 1 << K->cells_log2;
  const size_t fixed = smem_fixed_bytes(slots_log2, nmp, cells);
  if (fixed + 16 * 1024 > kSmem4) return false;
  const float width = 2.0f * kRankMaxHalfRange;
  const int nx = (int)(width * K->groups[RANK_X]) + 3, ny = (int)(width * K->groups[RANK_Y]) + 3;
  const size_t widest = sizeof(uint32_t) * (((size_t)32 >> lanes_log2) * ((nx + 1) | 1) * (ny + 1) + 8);
  K->ctas_per_sm = fixed + widest <= kSmem5 ? 5 : 4;
  K->pool_words = (int)(((K->ctas_per_sm == 5 ? kSmem5 : kSmem4) - fixed) / 4) & ~3;
  if (K->seq_rewards && reward_smem_bytes(*K, nmp) > kRewardSmem) return false;
  K->nrp = (nrzns + 127) / 128 * 128;
  K->nblocks = K->nrp / 128;
  // subsets of the cells: a warp's work item is 128 realisations x one subset.
  // Fewer subsets load the coefficients less often (about a cell's worth of
  // work), more of them spread few realisation blocks over the warps.
  double best = 1e30;
  for (int l = 0; l <= 2; ++l) {
    const double cost = (((K->nblocks << l) + kWarps - 1) / kWarps) * ((cells >> l) + 1.0);
    if (cost < best) {
      best = cost;
      K->nsub_log2 = l;
    }
  }
  return true;
}

cudaError_t launch_rank_prepare(const DevProblem& P, const DevFields& F, const RankArgs& K, cudaStream_t st) {
  const dim3 grid((unsigned)(K.t1 - K.t0), (unsigned)(1 + (P.g + 31) / 32));
  return dispatch_nm(rank_padded_modes(P.nm), [&](auto nm) -> cudaError_t {
    k_rank_prepare<decltype(nm)::value><<<grid, 1024, 0, st>>>(P, F, K, const_cast<float*>(K.yt),
                                                                const_cast<float*>(K.ystat),
                                                                const_cast<uint32_t*>(K.obits));
    return cudaGetLastError();
  });
}

cudaError_t launch_build_ranks(const BuildArgs& A, const RankArgs& K, cudaStream_t st) {
  const int nmp = rank_padded_modes(A.P.nm);
  const size_t sm = smem_fixed_bytes(K.slots_log2, nmp, 1 << K.cells_log2) + 4 * (size_t)K.pool_words;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  const int64_t nc = (int64_t)A.P.g * A.P.g;
  const int64_t tasks = (int64_t)(K.t1 - K.t0) * ((nc + (1 << K.cells_log2) - 1) >> K.cells_log2);
  const unsigned grid = (unsigned)std::min<int64_t>(tasks, K.ctas_per_sm * (int64_t)sms);
  if (grid == 0) return cudaSuccess;
  return dispatch_nm(nmp, [&](auto nm) -> cudaError_t {
    auto kern = k_build_ranks<decltype(nm)::value>;
    {
      std::lock_guard<std::mutex> lk(g_cap_mu);
      if (dev < 0 || dev >= 64 || !g_cap_set[dev][nmp / 2]) {
        cudaError_t e2 = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem4);
        if (e2 != cudaSuccess) return e2;
        if (dev >= 0 && dev < 64) g_cap_set[dev][nmp / 2] = true;
      }
    }
    kern<<<grid, kThreads, sm, st>>>(A, K);
    cudaError_t e2 = cudaGetLastError();
    if (e2 != cudaSuccess || !K.seq_rewards) return e2;
    const size_t rb = reward_smem_bytes(K, nmp);  // (at most kRewardSmem: rank_shape)
    // as many CTAs as are resident: each takes the same number of tasks
    int per_sm = 0;
    e2 = cudaFuncSetAttribute(k_rank_rewards<decltype(nm)::value>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)kRewardSmem);
    if (e2 != cudaSuccess) return e2;
    e2 = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_rank_rewards<decltype(nm)::value>, kThreads, rb);
    if (e2 != cudaSuccess) return e2;
    k_rank_rewards<decltype(nm)::value>
        <<<(unsigned)std::min<int64_t>(tasks, std::max(per_sm, 1) * (int64_t)sms), kThreads, rb, st>>>(A, K);
    return cudaGetLastError();
  });
}

}  // namespace e2e
