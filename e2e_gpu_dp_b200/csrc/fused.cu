// Build and solve in one backward pass, never storing the transition model.
//
// The reference builds every (t, a) block of the model (src/build_model.cu:
// 696-892), writes it to disk, and spvi_2 reads it back and iterates
// (src/spvi_2.cu:650-726).  Transitions only go from layer t to t+1
// (src/build_model.cu:635) and the last layer has no rows (:1173-1176), so the
// values of layer t are final as soon as layer t+1's are: the layered schedule
// reaches the Jacobi fixed point in one pass.  Here the builder runs over a few
// layers at a time, from the last, into a staging area of bounded size, and
// k_backup_layers backs the rows up from there, layer by layer.  (The pass
// before this one backed rows up in the builder's epilogue, each tile waiting
// for the rows of the layer after its own; that tied it to the counting
// builder: 100x100x60, 1000 realisations 13.0 ms, now 3.9 ms.)
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>

#include "e2e_dp.h"
#include "grid_sync.cuh"
#include "internal.h"
#include "kernels.h"

using namespace e2e;

#define CK(call)                                        \
  do {                                                  \
    cudaError_t _e = (call);                            \
    if (_e != cudaSuccess) return cuda_fail(_e, #call); \
  } while (0)

namespace {

constexpr int kThreads = 256;
// bytes of a block of layers' staging (tests: E2E_TEST_STAGE_BYTES)
size_t stage_budget() {
  const char* v = std::getenv("E2E_TEST_STAGE_BYTES");
  return v ? (size_t)std::strtoull(v, nullptr, 10) : size_t(256) << 20;
}

struct BackupArgs {
  int t0, t1, na, lanes_log2, cells_log2, nrzns;  // 1 << cells_log2 cells per emission tile
  int nc;
  int64_t etiles_per_layer;
  const uint32_t* row_off;  // these four and stage_* hold layers [t0, t1): index from layer t0
  const int64_t* tile_base;
  const int32_t* tile_len;
  const float* R;
  const int32_t* stage_col;
  const uint16_t* stage_cnt;
  float* V;
  int32_t* pi;
  unsigned int* sync;
  WaitBound wb;
};

// Backups of the staged rows of layers t1-1 down to t0, one cooperative launch:
// P lanes a cell (P = next power of two >= actions).  Q = R + (sum over the
// row's entries in column order of fma(count, V[next], acc)) / nrzns, the
// arithmetic of the sweeps over a stored model (solver_do_backup,
// src/spvi_2.cu:174-260); the first maximum over the cell's lanes
// (select_best_action, :93-122: strict '>', NaN never taken, values at or below
// -1e6 give -1e6 / -1).  Bound by the chain of a layer: the grid barrier (its waits
// are bounded as the sweeps' are), the gathers, the sums.  What does not depend on
// values, a lane's first row with four of its entries, is read before the wait, and
// four gathers are in flight together: 100x100x60, 16 actions, 1000 realisations 3.93 ->
// 3.78 ms a pass, 50x50x30 0.32 -> 0.29.
struct StagedRow {
  bool valid;
  int cell;
  float R;
  int64_t e, end;
  int32_t col[4];
  uint16_t cnt[4];
};

__device__ __forceinline__ void load_entries(const BackupArgs& A, StagedRow& r) {
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    r.col[b] = r.e + b < r.end ? __ldcs(A.stage_col + r.e + b) : 0;
    r.cnt[b] = r.e + b < r.end ? __ldcs(A.stage_cnt + r.e + b) : (uint16_t)0;
  }
}

__device__ __forceinline__ void load_row(const BackupArgs& A, int64_t layer, int64_t k, int64_t n, int a, StagedRow& r) {
  r.cell = (int)(k >> A.lanes_log2);
  r.valid = k < n && a < A.na;
  r.R = 0.f;
  r.e = r.end = 0;
  if (r.valid) {
    const int64_t row = (layer * A.nc + r.cell) * A.na + a;
    const int64_t tile = layer * A.etiles_per_layer + (r.cell >> A.cells_log2);
    // the tile's last row ends with the tile
    const bool last = a == A.na - 1 && (((r.cell + 1) & ((1 << A.cells_log2) - 1)) == 0 || r.cell + 1 == A.nc);
    const uint32_t off = __ldg(A.row_off + row);
    const uint32_t end = last ? (uint32_t)__ldg(A.tile_len + tile) : __ldg(A.row_off + row + 1);
    const int64_t base = __ldg(A.tile_base + tile);
    r.R = __ldg(A.R + row);
    r.e = base + off;
    r.end = base + end;
  }
  load_entries(A, r);
}

__global__ void __launch_bounds__(kThreads) k_backup_layers(BackupArgs A) {
  const int64_t n = (int64_t)A.nc << A.lanes_log2, stride = (int64_t)gridDim.x * kThreads;
  const int64_t first = (int64_t)blockIdx.x * kThreads;
  const int a = threadIdx.x & ((1 << A.lanes_log2) - 1);
  unsigned int gen = 0;
  const float* Vn = A.V;  // written by other CTAs of this launch: plain loads, ordered by the barrier
  for (int t = A.t1 - 1; t >= A.t0; --t) {
    StagedRow r;
    load_row(A, t - A.t0, first + threadIdx.x, n, a, r);
    if (gen && !grid_wait(A.sync, gen * gridDim.x, A.wb)) return;
    for (int64_t k0 = first; k0 < n; k0 += stride) {  // whole warps
      if (k0 != first) load_row(A, t - A.t0, k0 + threadIdx.x, n, a, r);
      float q = -INFINITY;
      if (r.valid) {
        float acc = 0.f;
        while (r.e < r.end) {
          float v[4];
#pragma unroll
          for (int b = 0; b < 4; ++b) v[b] = r.e + b < r.end ? Vn[r.col[b]] : 0.f;
#pragma unroll
          for (int b = 0; b < 4; ++b)
            if (r.e + b < r.end) acc = fmaf((float)r.cnt[b], v[b], acc);
          r.e += 4;
          if (r.e < r.end) load_entries(A, r);
        }
        q = finish_row(r.R, acc, 0.f, A.nrzns, true);
        if (isnan(q)) q = -INFINITY;
      }
      int ba = a;
      for (int o = (1 << A.lanes_log2) >> 1; o > 0; o >>= 1) {
        const float oq = __shfl_xor_sync(0xffffffffu, q, o);
        const int oa = __shfl_xor_sync(0xffffffffu, ba, o);
        if (oq > q || (oq == q && oa < ba)) {
          q = oq;
          ba = oa;
        }
      }
      if (r.valid && a == 0) {
        const bool ok = q > -1e6f;
        A.V[(int64_t)t * A.nc + r.cell] = ok ? q : -1e6f;
        A.pi[(int64_t)t * A.nc + r.cell] = ok ? ba : -1;
      }
    }
    if (t > A.t0) {
      ++gen;
      grid_arrive(A.sync);
    }
  }
}

}  // namespace

extern "C" e2e_status e2e_build_solve(const e2e_problem* p, const e2e_fields* f, int where,
                                      int32_t* policy_out, float* value_out, int out_where,
                                      e2e_fused_stats* stats, void* stream) {
  e2e_status vs = validate_problem(p);
  if (vs != E2E_OK) return vs;
  if (!f || !f->u || !f->v || !f->yi || !f->s || !f->mask || (p->nmodes > 0 && (!f->ui || !f->vi)))
    return fail(E2E_ERR_INVALID, "null field pointer");
  if (where != E2E_HOST && where != E2E_DEVICE) return fail(E2E_ERR_INVALID, "bad fields_where");
  if (out_where != E2E_HOST && out_where != E2E_DEVICE) return fail(E2E_ERR_INVALID, "bad out_where");
  cudaStream_t st = (cudaStream_t)stream;

  BuildPlan pl;
  e2e_status s = plan_build(p, 16, 0, &pl);
  if (s != E2E_OK) return s;
  SettleOnExit settle(st);
  DeviceScratch scratch(st);
  FieldsOnDevice fd;
  s = fields_to_device(p, f, where, st, &fd, &scratch);
  if (s != E2E_OK) return s;
  DevProblem D;
  s = make_dev_problem(p, st, &D, &scratch);
  if (s != E2E_OK) return s;
  const int64_t ns = pl.ns, nc = pl.ncells;
  float* dV = nullptr;
  int32_t* dpi = nullptr;
  if (out_where == E2E_DEVICE && value_out) {
    dV = value_out;
  } else {
    CK(dalloc((void**)&dV, sizeof(float) * (size_t)ns, st));
    scratch.add(dV);
  }
  if (out_where == E2E_DEVICE && policy_out) {
    dpi = policy_out;
  } else {
    CK(dalloc((void**)&dpi, sizeof(int32_t) * (size_t)ns, st));
    scratch.add(dpi);
  }
  // the last layer has no rows: value 0 and action 0 (the first of equal
  // zero Q values), as the sweeps give it
  const int64_t last = (int64_t)(p->nt - 1) * nc;
  CK(cudaMemsetAsync(dV + last, 0, sizeof(float) * (size_t)nc, st));
  CK(cudaMemsetAsync(dpi + last, 0, sizeof(int32_t) * (size_t)nc, st));

  // blocks of layers, of about equal size within the staging budget, or of fewer layers
  // where memory for that is missing
  LayerBuild L(st);
  s = layer_build_buffers(p, pl, &L);
  if (s != E2E_OK) return s;
  BuildStaging buf(st);
  struct {
    uint32_t* row_off;
    float* R;
    int64_t* tile_base;
    int32_t* tile_len;
  } blk;
  const int layers = p->nt - 1;
  const int64_t rows = nc * pl.na;
  const size_t per_layer = (size_t)rows * (sizeof(uint32_t) + sizeof(float) + 4 * 6);
  int64_t pool_units = pl.pool_units, cap = 0, least = 0;
  int most = (int)std::max<size_t>(1, std::min<size_t>((size_t)layers, stage_budget() / per_layer));
  int nblocks = 0, bl = 0;
  for (;;) {
    nblocks = (layers + most - 1) / most;
    bl = (layers + nblocks - 1) / nblocks;
    cap = least = rows * bl * 4 + 4096;
    const size_t n = (size_t)rows * bl, nt = (size_t)pl.etiles_per_layer * bl;
    char* at = nullptr;
    cudaError_t e = dalloc((void**)&at, sizeof(int64_t) * nt + sizeof(int32_t) * nt + (sizeof(uint32_t) + sizeof(float)) * n, st);
    if (e == cudaSuccess) {
      e = buf.provide(&cap, least, sizeof(uint16_t), pool_units, p->neighb_gsize, nullptr);
      if (e == cudaSuccess) {
        scratch.add(at);
        blk.tile_base = reinterpret_cast<int64_t*>(at);
        blk.row_off = reinterpret_cast<uint32_t*>(blk.tile_base + nt);
        blk.R = reinterpret_cast<float*>(blk.row_off + n);
        blk.tile_len = reinterpret_cast<int32_t*>(blk.R + n);
        break;
      }
      dfree(at, st);
    }
    if (e != cudaErrorMemoryAllocation || (most == 1 && !L.ranked)) return cuda_fail(e, "buffers of a block of layers");
    cudaGetLastError();
    if (most > 1) most /= 2;
    else L.drop();
  }
  // per block: the builder's counters, then the barrier words of its backup
  unsigned long long* ctr = nullptr;
  const size_t ctr_words = CTR_COUNT + 1;
  CK(dalloc((void**)&ctr, sizeof(unsigned long long) * ctr_words * nblocks, st));
  scratch.add(ctr);
  CK(cudaMemsetAsync(ctr, 0, sizeof(unsigned long long) * ctr_words * nblocks, st));
  const int mm = p->neighb_gsize * p->neighb_gsize;

  int dev = 0, sms = 0, per_sm = 0;
  CK(cudaGetDevice(&dev));
  CK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_backup_layers, kThreads, 0));
  if (per_sm < 1) return fail(E2E_ERR_DEVICE, "the backup kernel does not fit the device");

  cudaEvent_t ev[2];
  for (int k = 0; k < 2; ++k) CK(cudaEventCreate(&ev[k]));
  struct EvFree {
    cudaEvent_t* e;
    ~EvFree() { for (int k = 0; k < 2; ++k) cudaEventDestroy(e[k]); }
  } evfree{ev};
  CK(cudaEventRecord(ev[0], st));
  int launches = 0;
  unsigned long long sum[CTR_COUNT] = {}, *bc = ctr;
  for (int b = 0, t1 = layers; t1 > 0; ++b, t1 = std::max(0, t1 - bl)) {
    const int t0 = std::max(0, t1 - bl);
    bc = ctr + ctr_words * b;
    unsigned long long hc[CTR_COUNT + 1];
    for (int attempt = 0;; ++attempt) {
      CK(buf.provide(&cap, least, sizeof(uint16_t), pool_units, p->neighb_gsize, &L));
      if (attempt) CK(cudaMemsetAsync(bc, 0, sizeof(unsigned long long) * CTR_COUNT, st));
      BuildArgs A{};
      A.P = D;
      A.F = fd.F;
      A.t0 = t0;
      A.t1 = t1;
      A.etiles_per_layer = pl.etiles_per_layer;
      A.tiles_per_layer = (int)pl.tiles_per_layer;
      A.rc = pl.rc;
      A.ybufs = pl.ybufs;
      A.lanes_log2 = build_lanes_log2(pl.na);
      A.counters = bc;
      A.pool = static_cast<uint32_t*>(buf.pool);
      A.pool_units = pool_units;
      A.stage_col = static_cast<int32_t*>(buf.col);
      A.stage_cnt = buf.cnt;
      A.stage_cap = cap;
      // the builder indexes by layer: the block's first one at the buffers' start
      A.row_off = blk.row_off - rows * t0;
      A.R = blk.R - rows * t0;
      A.tile_base = blk.tile_base - pl.etiles_per_layer * t0;
      A.tile_len = blk.tile_len - pl.etiles_per_layer * t0;
      CK(launch_layers(A, pl, L, t0, t1, st));
      CK(launch_leftover(A, pl, L, t0, t1, st));
      ++launches;
      // sleep through a long block, then read its counters and the error word of the
      // backup before it
      if (pl.long_build) CK(sleep_sync(st));
      CK(cudaMemcpyAsync(hc, b ? bc - 1 : bc, sizeof(unsigned long long) * (CTR_COUNT + (b ? 1 : 0)),
                         cudaMemcpyDeviceToHost, st));
      CK(cudaStreamSynchronize(st));
      if (b) {
        if (hc[0] >> 32) return fail(E2E_ERR_DEVICE, "build+solve: a wait for a layer's completion ran out of its bound");
        std::copy(hc + 1, hc + 1 + CTR_COUNT, hc);
      }
      bool again = false;
      int64_t lost = 0;  // rows without a histogram
      if (hc[CTR_FLAGS] & FLAG_POOL_EXHAUSTED) {
        buf.drop_pool();
        lost = (int64_t)hc[CTR_POOL] - pool_units;
        pool_units = (int64_t)hc[CTR_POOL];
        if ((double)pool_units * mm * 4 > 32.0 * (1ull << 30))
          return fail(E2E_ERR_UNSUPPORTED, "transition spread too wide: dense-histogram pool above 32 GiB");
        again = true;
      }
      const int64_t staged = (int64_t)hc[CTR_STAGE];
      if (staged + lost * BuildStaging::kLostRowEntries > cap) {
        buf.drop_stage();
        least = std::max(cap, staged + staged / 8);  // (later blocks differ a little)
        cap = std::max(least, staged + lost * BuildStaging::kLostRowEntries);
        again = true;
      }
      if (!again) break;
      if (attempt == 2) return fail(E2E_ERR_DEVICE, "build did not settle after re-runs");
    }
    for (int k = 0; k < CTR_COUNT; ++k) sum[k] += hc[k];
    BackupArgs B{};
    B.t0 = t0;
    B.t1 = t1;
    B.na = pl.na;
    B.lanes_log2 = build_lanes_log2(pl.na);
    B.cells_log2 = 5 - B.lanes_log2;
    B.nrzns = p->nrzns;
    B.nc = (int)nc;
    B.etiles_per_layer = pl.etiles_per_layer;
    B.row_off = blk.row_off;
    B.tile_base = blk.tile_base;
    B.tile_len = blk.tile_len;
    B.R = blk.R;
    B.stage_col = static_cast<const int32_t*>(buf.col);
    B.stage_cnt = static_cast<const uint16_t*>(buf.cnt);
    B.V = dV;
    B.pi = dpi;
    B.sync = reinterpret_cast<unsigned int*>(bc + CTR_COUNT);
    B.wb = wait_bound_from_env();
    const int64_t need = ((nc << B.lanes_log2) + kThreads - 1) / kThreads;
    const unsigned grid = (unsigned)std::min<int64_t>(need, (int64_t)per_sm * sms);
    void* args[] = {&B};
    CK(cudaLaunchCooperativeKernel((const void*)k_backup_layers, dim3(grid), dim3(kThreads), args, 0, st));
    ++launches;
  }
  CK(cudaEventRecord(ev[1], st));
  if (out_where == E2E_HOST) {
    if (value_out) CK(cudaMemcpyAsync(value_out, dV, sizeof(float) * ns, cudaMemcpyDeviceToHost, st));
    if (policy_out) CK(cudaMemcpyAsync(policy_out, dpi, sizeof(int32_t) * ns, cudaMemcpyDeviceToHost, st));
  }
  unsigned long long err = 0;
  CK(cudaMemcpyAsync(&err, bc + CTR_COUNT, sizeof(err), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  settle.done = true;
  if (err >> 32) return fail(E2E_ERR_DEVICE, "build+solve: a wait for a layer's completion ran out of its bound");
  float ms = 0.f;
  CK(cudaEventElapsedTime(&ms, ev[0], ev[1]));
  if (stats) {
    stats->seconds = ms * 1e-3;
    stats->n_rows = pl.n_rows;
    stats->nnz = (int64_t)sum[CTR_STAGE];
    stats->dropped = sum[CTR_DROPPED];
    stats->misbinned = sum[CTR_MISBIN];
    stats->overflow_rows = sum[CTR_OVERFLOW_ROWS];
    stats->launches = launches;
    stats->general_tiles = (int32_t)std::min<int64_t>(L.ranked ? (int64_t)sum[CTR_DEFERRED] : pl.n_tiles, INT32_MAX);
    stats->h2d_bytes = (int64_t)fd.h2d_bytes;
  }
  return E2E_OK;
}
