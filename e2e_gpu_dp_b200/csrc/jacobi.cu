// Jacobi value iteration of a time-layered model, all sweeps of a layer at once.
//
// The reference sweeps the whole model until the sup-norm of an update falls
// below the threshold (solver_spvi_solve, src/spvi_2.cu:650-726): about as many
// sweeps as layers, each streaming the model from HBM.  Transitions lead from
// layer t to t+1 only, so sweep j of layer t needs sweep j-1 of layer t+1 and
// nothing else, and from sweep (layers - t) on a layer repeats itself.  Here a
// layer's rows are read once and take every sweep j = 1 .. layers - t together:
// a warp holds a state, its lanes the sweeps, and the history of layer t+1 is
// stored state by state with the sweeps side by side, so an entry is one
// coalesced read and a multiply-add per 32 sweeps.  Each sweep's sum, division
// and argmax are those of the sweep kernels, in their order: values, policies,
// the FP64 residual of every sweep and the sweep that ends the iteration are the
// same.  Afterwards V of the last but one sweep is gathered from the history and
// one ordinary sweep gives the result.
//
// The model is read once instead of once per sweep (sweeps: 0.35 ms each at the
// copy bandwidth).  What bounds it is issue: the reads and multiply-adds, the
// exact quotients, the set-up of a state.  200x200x120, 500 realisations: 120 sweeps
// 42.9 -> 8.8 ms; 137x137x53, 12 actions 4.1 -> 1.7 ms; 50x50x30 0.84 -> 0.34 ms.
#include <math.h>

#include <algorithm>
#include <type_traits>

#include "internal.h"

namespace e2e {

namespace {

constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;
constexpr int kStage = 128;  // entries of a state staged at a time

// (out of line: inlined, the division is evaluated beside the correction every time)
__device__ __noinline__ float divide(float a, float b) { return a / b; }

// acc / n for a count n: the correctly rounded quotient, as the division
// operator gives it, by Markstein's correction of acc * (1/n) (P. W. Markstein,
// IBM J. Res. Dev. 34(1), 1990: with the correctly rounded reciprocal, a quotient
// within an ulp plus its exact remainder times the reciprocal rounds correctly;
// the first correction brings it within an ulp).  For sums that are 0 or far from
// under- and overflow (see kPlainMin).
__device__ __forceinline__ float quotient(float acc, float n, float rn) {
  float q = acc * rn;
  q = fmaf(fmaf(-q, n, acc), rn, q);
  return fmaf(fmaf(-q, n, acc), rn, q);
}

// Values that are 0 or between these are `plain`: a sum of counts times such
// values, whatever cancels, is 0 or between 1e-18 and 1e30.  A layer with other
// values (its flag is set) is divided with the operator itself.
constexpr float kPlainMin = 1e-10f, kPlainMax = 1e25f;

// The rows of a state that are staged in ent[0 .. cnt): a batch of entries at a
// time, every read of the history, then the multiply-adds in entry order; bit k of
// ends says that entry k is its row's last, whose Q is then formed with the next
// of the rewards r.  (One pass over the entries whatever the rows' lengths: with a
// switch on each row's length 200x200x120 took 11.3 ms, now 8.8; batches of 8 for all
// counts of sweeps 10.0, of 4 9.0.)
template <int NB, bool PLAIN>
__device__ __forceinline__ void take_rows(const uint2* ent, int cnt, const unsigned (&ends)[kStage / 32], const char* hn,
                                          bool counts, float n, float rn, const float*& r, float (&acc)[NB],
                                          float (&bq)[NB]) {
  constexpr int B = NB > 2 ? 4 : 8;
#pragma unroll
  for (int w = 0; w < kStage / 32; ++w) {
    if (32 * w >= cnt) break;
    unsigned m = ends[w];
    const uint2* p = ent + 32 * w;
    const int todo = min(cnt - 32 * w, 32);
    for (int k = 0; k < todo; k += B, p += B, m >>= B) {
      float v[B][NB], f[B];
#pragma unroll
      for (int i = 0; i < B; ++i) {
        const uint2 x = p[i];
        f[i] = __uint_as_float(x.y);
#pragma unroll
        for (int b = 0; b < NB; ++b) v[i][b] = __ldg(reinterpret_cast<const float*>(hn + (size_t)x.x) + 32 * b);
      }
#pragma unroll
      for (int i = 0; i < B; ++i) {
#pragma unroll
        for (int b = 0; b < NB; ++b) acc[b] = fmaf(f[i], v[i][b], acc[b]);
        if (m >> i & 1u) {
          const float rr = *r++;
#pragma unroll
          for (int b = 0; b < NB; ++b) {
            const float q = PLAIN ? (counts ? quotient(acc[b], n, rn) : acc[b]) : divide(acc[b], n);
            bq[b] = fmaxf(bq[b], rr + q);  // (NaN is never taken)
            acc[b] = 0.f;
          }
        }
      }
    }
  }
}

// Sweeps j0 + 1 .. j0 + 32 NB (up to J) of the layer of states [s0, s0 + nc).
// Hn: history of the next layer, row stride sn, entry j = V after j sweeps (null
// for states without rows); H: this layer's, stride s.
template <typename PtrT, typename CntT, int NB>
__global__ void __launch_bounds__(kThreads) k_jacobi_layer(ViModel M, int64_t s0, int nc, int j0, int J, const float* Hn,
                                                           uint32_t sn, float* H, int s, unsigned long long* resid,
                                                           const unsigned int* odd_next, unsigned int* odd) {
  __shared__ double red[kWarps][NB * 32];
  // entries of a warp's state: (offset of the next state's history, weight)
  __shared__ __align__(16) uint2 ents[kWarps][kStage];
  __shared__ float rews[kWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const bool counts = M.count_type != VAL_F32;
  const float n = (float)M.nrzns, rn = 1.0f / n;
  const int64_t next0 = s0 + nc;
  const PtrT* __restrict__ rp = reinterpret_cast<const PtrT*>(M.row_ptr);
  const CntT* __restrict__ cnt = reinterpret_cast<const CntT*>(M.cnt);
  const char* const hn = reinterpret_cast<const char*>(Hn + j0 + lane);
  const bool plain = !counts || !odd_next || *odd_next == 0u;
  bool other = false;
  double dmax[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b) dmax[b] = 0.0;
  for (int c = blockIdx.x * kWarps + warp; c < nc; c += gridDim.x * kWarps) {
    const int64_t st = s0 + c;
    const bool rows = st < M.n_row_states;
    float bq[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) bq[b] = -INFINITY;
    const float rv = lane < M.na ? __ldg(M.R + st * M.na + lane) : 0.f;
    if (!rows) {  // Q = R, as the sweeps take it
      for (int a = 0; a < M.na; ++a) {
        const float r = __shfl_sync(0xffffffffu, rv, a);
#pragma unroll
        for (int b = 0; b < NB; ++b) bq[b] = fmaxf(bq[b], r);  // (NaN is never taken)
      }
    } else {
      const int64_t r0 = st * M.na, e0 = (int64_t)__ldg(rp + r0);
      // lane a: end of row a, relative to the state's first entry
      const int ends = (int)((int64_t)__ldg(rp + r0 + min(lane + 1, M.na)) - e0);
      const int last = __shfl_sync(0xffffffffu, ends, M.na - 1);
      const int begin = __shfl_up_sync(0xffffffffu, ends, 1);
      const bool some = lane < M.na && ends > (lane ? begin : 0);
      const unsigned filled = __ballot_sync(0xffffffffu, some);
      uint2* const ent = ents[warp];
      // rows without entries: Q = R + 0 / n
      for (unsigned none = ~filled & (M.na == 32 ? ~0u : (1u << M.na) - 1u); none; none &= none - 1) {
        const float r = __shfl_sync(0xffffffffu, rv, __ffs(none) - 1);
#pragma unroll
        for (int b = 0; b < NB; ++b) bq[b] = fmaxf(bq[b], r + 0.f);
      }
      __syncwarp();
      if (some) rews[warp][__popc(filled & ((1u << lane) - 1u))] = rv;  // of the others, in order
      const float* r = rews[warp];
      float acc[NB];
#pragma unroll
      for (int b = 0; b < NB; ++b) acc[b] = 0.f;
      for (int at = 0; at < last; at += kStage) {
        const int staged = min(last - at, kStage);
        __syncwarp();
        for (int k = lane; k < ((staged + 7) & ~7); k += 32) {
          // (behind the last row of the state the sums are not used)
          uint2 x = make_uint2(0u, 0u);
          if (k < staged) {
            const uint32_t col = (uint32_t)((int64_t)__ldg(M.col + e0 + at + k) - next0);
            x = make_uint2(col * sn * 4u, __float_as_uint(to_f(__ldg(cnt + e0 + at + k))));
          }
          ent[k] = x;
        }
        unsigned marks[kStage / 32];
#pragma unroll
        for (int w = 0; w < kStage / 32; ++w) {
          const int k = ends - 1 - at - 32 * w;
          marks[w] = __reduce_or_sync(0xffffffffu, some && k >= 0 && k < 32 ? 1u << k : 0u);
        }
        __syncwarp();
        if (plain) take_rows<NB, true>(ent, staged, marks, hn, counts, n, rn, r, acc, bq);
        else take_rows<NB, false>(ent, staged, marks, hn, counts, n, rn, r, acc, bq);
      }
    }
    float* h = H + (int64_t)c * s;
    if (j0 == 0 && lane == 0) h[0] = 0.f;  // V before the first sweep
    float before = j0 == 0 ? 0.f : h[j0];  // V_j0 (of the launch before)
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const int j = j0 + 32 * b + lane + 1;
      const float v = bq[b] > -1e6f ? bq[b] : -1e6f;
      float pv = __shfl_up_sync(0xffffffffu, v, 1);
      if (lane == 0) pv = before;
      before = __shfl_sync(0xffffffffu, v, 31);
      if (j <= J) {
        h[j] = v;
        other = other || !(fabsf(v) <= kPlainMax && (fabsf(v) >= kPlainMin || v == 0.f));
        dmax[b] = fmax(dmax[b], fabs((double)v - (double)pv));
      }
    }
  }
  if (other) atomicOr(odd, 1u);
#pragma unroll
  for (int b = 0; b < NB; ++b) red[warp][32 * b + lane] = dmax[b];
  __syncthreads();
  for (int k = threadIdx.x; k < NB * 32; k += kThreads) {
    double mx = 0.0;
    for (int q = 0; q < kWarps; ++q) mx = fmax(mx, red[q][k]);
    const int j = j0 + k + 1;
    if (j <= J && mx > 0.0) atomicMax(resid + j, (unsigned long long)__double_as_longlong(mx));
  }
}

// V of one layer after sweep j
__global__ void k_jacobi_gather(const float* H, int s, int nc, int j, float* V) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < nc) V[c] = H[(int64_t)c * s + j];
}

template <typename F>
cudaError_t dispatch(const ViModel& M, F&& f) {
  if (M.index_bits == 32) {
    if (M.count_type == CNT_U16) return f((int32_t*)0, (uint16_t*)0);
    if (M.count_type == CNT_U32) return f((int32_t*)0, (uint32_t*)0);
    return f((int32_t*)0, (float*)0);
  }
  if (M.count_type == CNT_U16) return f((int64_t*)0, (uint16_t*)0);
  if (M.count_type == CNT_U32) return f((int64_t*)0, (uint32_t*)0);
  return f((int64_t*)0, (float*)0);
}

// sweeps kept of layer t of L, and the row stride of its history
int sweeps_of(int L, int t, int J) { return std::min(J, L - t); }
int stride_of(int L, int t, int J) { return (sweeps_of(L, t, J) + 1 + 31) & ~31; }

}  // namespace

size_t jacobi_history_floats(int64_t nc, int nlayers, int sweeps) {
  size_t n = 0;
  for (int t = 0; t < nlayers; ++t) n += (size_t)nc * stride_of(nlayers, t, sweeps);
  return n;
}

cudaError_t launch_jacobi_layers(const ViModel& M, int64_t nc, int nlayers, int sweeps, float* hist,
                                 unsigned long long* resid, unsigned int* odd, int sms, cudaStream_t st) {
  float* next = nullptr;
  float* at = hist;
  for (int t = nlayers - 1; t >= 0; --t) {
    const int J = sweeps_of(nlayers, t, sweeps), s = stride_of(nlayers, t, sweeps);
    const int sn = t + 1 < nlayers ? stride_of(nlayers, t + 1, sweeps) : 0;
    for (int j0 = 0; j0 < J; j0 += 128) {
      const int nb = std::min(4, (J - j0 + 31) / 32);
      const unsigned grid = (unsigned)std::min<int64_t>((nc + kWarps - 1) / kWarps, 8 * (int64_t)sms);
      cudaError_t e = dispatch(M, [&](auto* pp, auto* pc) -> cudaError_t {
        using PtrT = std::remove_pointer_t<decltype(pp)>;
        using CntT = std::remove_pointer_t<decltype(pc)>;
        auto go = [&](auto kern) {
          kern<<<grid, kThreads, 0, st>>>(M, (int64_t)t * nc, (int)nc, j0, J, next, (uint32_t)sn, at, s, resid,
                                          t + 1 < nlayers ? odd + t + 1 : nullptr, odd + t);
          return cudaGetLastError();
        };
        switch (nb) {
          case 1: return go(k_jacobi_layer<PtrT, CntT, 1>);
          case 2: return go(k_jacobi_layer<PtrT, CntT, 2>);
          case 3: return go(k_jacobi_layer<PtrT, CntT, 3>);
          default: return go(k_jacobi_layer<PtrT, CntT, 4>);
        }
      });
      if (e != cudaSuccess) return e;
    }
    next = at;
    at += (size_t)nc * s;
  }
  return cudaSuccess;
}

cudaError_t launch_jacobi_gather(int64_t nc, int nlayers, int sweeps, const float* hist, int j, float* V,
                                 cudaStream_t st) {
  for (int t = nlayers - 1; t >= 0; --t) {
    const int s = stride_of(nlayers, t, sweeps);
    k_jacobi_gather<<<(unsigned)((nc + 255) / 256), 256, 0, st>>>(hist, s, (int)nc,
                                                                    std::min(j, sweeps_of(nlayers, t, sweeps)), V + t * nc);
    hist += (size_t)nc * s;
  }
  return cudaGetLastError();
}

}  // namespace e2e
