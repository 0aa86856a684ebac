// Environment generator on the GPU: double-gyre realisations -> per-time
// rank reduction -> interpolation to the planning grid, plus the moving
// scalar "cloud" field and the obstacle mask
// (src/data_input/build_environment_DG_with_westward_clouds.py:106-590).
//
// Per time step t, for a batch of steps at once (both fields' matrices of up to
// about 2 GB of steps: a step alone leaves the device idle, its Gram-Schmidt is
// one CTA; one matrix after another took 28.0 ms for the reference's parameters):
//   k_env_realisations  vx, vy, phi of every (sample k, coarse cell) in double,
//                       the reference's expressions in its evaluation order
//                       without contraction (:130-147, 20-84 for the cloud)
//   k_env_center        column means in sample order (np.mean over axis 1 is a
//                       sequential sum for this layout) and the centred matrix
//   rank reduction      the leading n_modes singular triplets of the centred
//                       matrix by a randomized range finder (n_modes + 10
//                       columns from a fixed hash, two power iterations) in
//                       hand-written double kernels: products X B and X^T B,
//                       Gram-Schmidt twice for the orthonormal bases, and the
//                       SVD of the projected matrix through its QR factor and a
//                       one-sided Jacobi SVD of that factor (relative accuracy,
//                       like LAPACK's).  Accepted when the explicit residual
//                       |X - Q Q^T X|_F is below 1e-10 s_1 (then every kept
//                       singular value is exact to ~|R|^2/s_k), or when s_1 is
//                       below 1e-10 of the data's own size (the t = 0 matrices,
//                       rounding noise of the centring, whose vectors no
//                       implementation determines); otherwise re-run with twice
//                       the columns and four power iterations.  The first
//                       n_modes give coefficients u_k s_k and modes v_k, signs
//                       fixed so that each coefficient column's largest-magnitude
//                       entry is positive (the reference's np.linalg.svd leaves
//                       the sign to LAPACK)
// then, for all steps, k_env_interpolate: the reference's griddata 'linear' on
// the coarse cell centres, evaluated from a table of (triangle vertices,
// barycentric weights) per fine point that the caller builds from the same
// Delaunay triangulation (scipy's), summed in griddata's order in double
// without contraction; points outside the hull read 0 (np.nan_to_num of the
// fill value).
#include <cuda_runtime.h>
#include <math.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <type_traits>
#include <vector>

#include "e2e_dp.h"
#include "internal.h"

using namespace e2e;

#define CK(call)                                        \
  do {                                                  \
    cudaError_t _e = (call);                            \
    if (_e != cudaSuccess) return cuda_fail(_e, #call); \
  } while (0)
namespace {

constexpr double kPi = 3.141592653589793;  // math.pi

__device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }

struct RealArgs {
  int g, nws, t0;
  double dt;  // ts[t] = t * dt
  double dxy, A, eps, wlo, whi, wx, wy;
  double* Xv;  // per step: nws x 2n, vx then vy
  double* Xp;  // per step: nws x n, phi
};

// DG_velocity_field.vx_vy / phi / sample_w / get_ij_from_xy (:130-166)
__global__ void k_env_realisations(RealArgs a) {
  const int n = a.g * a.g;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)a.nws * n) return;
  const int k = (int)(idx / n), c = (int)(idx - (int64_t)k * n);
  const int i = c / a.g, j = c - i * a.g;
  const double tt = mul((double)(a.t0 + (int)blockIdx.y), a.dt);
  double* const Xv = a.Xv + (int64_t)blockIdx.y * a.nws * 2 * n;
  double* const Xp = a.Xp + (int64_t)blockIdx.y * a.nws * n;
  // w = w_i + r (w_f - w_i), r = k / (n_wsamples - 1)
  const double r = a.nws > 1 ? (double)k / (double)(a.nws - 1) : 0.0;
  const double w = add(a.wlo, mul(r, sub(a.whi, a.wlo)));
  const double x = mul(add(0.5, (double)j), a.dxy);
  const double y = mul(add(0.5, (double)(a.g - 1 - i)), a.dxy);
  const double swt = sin(mul(w, tt));
  // f = eps sin(wt) x^2 + (1 - 2 eps sin(wt)) x;  fx = 2 eps sin(wt) (x - 1) + 1
  const double term1 = mul(mul(a.eps, swt), mul(x, x));
  const double e2s = mul(mul(2.0, a.eps), swt);
  const double term2 = mul(sub(1.0, e2s), x);
  const double f = add(term1, term2);
  const double fx = add(mul(e2s, sub(x, 1.0)), 1.0);
  const double swf = sin(mul(a.wx, f)), cwf = cos(mul(a.wx, f));
  const double swy = sin(mul(a.wy, y)), cwy = cos(mul(a.wy, y));
  const double vx = -mul(mul(mul(mul(0.5, a.A), kPi), swf), cwy);
  const double vy = mul(mul(mul(mul(a.A, kPi), swy), fx), cwf);
  const double ph = mul(mul(a.A, sin(mul(kPi, f))), swy);
  Xv[(int64_t)k * 2 * n + c] = vx;
  Xv[(int64_t)k * 2 * n + n + c] = vy;
  Xp[(int64_t)k * n + c] = ph;
}

// ---- the batch: nb steps' velocity matrices, then their scalar ones ------------
// Matrix z of a launch (blockIdx.z) is step z of kind 0, or step z - nb of kind 1;
// its arrays lie z * their size behind the kind's pointers.
struct RrKind {
  int ncols, k;        // columns; range-finder columns
  int nseg, seg_rows;  // row segments of X^T B and of the residual
  int colblocks;       // 128-column blocks
  double *X, *mean;                  // nws x ncols, ncols
  double *Q, *L;                     // nws x k
  double *Z, *Bt, *Ub;               // ncols x k
  double *R, *V, *U, *Vs, *S;        // k x k, S: k
  double *P, *part, *scal;           // nseg x k x ncols; nseg x colblocks; 2
  double *C, *M;                     // nws x r, r x ncols
  double* svals;                     // r
  int* sweeps;
};
struct RrBatch {
  RrKind kind[2];
  int nb, nws, r;
  const double* Om;  // test matrix (the same values for every matrix)
};
struct RrMat {
  int m;  // the step
  const RrKind* K;
};
__device__ __forceinline__ RrMat rr_mat(const RrBatch& b, int z) {
  return z >= b.nb ? RrMat{z - b.nb, &b.kind[1]} : RrMat{z, &b.kind[0]};
}

// column means: a sequential sum over the samples, then / n_wsamples (the loads of
// sixteen rows are in flight together, the additions keep their order)
__global__ void k_env_means(RrBatch b) {
  const RrMat t = rr_mat(b, blockIdx.z);
  const int ncols = t.K->ncols, c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncols) return;
  const double* X = t.K->X + (int64_t)t.m * b.nws * ncols + c;
  double s = X[0];
  int k = 1;
  for (; k + 16 <= b.nws; k += 16) {
    double v[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) v[u] = X[(int64_t)(k + u) * ncols];
#pragma unroll
    for (int u = 0; u < 16; ++u) s = add(s, v[u]);
  }
  for (; k < b.nws; ++k) s = add(s, X[(int64_t)k * ncols]);
  t.K->mean[(int64_t)t.m * ncols + c] = __ddiv_rn(s, (double)b.nws);
}

__global__ void k_env_subtract(RrBatch b) {
  const RrMat t = rr_mat(b, blockIdx.z);
  const int ncols = t.K->ncols, c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncols) return;
  const double m = t.K->mean[(int64_t)t.m * ncols + c];
  double* X = t.K->X + (int64_t)t.m * b.nws * ncols + c;
  for (int k = blockIdx.y; k < b.nws; k += gridDim.y) X[(int64_t)k * ncols] = sub(X[(int64_t)k * ncols], m);
}

// From the SVD of the centred matrix X (nws x ncols): coefficients C (nws x r)
// and modes M (r x ncols), mode q = the q-th largest singular value:
// C[k][q] = L[k][q] s_q (the left singular vectors scaled, rank_reduction's
// u1 diag(s1)), M[q][c] = Ub[c][q] (Vh's rows).  Signs: the
// largest-magnitude coefficient of each mode is made positive.
__global__ void k_env_modes(RrBatch a0) {
  const RrMat t = rr_mat(a0, blockIdx.z);
  const int nws = a0.nws, ncols = t.K->ncols, r = a0.r, kk = t.K->k;
  const int q = blockIdx.x;  // one block per mode
  const double s = t.K->S[(int64_t)t.m * kk + q];
  __shared__ double best_v[32];
  __shared__ int best_k[32];
  const double* u = t.K->L + ((int64_t)t.m * kk + q) * nws;
  double bv = -1.0;
  int bk = 0x7fffffff;
  for (int k = threadIdx.x; k < nws; k += blockDim.x) {
    const double v = fabs(u[k] * s);
    if (v > bv || (v == bv && k < bk)) {
      bv = v;
      bk = k;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const double ov = __shfl_xor_sync(0xffffffffu, bv, o);
    const int ok = __shfl_xor_sync(0xffffffffu, bk, o);
    if (ov > bv || (ov == bv && ok < bk)) {
      bv = ov;
      bk = ok;
    }
  }
  if ((threadIdx.x & 31) == 0) {
    best_v[threadIdx.x >> 5] = bv;
    best_k[threadIdx.x >> 5] = bk;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
      if (best_v[w] > bv || (best_v[w] == bv && best_k[w] < bk)) {
        bv = best_v[w];
        bk = best_k[w];
      }
    best_k[0] = bk;
  }
  __syncthreads();
  const double sgn = u[best_k[0]] < 0.0 ? -1.0 : 1.0;
  if (threadIdx.x == 0) t.K->svals[(int64_t)t.m * r + q] = s;
  for (int k = threadIdx.x; k < nws; k += blockDim.x) t.K->C[((int64_t)t.m * nws + k) * r + q] = sgn * (u[k] * s);
  const double* v = t.K->Ub + ((int64_t)t.m * kk + q) * ncols;
  for (int c = threadIdx.x; c < ncols; c += blockDim.x) t.K->M[((int64_t)t.m * r + q) * ncols + c] = sgn * v[c];
}

// test matrix of the range finder: deterministic values in [-1, 1) from a
// 64-bit mix of the index (any matrix of full rank with the range works)
__global__ void k_env_test_matrix(double* O, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint64_t z = (uint64_t)i * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E019ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  z ^= z >> 31;
  O[i] = (double)(z >> 11) * (2.0 / 9007199254740992.0) - 1.0;
}

// coarse arrays of step t: [u, v, phi, ui_0.., vi_0.., phi_i_0..] (3 + 3r arrays
// of n) and the coefficients of both rank reductions.  The reference holds the
// coarse means and modes in float32 arrays except all_phi_mat, a float64 array
// (:271), so every value but phi's mean is rounded to float before it is
// interpolated.
__global__ void k_env_store(RrBatch b, int n, double* coarse0, float* yi0, float* phi_yi0) {
  const int nws = b.nws, r = b.r, t = blockIdx.y;
  const double* mv = b.kind[0].mean + (int64_t)t * 2 * n;
  const double* mp = b.kind[1].mean + (int64_t)t * n;
  const double* Mv = b.kind[0].M + (int64_t)t * r * 2 * n;
  const double* Mp = b.kind[1].M + (int64_t)t * r * n;
  const double* Cv = b.kind[0].C + (int64_t)t * nws * r;
  const double* Cp = b.kind[1].C + (int64_t)t * nws * r;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t nb = (int64_t)(3 + 3 * r) * n;
  if (idx < nb) {
    double* coarse = coarse0 + (int64_t)t * nb;
    const int b2 = (int)(idx / n), c = (int)(idx - (int64_t)b2 * n);
    double v;
    if (b2 == 0) v = mv[c];
    else if (b2 == 1) v = mv[n + c];
    else if (b2 == 2) v = mp[c];
    else if (b2 < 3 + r) v = Mv[(int64_t)(b2 - 3) * 2 * n + c];
    else if (b2 < 3 + 2 * r) v = Mv[(int64_t)(b2 - 3 - r) * 2 * n + n + c];
    else v = Mp[(int64_t)(b2 - 3 - 2 * r) * n + c];
    coarse[idx] = b2 == 2 ? v : (double)(float)v;
  }
  const int64_t nc = (int64_t)nws * r;
  if (idx < nc) {
    yi0[(int64_t)t * nc + idx] = (float)Cv[idx];
    phi_yi0[(int64_t)t * nc + idx] = (float)Cp[idx];
  }
}

struct InterpArgs {
  int nt, r, n, G2;
  const double* coarse;  // nt x (3 + 3r) x n
  const int32_t* vert;   // G2 x 3 (vert[0] < 0: outside the hull)
  const double* wgt;     // G2 x 3
  unsigned int* err;     // set when a vertex index is outside the coarse grid
  float *u, *v, *phi, *ui, *vi, *phi_i;
};

// LinearNDInterpolator's evaluation (scipy/interpolate/_interpnd.pyx
// _do_evaluate): out = 0; out += c_j * value[vertex_j] for j = 0..2 in double
__global__ void k_env_interpolate(InterpArgs a) {
  const int nb = 3 + 3 * a.r;
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)a.nt * nb * a.G2) return;
  const int p = (int)(idx % a.G2);
  const int64_t tb = idx / a.G2;
  const int b = (int)(tb % nb), t = (int)(tb / nb);
  const double* src = a.coarse + ((int64_t)t * nb + b) * a.n;
  float out = 0.f;  // np.nan_to_num of the fill value outside the hull
  const int v0 = a.vert[3 * p], v1 = a.vert[3 * p + 1], v2 = a.vert[3 * p + 2];
  if (v0 >= 0) {
    if (v0 >= a.n || v1 < 0 || v1 >= a.n || v2 < 0 || v2 >= a.n) {
      atomicOr(a.err, 1u);  // a caller's table that does not index the coarse grid
    } else {
      double o = 0.0;
      o = add(o, mul(a.wgt[3 * p + 0], src[v0]));
      o = add(o, mul(a.wgt[3 * p + 1], src[v1]));
      o = add(o, mul(a.wgt[3 * p + 2], src[v2]));
      out = isnan(o) ? 0.f : (float)o;
    }
  }
  float* dst;
  if (b == 0) dst = a.u + (int64_t)t * a.G2;
  else if (b == 1) dst = a.v + (int64_t)t * a.G2;
  else if (b == 2) dst = a.phi + (int64_t)t * a.G2;
  else if (b < 3 + a.r) dst = a.ui + ((int64_t)t * a.r + (b - 3)) * a.G2;
  else if (b < 3 + 2 * a.r) dst = a.vi + ((int64_t)t * a.r + (b - 3 - a.r)) * a.G2;
  else dst = a.phi_i + ((int64_t)t * a.r + (b - 3 - 2 * a.r)) * a.G2;
  dst[p] = out;
}

// DG_scalar_field.generate_phi (:20-98) on the fine grid (its interpolate_degree
// is the default 1, so T = t / 2), and fill_obstacles (:441-468)
struct CloudArgs {
  int nt, G;
  double dxy;  // fine spacing
  double A_sc;
  int obst_mode;
  double ou, ol, ow, osx, osy;
  float* s;
  int32_t* mask;
};

__global__ void k_env_cloud(CloudArgs a) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t G2 = (int64_t)a.G * a.G;
  if (idx >= (int64_t)a.nt * G2) return;
  const int t = (int)(idx / G2);
  const int p = (int)(idx - (int64_t)t * G2);
  const int i = p / a.G, j = p - i * a.G;
  const double x = mul(add(0.5, (double)j), a.dxy);
  const double xl = mul(add(0.5, (double)(a.G - 1)), a.dxy);  // xs[-1]
  const double T = __ddiv_rn((double)t, 2.0);
  const double l = __ddiv_rn(xl, 2.0);
  const double dom = add(xl, a.dxy);
  const double xt = add(x, mul(T, a.dxy));
  double f;
  if (xt <= l) {
    f = 1.0;
  } else if (l < xt && xt < add(l, mul(0.2, dom))) {
    const double slope = __ddiv_rn(1.0, mul(-0.2, dom));
    f = add(1.0, mul(slope, sub(x, sub(l, mul(T, a.dxy)))));
  } else {
    f = 0.0;
  }
  a.s[idx] = (float)mul(a.A_sc, f);
  int m = 0;
  if (a.obst_mode == E2E_OBST_STATIC) {
    const int ru = (int)(0.4 * a.G), rd = (int)(0.5 * a.G), cl = (int)(0.5 * a.G), cr = (int)(0.6 * a.G);
    m = (i >= ru && i < rd && j >= cl && j < cr) ? 1 : 0;
  } else if (a.obst_mode == E2E_OBST_DYNAMIC) {
    const double clf = floor(add(a.ol, mul((double)t, a.osx)));
    const double ruf = floor(add(a.ou, mul((double)t, a.osy)));
    const double crf = trunc(add(clf, a.ow)), rdf = trunc(add(ruf, a.ow));
    const double hi = (double)(a.G - 1);
    const bool inside = (0.0 < clf && clf < hi) && (0.0 < crf && crf < hi) && (0.0 < ruf && ruf < hi) &&
                        (0.0 < rdf && rdf < hi);
    m = (inside && i >= (int)ruf && i < (int)rdf && j >= (int)clf && j < (int)crf) ? 1 : 0;
  }
  a.mask[idx] = m;
}

// ---- rank reduction: the leading singular triplets of the centred matrix ----
//
// X is row-major nws x ncols on the device.  A randomized range finder with k
// columns (n_modes + 10): Q = orth(X Om), two power iterations
// Q <- orth(X orth(X^T Q)), Bt = X^T Q (ncols x k), the explicit residual
// |X - Q Bt^T|_F, then the SVD of Bt through its QR: Bt = Qb R, R = U_R S V_R^T
// by one-sided Jacobi (relative accuracy: each singular value of R equals one
// of Bt's to about eps s_1, so a Gram-matrix eigensolve's (s_1/s_k)^2 loss is
// avoided), Ub = Qb U_R, and the sample-side vectors L = Q V_R.  Every product
// and reduction runs in a fixed order (warp trees, segment sums in segment
// order), so a generation is deterministic.  Matrices besides X are
// column-major with the leading dimension of their row count.

constexpr int kRrMaxK = 64;       // range-finder columns at most
constexpr int kRrMaxSweeps = 60;  // Jacobi sweeps at most (convergence is quadratic)

// partial products of X^T B over row segments: P[seg][c][j] = sum over the
// segment's rows i, in order, of X[i][j] B[i][c]; a thread per column j
template <int K>
__global__ void __launch_bounds__(128) k_rr_xtb(RrBatch b) {
  const RrMat t = rr_mat(b, blockIdx.z);
  const int nws = b.nws, ncols = t.K->ncols, k = t.K->k, seg_rows = t.K->seg_rows, ldb = nws;
  if ((int)blockIdx.x >= t.K->colblocks || (int)blockIdx.y >= t.K->nseg) return;
  const double* X = t.K->X + (int64_t)t.m * nws * ncols;
  const double* B = t.K->Q + (int64_t)t.m * nws * k;
  double* P = t.K->P + (int64_t)t.m * t.K->nseg * k * ncols;
  __shared__ double Bs[32][K];
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i0 = blockIdx.y * seg_rows, i1 = min(nws, i0 + seg_rows);
  double acc[K];
#pragma unroll
  for (int c = 0; c < K; ++c) acc[c] = 0.0;
  for (int it = i0; it < i1; it += 32) {
    const int nrow = min(32, i1 - it);
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * K; e += blockDim.x) {
      const int rr = e / K, c = e - rr * K;
      Bs[rr][c] = (rr < nrow && c < k) ? B[(int64_t)c * ldb + it + rr] : 0.0;
    }
    __syncthreads();
    if (j < ncols) {
      for (int rr = 0; rr < nrow; ++rr) {
        const double x = X[(int64_t)(it + rr) * ncols + j];
#pragma unroll
        for (int c = 0; c < K; ++c) acc[c] = fma(x, Bs[rr][c], acc[c]);
      }
    }
  }
  if (j < ncols) {
#pragma unroll
    for (int c = 0; c < K; ++c)
      if (c < k) P[((int64_t)blockIdx.y * k + c) * ncols + j] = acc[c];
  }
}

// C[j + c ncols] = sum over segments s = 0.. in order of P[s][c][j], C = Bt or Z
__global__ void k_rr_sum_segments(RrBatch b, bool to_bt) {
  const RrMat t = rr_mat(b, blockIdx.z);
  const int nseg = t.K->nseg, ncols = t.K->ncols, k = t.K->k, ldc = ncols;
  const double* P = t.K->P + (int64_t)t.m * nseg * k * ncols;
  double* C = (to_bt ? t.K->Bt : t.K->Z) + (int64_t)t.m * ncols * k;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)ncols * k) return;
  const int c = (int)(e / ncols), j = (int)(e - (int64_t)c * ncols);
  double s = P[(int64_t)c * ncols + j];
  for (int g = 1; g < nseg; ++g) s += P[((int64_t)g * k + c) * ncols + j];
  C[(int64_t)c * ldc + j] = s;
}

// Q (nws x k) = X B, B ncols x k (Z, or the test matrix): a warp takes ROWS rows
// of X, lanes over the columns, lane sums reduced by a shuffle tree (lane 0's
// result is written).  Reading B once for four rows instead of one: 0.68 -> 0.19
// ms for the 20 matrices of the reference's parameters.
template <int K, int ROWS>
__global__ void __launch_bounds__(128) k_rr_xb(RrBatch b, bool test) {
  const RrMat t = rr_mat(b, blockIdx.z);
  const int nws = b.nws, ncols = t.K->ncols, k = t.K->k, ldb = ncols, ldc = nws;
  const double* B = test ? b.Om : t.K->Z + (int64_t)t.m * ncols * k;
  double* C = t.K->Q + (int64_t)t.m * nws * k;
  const int row0 = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * ROWS, lane = threadIdx.x & 31;
  if (row0 >= nws) return;  // whole warps
  const double* x[ROWS];
#pragma unroll
  for (int r = 0; r < ROWS; ++r) x[r] = t.K->X + ((int64_t)t.m * nws + min(row0 + r, nws - 1)) * ncols;
  double acc[ROWS][K];
#pragma unroll
  for (int r = 0; r < ROWS; ++r)
#pragma unroll
    for (int c = 0; c < K; ++c) acc[r][c] = 0.0;
  for (int j = lane; j < ncols; j += 32) {
    double xv[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) xv[r] = x[r][j];
#pragma unroll
    for (int c = 0; c < K; ++c) {
      if (c < k) {
        const double bv = B[(int64_t)c * ldb + j];
#pragma unroll
        for (int r = 0; r < ROWS; ++r) acc[r][c] = fma(xv[r], bv, acc[r][c]);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < ROWS; ++r) {
#pragma unroll
    for (int c = 0; c < K; ++c) {
      if (c < k) {
        double v = acc[r][c];
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0 && row0 + r < nws) C[(int64_t)c * ldc + row0 + r] = v;
      }
    }
  }
}

// Ub = Bt U (ncols x k), or L = Q Vs (nws x k): a thread per entry, sum in order
__global__ void k_rr_small(RrBatch b, bool left) {
  const RrMat t = rr_mat(b, blockIdx.z);
  const int k = t.K->k, rows = left ? b.nws : t.K->ncols, lda = rows, ldc = rows;
  const double* A = (left ? t.K->Q : t.K->Bt) + (int64_t)t.m * rows * k;
  const double* W = (left ? t.K->Vs : t.K->U) + (int64_t)t.m * k * k;
  double* C = (left ? t.K->L : t.K->Ub) + (int64_t)t.m * rows * k;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (int64_t)rows * k) return;
  const int c = (int)(e / rows), i = (int)(e - (int64_t)c * rows);
  double s = 0.0;
  for (int l = 0; l < k; ++l) s = fma(A[(int64_t)l * lda + i], W[l + c * k], s);
  C[(int64_t)c * ldc + i] = s;
}

// block-wide sum of v (fixed order: a shuffle tree per warp, then the warps in
// order by thread 0); every thread returns it.  red: 33 doubles of shared memory
__device__ double rr_block_sum(double v, double* red) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = red[0];
    for (int w = 1; w < nw; ++w) s += red[w];
    red[32] = s;
  }
  __syncthreads();
  return red[32];
}

// Orthonormal columns in place: A (rows x k, ld lda) = Q R by classical
// Gram-Schmidt applied twice per column (orthogonal to working precision); R
// (k x k, ld k, upper triangular, may be null) receives both passes'
// coefficients and the norms.  A column that the second pass shrinks below
// half its length lies in the span of the earlier ones to working precision
// (what is left is rounding, which no further pass makes orthogonal): it
// becomes zero, as does a zero column (R's diagonal 0).  One CTA a matrix: Q, Z,
// or Bt with R kept.
enum : int { RR_Q = 0, RR_Z = 1, RR_BT = 2 };
template <int K>
__global__ void __launch_bounds__(256) k_rr_cgs2(RrBatch b, int which) {
  const RrMat t = rr_mat(b, blockIdx.z);
  const int k = t.K->k, rows = which == RR_Q ? b.nws : t.K->ncols, lda = rows;
  double* A = (which == RR_Q ? t.K->Q : which == RR_Z ? t.K->Z : t.K->Bt) + (int64_t)t.m * rows * k;
  double* R = which == RR_BT ? t.K->R + (int64_t)t.m * k * k : nullptr;
  __shared__ double red[33];
  __shared__ double wsum[8][K];
  __shared__ double d[K];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  if (R)
    for (int e = tid; e < k * k; e += blockDim.x) R[e] = 0.0;
  __syncthreads();
  for (int j = 0; j < k; ++j) {
    double* aj = A + (int64_t)j * lda;
    double n1 = 0.0;  // length after the first pass
    for (int pass = 0; pass < 2 && j > 0; ++pass) {
      double part[K];
#pragma unroll
      for (int i = 0; i < K; ++i) part[i] = 0.0;
      for (int row = tid; row < rows; row += blockDim.x) {
        const double v = aj[row];
#pragma unroll
        for (int i = 0; i < K; ++i)
          if (i < j) part[i] = fma(A[(int64_t)i * lda + row], v, part[i]);
      }
#pragma unroll
      for (int i = 0; i < K; ++i) {
        if (i < j) {
          double v = part[i];
          for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
          if (lane == 0) wsum[warp][i] = v;
        }
      }
      __syncthreads();
      if (tid < j) {
        double s = wsum[0][tid];
        for (int w = 1; w < nw; ++w) s += wsum[w][tid];
        d[tid] = s;
        if (R) R[tid + j * k] += s;
      }
      __syncthreads();
      for (int row = tid; row < rows; row += blockDim.x) {
        double v = aj[row];
        for (int i = 0; i < j; ++i) v = fma(-d[i], A[(int64_t)i * lda + row], v);
        aj[row] = v;
      }
      __syncthreads();
      if (pass == 0) {
        double t2 = 0.0;
        for (int row = tid; row < rows; row += blockDim.x) t2 = fma(aj[row], aj[row], t2);
        n1 = sqrt(rr_block_sum(t2, red));
      }
    }
    double s2 = 0.0;
    for (int row = tid; row < rows; row += blockDim.x) s2 = fma(aj[row], aj[row], s2);
    const double n2 = sqrt(rr_block_sum(s2, red));
    const double nrm = (j > 0 && n2 < 0.5 * n1) ? 0.0 : n2;
    if (R && tid == 0) R[j + j * k] = nrm;
    for (int row = tid; row < rows; row += blockDim.x) aj[row] = nrm > 0.0 ? aj[row] / nrm : 0.0;
    __syncthreads();
  }
}

// One-sided Jacobi SVD of the k x k matrix W (ld k, destroyed): its columns are
// rotated until pairwise orthogonal (|w_p . w_q| <= k eps |w_p| |w_q|), the
// rotations accumulated in V; then W_in = U diag(S) V^T.  Outputs sorted by
// descending singular value (ties: lower column first): S (k), U and Vs (k x k,
// ld k; a zero singular value gives a zero U column).  Rounds of disjoint
// pairs (a round-robin tournament over the columns), a warp per pair, each
// warp's reductions broadcast from lane 0 so all lanes rotate alike.  One CTA a matrix.
__global__ void __launch_bounds__(256) k_rr_jacobi(RrBatch b) {
  const RrMat t = rr_mat(b, blockIdx.z);
  const int k = t.K->k;
  double* W = t.K->R + (int64_t)t.m * k * k;
  double* V = t.K->V + (int64_t)t.m * k * k;
  double* U = t.K->U + (int64_t)t.m * k * k;
  double* Vs = t.K->Vs + (int64_t)t.m * k * k;
  double* S = t.K->S + (int64_t)t.m * k;
  int* sweeps = t.K->sweeps + t.m;
  __shared__ int rotated;
  __shared__ double sv[kRrMaxK];
  __shared__ int order[kRrMaxK];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
  for (int e = tid; e < k * k; e += blockDim.x) V[e] = (e % k == e / k) ? 1.0 : 0.0;
  const int kk = k + (k & 1);  // players (index k: a bye)
  const double tol = (double)k * 2.220446049250313e-16;
  int sweep = 0;
  for (; sweep < kRrMaxSweeps; ++sweep) {
    if (tid == 0) rotated = 0;
    __syncthreads();
    for (int round = 0; round < kk - 1; ++round) {
      for (int pi = warp; pi < kk / 2; pi += nw) {
        // position 0 holds player 0, position i >= 1 player 1 + (i - 1 + round) mod (kk - 1)
        const int ia = pi, ib = kk - 1 - pi;
        const int pa = ia == 0 ? 0 : 1 + (ia - 1 + round) % (kk - 1);
        const int pb = 1 + (ib - 1 + round) % (kk - 1);
        if (pa >= k || pb >= k) continue;
        const int p = min(pa, pb), q = max(pa, pb);
        double* wp = W + p * k;
        double* wq = W + q * k;
        double al = 0.0, be = 0.0, ga = 0.0;
        for (int r = lane; r < k; r += 32) {
          al = fma(wp[r], wp[r], al);
          be = fma(wq[r], wq[r], be);
          ga = fma(wp[r], wq[r], ga);
        }
        for (int o = 16; o > 0; o >>= 1) {
          al += __shfl_xor_sync(0xffffffffu, al, o);
          be += __shfl_xor_sync(0xffffffffu, be, o);
          ga += __shfl_xor_sync(0xffffffffu, ga, o);
        }
        al = __shfl_sync(0xffffffffu, al, 0);
        be = __shfl_sync(0xffffffffu, be, 0);
        ga = __shfl_sync(0xffffffffu, ga, 0);
        if (!(fabs(ga) > tol * sqrt(al) * sqrt(be))) continue;
        const double zeta = (be - al) / (2.0 * ga);
        const double t = fabs(zeta) > 1e150 ? 0.5 / zeta
                                            : copysign(1.0, zeta) / (fabs(zeta) + sqrt(fma(zeta, zeta, 1.0)));
        const double c = 1.0 / sqrt(fma(t, t, 1.0)), s = c * t;
        double* vp = V + p * k;
        double* vq = V + q * k;
        for (int r = lane; r < k; r += 32) {
          const double a = wp[r], b = wq[r];
          wp[r] = c * a - s * b;
          wq[r] = s * a + c * b;
          const double va = vp[r], vb = vq[r];
          vp[r] = c * va - s * vb;
          vq[r] = s * va + c * vb;
        }
        if (lane == 0) rotated = 1;
      }
      __syncthreads();
    }
    const int any = rotated;
    __syncthreads();
    if (!any) break;
  }
  for (int j = tid; j < k; j += blockDim.x) {
    double s2 = 0.0;
    for (int r = 0; r < k; ++r) s2 = fma(W[j * k + r], W[j * k + r], s2);
    sv[j] = sqrt(s2);
  }
  __syncthreads();
  if (tid == 0) {
    for (int j = 0; j < k; ++j) order[j] = j;
    for (int a = 0; a < k; ++a) {
      int best = a;
      for (int b = a + 1; b < k; ++b)
        if (sv[order[b]] > sv[order[best]] || (sv[order[b]] == sv[order[best]] && order[b] < order[best])) best = b;
      const int tmp = order[a];
      order[a] = order[best];
      order[best] = tmp;
    }
    if (sweeps) *sweeps = sweep;
  }
  __syncthreads();
  for (int e = tid; e < k * k; e += blockDim.x) {
    const int c = e / k, r = e - c * k, src = order[c];
    const double s = sv[src];
    if (r == 0) S[c] = s;
    U[e] = s > 0.0 ? W[src * k + r] / s : 0.0;
    Vs[e] = V[src * k + r];
  }
}

// partial sums of squares of the residual X - Q Bt^T (Q nws x k, Bt ncols x
// k): a thread per column j over a row segment, one partial per CTA
template <int K>
__global__ void __launch_bounds__(128) k_rr_resid(RrBatch bt) {
  const RrMat t = rr_mat(bt, blockIdx.z);
  const int nws = bt.nws, ncols = t.K->ncols, k = t.K->k, seg_rows = t.K->seg_rows;
  if ((int)blockIdx.x >= t.K->colblocks || (int)blockIdx.y >= t.K->nseg) return;  // whole CTAs
  const double* X = t.K->X + (int64_t)t.m * nws * ncols;
  const double* Q = t.K->Q + (int64_t)t.m * nws * k;
  const double* Bt = t.K->Bt + (int64_t)t.m * ncols * k;
  double* part = t.K->part + (int64_t)t.m * t.K->nseg * t.K->colblocks;
  __shared__ double Qs[32][K];
  __shared__ double red[33];
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  const int i0 = blockIdx.y * seg_rows, i1 = min(nws, i0 + seg_rows);
  double b[K];
#pragma unroll
  for (int c = 0; c < K; ++c) b[c] = (j < ncols && c < k) ? Bt[(int64_t)c * ncols + j] : 0.0;
  double ssq = 0.0;
  for (int it = i0; it < i1; it += 32) {
    const int nrow = min(32, i1 - it);
    __syncthreads();
    for (int e = threadIdx.x; e < 32 * K; e += blockDim.x) {
      const int rr = e / K, c = e - rr * K;
      Qs[rr][c] = (rr < nrow && c < k) ? Q[(int64_t)c * nws + it + rr] : 0.0;
    }
    __syncthreads();
    if (j < ncols) {
      for (int rr = 0; rr < nrow; ++rr) {
        double v = X[(int64_t)(it + rr) * ncols + j];
#pragma unroll
        for (int c = 0; c < K; ++c) v = fma(-Qs[rr][c], b[c], v);
        ssq = fma(v, v, ssq);
      }
    }
  }
  const double s = rr_block_sum(ssq, red);
  if (threadIdx.x == 0) part[(int64_t)blockIdx.y * t.K->colblocks + blockIdx.x] = s;
}

// scal[0] = sum of the residual's partials in order (one thread: a few hundred)
__global__ void k_rr_sum_serial(RrBatch b) {
  if (threadIdx.x != 0) return;
  const RrMat t = rr_mat(b, blockIdx.z);
  const int n = t.K->nseg * t.K->colblocks;
  const double* v = t.K->part + (int64_t)t.m * n;
  double s = 0.0;
  int i = 0;
  for (; i + 8 <= n; i += 8) {
    double x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = v[i + u];
#pragma unroll
    for (int u = 0; u < 8; ++u) s += x[u];
  }
  for (; i < n; ++i) s += v[i];
  t.K->scal[2 * t.m] = s;
}

// scal[1] = sum of squares of the mean, one CTA a matrix, fixed order
__global__ void __launch_bounds__(256) k_rr_sumsq(RrBatch b) {
  __shared__ double red[33];
  const RrMat t = rr_mat(b, blockIdx.z);
  const int n = t.K->ncols;
  const double* v = t.K->mean + (int64_t)t.m * n;
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s = fma(v[i], v[i], s);
  s = rr_block_sum(s, red);
  if (threadIdx.x == 0) t.K->scal[2 * t.m + 1] = s;
}

constexpr int kMaxBatch = 65535 / 2;  // steps of a batch at most
constexpr int kRrSegs = 16;  // row segments of the X^T B products at most

// row segments for X^T B / the residual: enough CTAs to cover the SMs for one
// matrix (the sums' order is part of the result: it does not depend on the batch)
void rr_segments(int nws, int ncols, int* nseg, int* seg_rows) {
  const int colblocks = (ncols + 127) / 128;
  int s = std::max(1, std::min(kRrSegs, (296 + colblocks - 1) / colblocks));
  s = std::min(s, (nws + 31) / 32);
  int rows = (nws + s - 1) / s;
  rows = (rows + 31) / 32 * 32;
  *seg_rows = rows;
  *nseg = (nws + rows - 1) / rows;
}

// f(bucket of the range-finder columns)
template <typename F>
void rr_bucket(int k, F&& f) {
  if (k <= 16) f(std::integral_constant<int, 16>{});
  else if (k <= 32) f(std::integral_constant<int, 32>{});
  else f(std::integral_constant<int, 64>{});
}

// doubles of one matrix' work arrays (RrKind from Q on, but mean, C, M, svals)
size_t rr_work_doubles(int nws, int ncols, int k) {
  int nseg, rows;
  rr_segments(nws, ncols, &nseg, &rows);
  return (size_t)2 * nws * k + (size_t)3 * ncols * k + (size_t)4 * k * k + k + (size_t)nseg * k * ncols +
         (size_t)nseg * ((ncols + 127) / 128) + 2 + 1;
}

// carve the work arrays of nb matrices from p
double* rr_carve(RrKind* K, int nws, int ncols, int k, int nb, double* p) {
  K->ncols = ncols;
  K->k = k;
  K->colblocks = (ncols + 127) / 128;
  rr_segments(nws, ncols, &K->nseg, &K->seg_rows);
  auto take = [&](size_t each) {
    double* q = p;
    p += each * nb;
    return q;
  };
  K->Q = take((size_t)nws * k);
  K->L = take((size_t)nws * k);
  K->Z = take((size_t)ncols * k);
  K->Bt = take((size_t)ncols * k);
  K->Ub = take((size_t)ncols * k);
  K->R = take((size_t)k * k);
  K->V = take((size_t)k * k);
  K->U = take((size_t)k * k);
  K->Vs = take((size_t)k * k);
  K->S = take(k);
  K->P = take((size_t)K->nseg * k * ncols);
  K->part = take((size_t)K->nseg * K->colblocks);
  K->scal = take(2);
  K->sweeps = reinterpret_cast<int*>(take(1));
  return p;
}

// Randomized SVDs of the nz centred matrices of a batch (nz = nb: the first kind
// alone) with k columns and `power` power iterations, then coefficients and modes
// of all of them.  The caller checks the certificates (rr_certified) from scal
// and S.
e2e_status randomized_svds(const RrBatch& b, int nz, int power, double* Om, cudaStream_t st) {
  const bool both = nz > b.nb;
  const int ncols = both ? std::max(b.kind[0].ncols, b.kind[1].ncols) : b.kind[0].ncols;
  const int k = both ? std::max(b.kind[0].k, b.kind[1].k) : b.kind[0].k;
  const int nseg = both ? std::max(b.kind[0].nseg, b.kind[1].nseg) : b.kind[0].nseg;
  const unsigned z = (unsigned)nz;
  const dim3 cols((unsigned)((ncols + 127) / 128), (unsigned)nseg, z);
  const dim3 per_col((unsigned)(((int64_t)ncols * k + 255) / 256), 1, z);
  const dim3 per_row((unsigned)(((int64_t)b.nws * k + 255) / 256), 1, z);
  const dim3 one(1, 1, z);
  const int64_t no = (int64_t)ncols * k;
  k_env_test_matrix<<<(unsigned)((no + 255) / 256), 256, 0, st>>>(Om, no);
  rr_bucket(k, [&](auto bucket) {
    constexpr int K = decltype(bucket)::value, kRows = K == 16 ? 4 : 1;
    const dim3 rows((unsigned)((b.nws + 4 * kRows - 1) / (4 * kRows)), 1, z);  // 4 warps a CTA
    auto xtb = [&](bool to_bt) {
      k_rr_xtb<K><<<cols, 128, 0, st>>>(b);
      k_rr_sum_segments<<<per_col, 256, 0, st>>>(b, to_bt);
    };
    k_rr_xb<K, kRows><<<rows, 128, 0, st>>>(b, true);  // Q = X Om
    k_rr_cgs2<K><<<one, 256, 0, st>>>(b, RR_Q);
    for (int it = 0; it < power; ++it) {  // Q <- orth(X orth(X^T Q))
      xtb(false);
      k_rr_cgs2<K><<<one, 256, 0, st>>>(b, RR_Z);
      k_rr_xb<K, kRows><<<rows, 128, 0, st>>>(b, false);
      k_rr_cgs2<K><<<one, 256, 0, st>>>(b, RR_Q);
    }
    xtb(true);  // Bt = X^T Q
    k_rr_resid<K><<<cols, 128, 0, st>>>(b);
    k_rr_sum_serial<<<one, 32, 0, st>>>(b);
    k_rr_sumsq<<<one, 256, 0, st>>>(b);
    // Bt = Qb R (Bt becomes Qb), R = U_R S V_R^T, Ub = Qb U_R, L = Q V_R
    k_rr_cgs2<K><<<one, 256, 0, st>>>(b, RR_BT);
  });
  k_rr_jacobi<<<one, 256, 0, st>>>(b);
  k_rr_small<<<per_col, 256, 0, st>>>(b, false);
  k_rr_small<<<per_row, 256, 0, st>>>(b, true);
  k_env_modes<<<dim3((unsigned)b.r, 1, z), 256, 0, st>>>(b);
  CK(cudaGetLastError());
  return E2E_OK;
}

// A reduction stands when
//  * |X - Q Q^T X|_F <= 1e-10 s_1 (then each kept singular value is exact to
//    about |R|^2 / s_k, machine precision relative to s_1), or
//  * s_1 <= 1e-10 sqrt(nws) |mean|: the centred matrix is below the rounding of
//    the data it was centred from (every realisation alike, as at t = 0), so
//    its singular vectors are not determined by the data and the computed ones
//    stand, as LAPACK's do for the reference.
bool rr_certified(const double* scal, double s1, int nws) {
  const double rnorm = sqrt(scal[0]), mnorm = sqrt(scal[1]);
  const bool ok = (s1 > 0.0 && rnorm <= 1e-10 * s1) || !(s1 > 1e-10 * sqrt((double)nws) * mnorm);
  return ok && std::isfinite(rnorm) && std::isfinite(s1);
}

// One matrix (X, mean, outputs as in `one.kind[0]`) whose first reduction did not
// stand: twice the columns (up to 64 and the matrix's smaller side) and four
// power iterations until it does.  When the columns span the whole smaller side
// the residual is rounding only, so only n_modes above 54 on a matrix wider than
// 64 can end uncertified: then an error.
e2e_status enlarge_svd(RrBatch one, int k, double* Om, cudaStream_t st, int* enlarged) {
  const int nws = one.nws, ncols = one.kind[0].ncols, nsmall = std::min(nws, ncols);
  one.nb = 1;
  for (bool first = true;; first = false) {
    const int k2 = std::min(std::min(2 * k, kRrMaxK), nsmall);
    if (k2 == k && !first)
      return fail(E2E_ERR_DEVICE, "rank reduction not certified with " + std::to_string(k) +
                                      " columns (|X - QQ^T X| above 1e-10 s_1)");
    ++*enlarged;
    k = k2;
    DeviceScratch scratch(st);
    double* work = nullptr;
    CK(dalloc((void**)&work, sizeof(double) * rr_work_doubles(nws, ncols, k), st));
    scratch.add(work);
    rr_carve(&one.kind[0], nws, ncols, k, 1, work);
    e2e_status s = randomized_svds(one, 1, 4, Om, st);
    if (s != E2E_OK) return s;
    double h[3];
    CK(cudaMemcpyAsync(h, one.kind[0].scal, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(h + 2, one.kind[0].S, sizeof(double), cudaMemcpyDeviceToHost, st));
    CK(cudaStreamSynchronize(st));
    if (rr_certified(h, h[2], nws)) return E2E_OK;
  }
}

}  // namespace

extern "C" e2e_status e2e_env_generate(const e2e_env_params* p, const int32_t* interp_vertices,
                                       const double* interp_weights, int out_where, const e2e_env_fields* out,
                                       double* svals_out, e2e_env_stats* stats, void* stream) {
  if (!p || !out) return fail(E2E_ERR_INVALID, "null argument");
  if (out_where != E2E_HOST && out_where != E2E_DEVICE) return fail(E2E_ERR_INVALID, "bad out_where");
  const int g = p->init_gsize, nt = p->nt, nws = p->n_wsamples, r = p->n_modes, d = p->interpolate_degree;
  if (g < 2 || nt < 1 || nws < 2 || r < 1 || d < 1)
    return fail(E2E_ERR_INVALID, "init_gsize >= 2, nt >= 1, n_wsamples >= 2, n_modes >= 1, interpolate_degree >= 1");
  const int n = g * g;
  // the reference asserts n_modes <= min(nt, n_wsamples, 2 n) (:213); the scalar
  // field's reduction needs n_modes <= min(n_wsamples, n) as well
  if (r > nt || r > nws || r > n) return fail(E2E_ERR_INVALID, "n_modes above min(nt, n_wsamples, init_gsize^2)");
  if (!interp_vertices || !interp_weights) return fail(E2E_ERR_INVALID, "null interpolation table");
  if (p->obstacle_mode < E2E_OBST_NONE || p->obstacle_mode > E2E_OBST_DYNAMIC)
    return fail(E2E_ERR_INVALID, "bad obstacle_mode");
  if (!out->u || !out->v || !out->ui || !out->vi || !out->yi || !out->phi || !out->phi_i || !out->phi_yi ||
      !out->s || !out->mask)
    return fail(E2E_ERR_INVALID, "null output array");
  const int64_t G = (int64_t)g * d, G2 = G * G;
  if (G > 46340) return fail(E2E_ERR_UNSUPPORTED, "fine grid too large");
  if ((int64_t)nws * 2 * n > (int64_t)0x7fffffff)
    return fail(E2E_ERR_UNSUPPORTED, "n_wsamples x 2 init_gsize^2 above 2^31 (32-bit solver dimensions)");
  if (!(p->dxy > 0.0) || !(p->dt >= 0.0)) return fail(E2E_ERR_INVALID, "dxy must be positive and dt non-negative");
  cudaStream_t st = (cudaStream_t)stream;
  DeviceScratch scratch(st);

  cudaEvent_t ev[2];
  for (int k = 0; k < 2; ++k) CK(cudaEventCreate(&ev[k]));
  struct EvFree {
    cudaEvent_t* e;
    ~EvFree() { for (int k = 0; k < 2; ++k) cudaEventDestroy(e[k]); }
  } evfree{ev};
  CK(cudaEventRecord(ev[0], st));

  // the interpolation table on the device
  int32_t* dvert = nullptr;
  double* dwgt = nullptr;
  CK(dalloc((void**)&dvert, sizeof(int32_t) * 3 * (size_t)G2, st));
  scratch.add(dvert);
  CK(dalloc((void**)&dwgt, sizeof(double) * 3 * (size_t)G2, st));
  scratch.add(dwgt);
  CK(cudaMemcpyAsync(dvert, interp_vertices, sizeof(int32_t) * 3 * (size_t)G2, cudaMemcpyDefault, st));
  CK(cudaMemcpyAsync(dwgt, interp_weights, sizeof(double) * 3 * (size_t)G2, cudaMemcpyDefault, st));

  // a batch of steps: matrices, reductions' work, coefficients and modes
  const int nb = 3 + 3 * r, nc2[2] = {2 * n, n};
  int kk[2];
  size_t step_doubles = 0;
  for (int q = 0; q < 2; ++q) {
    kk[q] = std::min(std::min(r + 10, kRrMaxK), std::min(nws, nc2[q]));
    if (kk[q] < r) return fail(E2E_ERR_UNSUPPORTED, "n_modes above the range finder's 64 columns");
    step_doubles += (size_t)nws * nc2[q] + nc2[q] + (size_t)nws * r + (size_t)r * nc2[q] + rr_work_doubles(nws, nc2[q], kk[q]);
  }
  // (both fields' matrices of a step are a launch's z index, of which there are 65535)
  int batch = (int)std::min<size_t>(std::min(nt, kMaxBatch), std::max<size_t>(1, (size_t(2) << 30) / (8 * step_doubles)));
  double *work, *Om, *sv, *coarse;
  CK(dalloc((void**)&Om, sizeof(double) * (size_t)2 * n * kRrMaxK, st));
  scratch.add(Om);
  CK(dalloc((void**)&sv, sizeof(double) * 2 * (size_t)nt * r, st));
  scratch.add(sv);
  CK(dalloc((void**)&coarse, sizeof(double) * (size_t)nt * nb * n, st));
  scratch.add(coarse);

  // outputs (device: the caller's arrays; host: staged and copied at the end)
  e2e_env_fields o = *out;
  const size_t b2 = sizeof(float) * (size_t)nt * G2, bm = b2 * r, by = sizeof(float) * (size_t)nt * nws * r;
  if (out_where == E2E_HOST) {
    float** fp[9] = {&o.u, &o.v, &o.ui, &o.vi, &o.yi, &o.phi, &o.phi_i, &o.phi_yi, &o.s};
    const size_t fb[9] = {b2, b2, bm, bm, by, b2, bm, by, b2};
    for (int k = 0; k < 9; ++k) {
      CK(dalloc((void**)fp[k], fb[k], st));
      scratch.add(*fp[k]);
    }
    CK(dalloc((void**)&o.mask, sizeof(int32_t) * (size_t)nt * G2, st));
    scratch.add(o.mask);
  }
  // the last of the buffers: a device with less free memory takes smaller batches, which
  // leave room for a reduction of more columns (enlarge_svd)
  void* room = nullptr;
  for (;; batch = (batch + 1) / 2) {
    const cudaError_t e = dalloc((void**)&work, sizeof(double) * step_doubles * batch, st);
    if (e == cudaSuccess) break;
    if (e != cudaErrorMemoryAllocation || batch == 1) {
      dfree(room, st);
      return cuda_fail(e, "work arrays of the rank reductions");
    }
    cudaGetLastError();
    if (!room) CK(dalloc(&room, sizeof(double) * rr_work_doubles(nws, 2 * n, std::min(kRrMaxK, std::min(nws, 2 * n))), st));
  }
  dfree(room, st);
  scratch.add(work);
  int enlarged = 0;
  for (int t0 = 0; t0 < nt; t0 += batch) {
    const int nbt = std::min(batch, nt - t0);
    RrBatch b{};
    b.nb = nbt;
    b.nws = nws;
    b.r = r;
    b.Om = Om;
    double* p2 = work;
    for (int q = 0; q < 2; ++q) {
      RrKind& K = b.kind[q];
      auto take = [&](size_t each) {
        double* at = p2;
        p2 += each * nbt;
        return at;
      };
      K.X = take((size_t)nws * nc2[q]);
      K.mean = take(nc2[q]);
      K.C = take((size_t)nws * r);
      K.M = take((size_t)r * nc2[q]);
      p2 = rr_carve(&K, nws, nc2[q], kk[q], nbt, p2);
      K.svals = sv + (size_t)(q * nt + t0) * r;
    }
    RealArgs ra{g, nws, t0, p->dt, p->dxy, p->A, p->eps, p->w_lo, p->w_hi, p->wx, 0.5 * kPi, b.kind[0].X, b.kind[1].X};
    const int64_t nr = (int64_t)nws * n;
    k_env_realisations<<<dim3((unsigned)((nr + 255) / 256), (unsigned)nbt), 256, 0, st>>>(ra);
    const unsigned cb = (unsigned)((2 * n + 127) / 128);
    k_env_means<<<dim3(cb, 1, 2 * nbt), 128, 0, st>>>(b);
    k_env_subtract<<<dim3(cb, (unsigned)std::min(nws, 64), 2 * nbt), 128, 0, st>>>(b);
    CK(cudaGetLastError());
    e2e_status s = randomized_svds(b, 2 * nbt, 2, Om, st);
    if (s != E2E_OK) return s;
    // certificates of the batch: residual and mean norms, largest singular value
    std::vector<double> scal[2], S[2];
    for (int q = 0; q < 2; ++q) {
      scal[q].resize(2 * (size_t)nbt);
      S[q].resize((size_t)kk[q] * nbt);
      CK(cudaMemcpyAsync(scal[q].data(), b.kind[q].scal, sizeof(double) * scal[q].size(), cudaMemcpyDeviceToHost, st));
      CK(cudaMemcpyAsync(S[q].data(), b.kind[q].S, sizeof(double) * S[q].size(), cudaMemcpyDeviceToHost, st));
    }
    CK(cudaStreamSynchronize(st));
    for (int q = 0; q < 2; ++q) {
      for (int m = 0; m < nbt; ++m) {
        if (rr_certified(&scal[q][2 * m], S[q][(size_t)kk[q] * m], nws)) continue;
        RrBatch one = b;
        RrKind& K = one.kind[0];
        K = b.kind[q];
        K.X += (int64_t)m * nws * nc2[q];
        K.mean += (int64_t)m * nc2[q];
        K.C += (int64_t)m * nws * r;
        K.M += (int64_t)m * r * nc2[q];
        K.svals += (int64_t)m * r;
        s = enlarge_svd(one, kk[q], Om, st, &enlarged);
        if (s != E2E_OK) return s;
      }
    }
    const int64_t ns = std::max<int64_t>((int64_t)nb * n, (int64_t)nws * r);
    k_env_store<<<dim3((unsigned)((ns + 255) / 256), (unsigned)nbt), 256, 0, st>>>(
        b, n, coarse + (int64_t)t0 * nb * n, o.yi + (int64_t)t0 * nws * r, o.phi_yi + (int64_t)t0 * nws * r);
    CK(cudaGetLastError());
  }
  unsigned int* derr = nullptr;
  CK(dalloc((void**)&derr, sizeof(unsigned int), st));
  scratch.add(derr);
  CK(cudaMemsetAsync(derr, 0, sizeof(unsigned int), st));
  InterpArgs ia{nt, r, n, (int)G2, coarse, dvert, dwgt, derr, o.u, o.v, o.phi, o.ui, o.vi, o.phi_i};
  const int64_t ni = (int64_t)nt * nb * G2;
  k_env_interpolate<<<(unsigned)((ni + 255) / 256), 256, 0, st>>>(ia);
  CK(cudaGetLastError());
  CloudArgs ca{nt, (int)G, p->dxy / d, p->A_sc, p->obstacle_mode, p->obs_upper_row, p->obs_left_col,
               p->obs_width, p->obs_speed_x, p->obs_speed_y, o.s, o.mask};
  const int64_t nc = (int64_t)nt * G2;
  k_env_cloud<<<(unsigned)((nc + 255) / 256), 256, 0, st>>>(ca);
  CK(cudaGetLastError());
  CK(cudaEventRecord(ev[1], st));

  if (out_where == E2E_HOST) {
    float* const* fp[9] = {&o.u, &o.v, &o.ui, &o.vi, &o.yi, &o.phi, &o.phi_i, &o.phi_yi, &o.s};
    float* const hp[9] = {out->u, out->v, out->ui, out->vi, out->yi, out->phi, out->phi_i, out->phi_yi, out->s};
    const size_t fb[9] = {b2, b2, bm, bm, by, b2, bm, by, b2};
    for (int k = 0; k < 9; ++k) CK(cudaMemcpyAsync(hp[k], *fp[k], fb[k], cudaMemcpyDeviceToHost, st));
    CK(cudaMemcpyAsync(out->mask, o.mask, sizeof(int32_t) * (size_t)nt * G2, cudaMemcpyDeviceToHost, st));
  }
  if (svals_out) CK(cudaMemcpyAsync(svals_out, sv, sizeof(double) * 2 * (size_t)nt * r, cudaMemcpyDefault, st));
  unsigned int herr = 0;
  CK(cudaMemcpyAsync(&herr, derr, sizeof(unsigned int), cudaMemcpyDeviceToHost, st));
  CK(cudaStreamSynchronize(st));
  if (herr) return fail(E2E_ERR_INVALID, "interpolation table: a vertex index outside the coarse grid");
  if (stats) {
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, ev[0], ev[1]));
    stats->seconds = ms * 1e-3;
    stats->fine_gsize = (int32_t)G;
    stats->transposed_vel = 0;
    stats->transposed_phi = 0;
    stats->full_svds = enlarged;
  }
  return E2E_OK;
}
