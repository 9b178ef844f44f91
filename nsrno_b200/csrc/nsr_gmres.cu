// Restarted right-preconditioned GMRES(m) for a batch of 5-point Helmholtz
// systems -- the reference's `gmres` (nsrno/wave_solver.py:9-36), which
// `solve_frequency` uses and which is the fallback of `solve_system`
// (nsrno/dense_wave.py:212-220).
//
// The systems of a batch share the Arnoldi index j, so j is a launch argument
// and one restart cycle is a fixed sequence of launches, replayed as a CUDA
// graph from the second cycle on.  Per Arnoldi step (5 launches):
//   fwd   v_j = (w - sum_i h'_i v_i) / h_{j,j-1} (the correction of the second
//         Gram-Schmidt pass; r / beta for j = 0), stored and row-transformed
//   cols  column FFT, shifted-Laplace multiply, inverse column FFT
//   rinv  inverse row FFT in place: W = M^-1 v_j
//   inv   5-point stencil: w = A W, and h_i = <v_i, w> (i <= j) of each tile
//   gs    w -= sum_i h_i v_i (classical Gram-Schmidt, pass 1), and of the
//         result h'_i = <v_i, w> (pass 2) and ||w||^2; the last CTA takes
//         ||w - V h'||^2 = ||w||^2 - sum |h'_i|^2 (V is orthonormal and h' is
//         of rounding size), applies the previous Givens rotations to column j
//         and forms the new one, all in FP64 on the device.
// So a step sweeps the basis four times: in fwd, in inv and twice in gs, whose
// second sweep finds the tile in cache while a CTA's tiles of the vectors fit
// (8 steps do, the longest restart does not).  Eleven 768 x 1024 systems, 8 steps: 9.1 ms
// with eight launches a step and one-thread-per-node dots, 4.9 ms in this form.
// At the end of a cycle: back substitution for y (FP64), u = V y fused with
// the forward row FFT, the column and inverse row passes, and an FP64 pass
// that applies x += M^-1 u and recomputes the true residual b - A x.
#include "nsr_internal.cuh"
#include "nsr_device.cuh"
#include "nsr_gs.cuh"

#include <stdlib.h>
#include <string.h>

#define NSR_GMRES_MAX_M 64

struct __align__(16) GSlot {
  int sys;        // system index, -1 when the slot is empty
  int done;       // finished (status written)
  int status;
  int iters;      // Arnoldi steps so far
  int used;       // Arnoldi steps of the current cycle
  int stop;       // the current cycle ends after step `used`
  int xpar;       // which x buffer holds the iterate
  int gidx;       // gain pair of the learned preconditioner
  double bnorm;   // ||b||
  double beta;    // ||r|| at the start of the cycle
  double resid;   // true relative residual at the start of the cycle
  double hlast;   // h_{j+1,j} of the last step (the norm that normalises v_{j+1})
  double freq, angle;
  SysScalars sc;  // scalars of freq (a double pow: formed once, not by every thread)
};

struct GArgs {
  Geo g;
  PrecTables tab;
  MatPlanes mat;
  int m;               // restart length
  int n_slots;
  int nb_max;          // most CTAs per slot of a reducing kernel
  int rows, tc;
  double tol;
  double shift;
  int max_it;
  int adjoint;
  GSlot* slots;
  int* arrive;         // [n_slots]
  double* partials;    // [n_slots][2 (m+1) + 1][nb_max]: value-major, the launch's CTAs contiguous
  double2* H;          // [n_slots][(m+1) m] column-major: H[j*(m+1) + i]
  double* cs;          // [n_slots][m]
  double2* sn;         // [n_slots][m]
  double2* gv;         // [n_slots][m+1]
  double2* hc;         // [n_slots][m+1]  coefficients of the first CGS pass
  double2* hc2;        // [n_slots][m+1]  and of the second
  double2* y;          // [n_slots][m]
  float2* V;           // [n_slots][m+1][n]; plane m: learned multiplier of the slot's system (a cycle's basis ends at m - 1)
  float2* w;           // [n_slots][n]
  float2* W;           // [n_slots][n]   FFT work field
  float2* r;           // [n_slots][n]
  double2* x;          // [n_slots][2][n]
  const double* freq;
  const double* angle;
  const float2* rhs;
  const float2* x0;
  // Learned preconditioner (all null: the fixed shifted-Laplace one).
  const float* lp;
  const float2* gains;
  const int* gain_index;
};

__device__ __forceinline__ bool g_active(const GSlot& S, int j) {
  return S.sys >= 0 && !S.done && !S.stop && j >= S.used;
}

__device__ __forceinline__ double cabs(double2 a) { return sqrt(a.x * a.x + a.y * a.y); }

__device__ __forceinline__ float2* g_sym(const GArgs& A, int slot, long long n) {
  return A.V + ((long long)slot * (A.m + 1) + A.m) * n;
}

__device__ __forceinline__ double* g_part(const GArgs& A, int slot) {
  return A.partials + (long long)slot * (2 * (A.m + 1) + 1) * A.nb_max;
}

// ---------------------------------------------------------------------------
// fwd: v_j from r (j = 0) or w and the second pass's coefficients (j > 0),
// stored in V and transformed by rows.
// ---------------------------------------------------------------------------
template <bool GEN>
__global__ void __launch_bounds__(256, GEN ? 2 : 4) gk_fwd(const __grid_constant__ GArgs A, int j) {
  extern __shared__ float2 sm[];
  const int slot = blockIdx.y;
  const GSlot& S = A.slots[slot];
  if (!g_active(S, j)) return;
  const Geo& g = A.g;
  const long long n = (long long)g.nz * g.nx;
  const int z0 = blockIdx.x * A.rows;
  const int nr = min(A.rows, g.nz - z0);
  const long long off = (long long)z0 * g.nx;
  const float2* __restrict__ src = (j == 0 ? A.r : A.w) + slot * n + off;
  const float scale = (float)(1.0 / (j == 0 ? S.beta : S.hlast));   // both real and positive
  __shared__ float2 c2[NSR_GMRES_MAX_M];
  for (int i = threadIdx.x; i < j; i += blockDim.x) c2[i] = to_f(A.hc2[(long long)slot * (A.m + 1) + i]);
  __syncthreads();
  const float2* __restrict__ V = A.V + (long long)slot * (A.m + 1) * n + off;
  float2* __restrict__ vj = A.V + ((long long)slot * (A.m + 1) + j) * n + off;
  const GainPair G = gain_pair(A.gains, S.gidx, n, A.adjoint);
  rows_forward<GEN>(sm, nr, A.tab.px, A.W + slot * n + off, [&](auto tag, int k0, int step, float2* v) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = src[k0 + q * step];
    for (int i = 0; i < j; ++i) {
      const float2 c = c2[i];
      const float2* __restrict__ Vi = V + i * n;
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = v[q] - c * Vi[k0 + q * step];
    }
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = scale * v[q];
#pragma unroll
    for (int q = 0; q < R; ++q) {
      vj[k0 + q * step] = v[q];
      if (G.pre) v[q] = gain_mul(G.pre, off + k0 + q * step, G.conj, v[q]);
    }
  });
}

// cols for slots active at step j (j < 0: slots that run a cycle-end update)
template <int TC, bool GEN, bool LEARNED>
__global__ void __launch_bounds__(GEN ? 256 : 512, 2) gk_cols(const __grid_constant__ GArgs A, int j) {
  extern __shared__ float2 sm[];
  const int slot = blockIdx.y;
  const GSlot& S = A.slots[slot];
  const bool on = j >= 0 ? g_active(S, j) : (S.sys >= 0 && !S.done && S.used > 0);
  if (!on) return;
  const long long n = (long long)A.g.nz * A.g.nx;
  float2* w = A.W + slot * n;
  const int c0 = blockIdx.x * TC;
  if (LEARNED) {
    const float2* __restrict__ symp = g_sym(A, slot, n);
    const int nx = A.g.nx, adjoint = A.adjoint;
    cols_pass_with<TC, GEN, false>(sm, A.g, A.tab, w, c0, [&](int c, int z) -> float2 {
      const float2 mul = symp[(long long)z * nx + c0 + c];
      return adjoint ? conjc(mul) : mul;
    });
  } else {
    cols_pass_fixed<TC, GEN>(sm, A.g, A.tab, w, S.freq, A.shift, A.adjoint, c0);
  }
}

// The learned multiplier depends on the system's frequency only: it is evaluated
// once per system, in the digit-reversed (z, x) order of the transformed field,
// and read by every column pass (94 us for eleven 768 x 1024 systems with the
// two tanh, the exponential and the sincos evaluated in the pass).
__global__ void __launch_bounds__(256) gk_sym(const __grid_constant__ GArgs A) {
  const GSlot& S = A.slots[blockIdx.y];
  if (S.sys < 0) return;
  const Geo& g = A.g;
  const long long n = (long long)g.nz * g.nx;
  const LearnedSpec L = load_learned_spec(A.lp);
  const float kh2 = (float)S.sc.kh2;
  float2* __restrict__ sym = g_sym(A, blockIdx.y, n);
  for (int z = blockIdx.x; z < g.nz; z += gridDim.x)
    for (int x = threadIdx.x; x < g.nx; x += blockDim.x)
      sym[(long long)z * g.nx + x] = learned_plane_value(L, g, A.tab, kh2, z, x);
}

// rinv: inverse row FFT of W in place, times the outer gain (W becomes M^-1 v_j,
// or M^-1 u at the end of a cycle when j < 0).
template <bool GEN>
__global__ void __launch_bounds__(256, GEN ? 2 : 4) gk_rinv(const __grid_constant__ GArgs A, int j) {
  extern __shared__ float2 sm[];
  const int slot = blockIdx.y;
  const GSlot& S = A.slots[slot];
  const bool on = j >= 0 ? g_active(S, j) : (S.sys >= 0 && !S.done && S.used > 0);
  if (!on) return;
  const Geo& g = A.g;
  const long long n = (long long)g.nz * g.nx;
  const int z0 = blockIdx.x * A.rows;
  const int nr = min(A.rows, g.nz - z0);
  const long long off = (long long)z0 * g.nx;
  float2* Wp = A.W + slot * n + off;
  const GainPair G = gain_pair(A.gains, S.gidx, n, A.adjoint);
  rows_inverse<GEN>(sm, nr, A.tab.px, Wp, [&](int k, float2 v, int, int) {
    Wp[k] = G.post ? gain_mul(G.post, off + k, G.conj, v) : v;
  });
}

// inv: w = A z with z = M^-1 v_j in W, and the tile's inner products with the
// basis.  One thread per column of a TZ x NSR_GST_TX tile walks down its rows
// with the north/centre/south values of z and a in registers.
#define NSR_GST_TX NSR_GS_THREADS
template <bool ADJ, int TZ>
__global__ void __launch_bounds__(NSR_GS_THREADS, 4) gk_inv(const __grid_constant__ GArgs A, int j) {
  extern __shared__ __align__(16) double2 wt[];   // TZ x NSR_GST_TX nodes of w
  __shared__ double tot[2 * (NSR_GMRES_MAX_M + 1)];
  __shared__ RowFactors<float> rowf[TZ];
  const int slot = blockIdx.y;
  const GSlot& S = A.slots[slot];
  if (!g_active(S, j)) return;
  const Geo& g = A.g;
  const long long n = (long long)g.nz * g.nx;
  const int nx = g.nx;
  const int nbx = (nx + NSR_GST_TX - 1) / NSR_GST_TX;
  const int rb = blockIdx.x / nbx, cb = blockIdx.x - rb * nbx;
  const int z0 = rb * TZ, c0 = cb * NSR_GST_TX;
  const int jj = c0 + threadIdx.x;
  {
    // The loads of RB rows are issued together; the north and centre values are
    // carried, east and west come from the adjacent lanes (loads at the warp's
    // ends).
    constexpr int RB = TZ < 4 ? TZ : 4;
    const SysScalars& sc = S.sc;
    const float kh2 = (float)sc.kh2, fpow = (float)sc.fpow;
    if (threadIdx.x < TZ) rowf[threadIdx.x] = row_factors<float>(g, sc, z0 + threadIdx.x);
    const ColFactors<float> cf = col_factors<float>(g, sc, jj);
    __syncthreads();
    const float* __restrict__ ca = A.mat.a32;
    const float* __restrict__ cbp = A.mat.b32;
    const float* __restrict__ ctp = A.mat.t32;
    const float2* __restrict__ z = A.W + slot * n;
    float2* __restrict__ w = A.w + slot * n;
    const float2 zero = make_float2(0.f, 0.f);
    const bool own = jj < nx;
    const int lane = threadIdx.x & 31;
    // lane 0 loads its west, lane 31 its east neighbour
    const int je = lane == 0 ? jj - 1 : jj + 1;
    const bool edge = (lane == 0 || lane == 31) && je >= 0 && je < nx;
    const bool has_e = jj + 1 < nx, has_w = jj > 0;
    const long long i0 = (long long)z0 * nx;
    // Loads take clamped addresses and are selected afterwards: a condition
    // around them would keep them from being issued together.
    const int jc = min(jj, nx - 1), jx = edge ? je : jc;
    const long long up = z0 > 0 ? i0 - nx : i0;
    float2 zu = z[up + jc], zc = z[i0 + jc];
    float a_n = __ldg(&ca[up + jc]), a_c = __ldg(&ca[i0 + jc]);
    if (z0 == 0) { zu = zero; a_n = 1.0f; }
    if (!own) { zc = zero; a_c = 1.0f; }
#pragma unroll
    for (int r0 = 0; r0 < TZ; r0 += RB) {
      float2 zs[RB], zx[RB];
      float as[RB], ax[RB], bb[RB], tt[RB];
#pragma unroll
      for (int q = 0; q < RB; ++q) {
        const int i = z0 + r0 + q;
        const long long ro = (long long)min(i, g.nz - 1) * nx, so = (long long)min(i + 1, g.nz - 1) * nx;
        zs[q] = z[so + jc];
        as[q] = __ldg(&ca[so + jc]);
        bb[q] = __ldg(&cbp[ro + jc]);
        tt[q] = __ldg(&ctp[ro + jc]);
        zx[q] = z[ro + jx];
        ax[q] = __ldg(&ca[ro + jx]);
      }
#pragma unroll
      for (int q = 0; q < RB; ++q)
        if (!own || z0 + r0 + q + 1 >= g.nz) { zs[q] = zero; as[q] = 1.0f; }
#pragma unroll
      for (int q = 0; q < RB; ++q) {
        const int i = z0 + r0 + q;
        float2 zw = make_float2(__shfl_up_sync(0xffffffffu, zc.x, 1), __shfl_up_sync(0xffffffffu, zc.y, 1));
        float2 ze = make_float2(__shfl_down_sync(0xffffffffu, zc.x, 1), __shfl_down_sync(0xffffffffu, zc.y, 1));
        float a_w = __shfl_up_sync(0xffffffffu, a_c, 1), a_e = __shfl_down_sync(0xffffffffu, a_c, 1);
        if (lane == 0) { zw = zx[q]; a_w = ax[q]; }
        if (lane == 31) { ze = zx[q]; a_e = ax[q]; }
        if (!has_e) { ze = zero; a_e = 1.0f; }
        if (!has_w) { zw = zero; a_w = 1.0f; }
        float2 v = zero;
        if (own && i < g.nz) {
          v = stencil_sep<float, ADJ>(kh2, fpow, rowf[r0 + q], cf, a_c, a_e, a_w, as[q], a_n, bb[q], tt[q], zc, ze, zw,
                                      zs[q], zu);
          w[(long long)i * nx + jj] = v;
        }
        wt[(r0 + q) * NSR_GST_TX + threadIdx.x] = to_d(v);
        zu = zc;
        zc = zs[q];
        a_n = a_c;
        a_c = as[q];
      }
    }
  }
  __syncthreads();
  const int nv = j + 1, nb = gridDim.x;
  double* part = g_part(A, slot);
  gs_dots<TZ * NSR_GST_TX>(wt, A.V + (long long)slot * (A.m + 1) * n, n, nv, [&](int e) -> long long {
    return (long long)min(z0 + e / NSR_GST_TX, g.nz - 1) * nx + min(c0 + e % NSR_GST_TX, nx - 1);
  }, part, nb, blockIdx.x);
  if (gs_arrive(part, nb, 2 * nv, &A.arrive[slot], tot))
    for (int i = threadIdx.x; i < nv; i += blockDim.x)
      A.hc[(long long)slot * (A.m + 1) + i] = make_double2(tot[2 * i], tot[2 * i + 1]);
}

// Column j of the Hessenberg matrix, its Givens rotations, and whether the cycle
// stops (the last CTA).
__device__ __noinline__ void g_finish_step(const GArgs& A, GSlot& S, int slot, int j, const double* tot) {
  __shared__ GsColumn k;
  const int m = A.m;
  gs_finish_column(k, j, tot, A.hc + (long long)slot * (m + 1), A.hc2 + (long long)slot * (m + 1),
                   A.H + (long long)slot * (m + 1) * m + j * (m + 1), A.cs + (long long)slot * m,
                   A.sn + (long long)slot * m, A.gv + (long long)slot * (m + 1),
                   [](double2 a, double b, double* c, double2* s, double2* d) {
                     const double aa = cabs(a);
                     const double nu = sqrt(aa * aa + b * b);
                     if (aa == 0.0) {
                       *c = 0.0;
                       *s = make_double2(1.0, 0.0);
                       *d = make_double2(b, 0.0);
                     } else {
                       const double2 ph = make_double2(a.x / aa, a.y / aa);
                       *c = aa / nu;
                       *s = make_double2(ph.x * b / nu, ph.y * b / nu);
                       *d = make_double2(ph.x * nu, ph.y * nu);
                     }
                   });
  if (threadIdx.x != 0) return;
  S.hlast = k.norm;
  S.used = j + 1;
  S.iters += 1;
  const double est = cabs(k.g1) / S.bnorm;
  // Stop the cycle on convergence of the estimate, on a happy breakdown
  // (nsrno/wave_solver.py:31-32), at the restart length or at the budget.
  if (est < 0.5 * A.tol || !(k.norm > 1e-12 * S.beta) || j + 1 == m || S.iters >= A.max_it || !isfinite(est))
    S.stop = 1;
}

// gs: w -= sum_i h_i v_i, then of the new w the second pass's inner products and
// ||w||^2; the last CTA finishes the step.
template <int TILE>
__global__ void __launch_bounds__(NSR_GS_THREADS, 4) gk_gs(const __grid_constant__ GArgs A, int j) {
  extern __shared__ __align__(16) double2 wt[];   // TILE nodes of w
  __shared__ double tot[2 * (NSR_GMRES_MAX_M + 1) + 1];
  __shared__ float2 coef[NSR_GMRES_MAX_M + 1];
  const int slot = blockIdx.y;
  GSlot& S = A.slots[slot];
  if (!g_active(S, j)) return;
  const long long n = (long long)A.g.nz * A.g.nx;
  const int nv = j + 1, nb = gridDim.x;
  for (int i = threadIdx.x; i < nv; i += blockDim.x) coef[i] = to_f(A.hc[(long long)slot * (A.m + 1) + i]);
  __syncthreads();
  constexpr int C = TILE / NSR_GS_THREADS;
  const long long base = (long long)blockIdx.x * TILE;
  float2* __restrict__ w = A.w + slot * n;
  const float2* __restrict__ V = A.V + (long long)slot * (A.m + 1) * n;
  const float2 zero = make_float2(0.f, 0.f);
  float2 acc[C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const long long k = base + c * NSR_GS_THREADS + threadIdx.x;
    acc[c] = k < n ? w[k] : zero;
  }
  for (int i = 0; i < nv; ++i) {
    const float2 h = coef[i];
    const float2* __restrict__ v = V + i * n;
    float2 x[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const long long k = base + c * NSR_GS_THREADS + threadIdx.x;
      x[c] = k < n ? v[k] : zero;
    }
#pragma unroll
    for (int c = 0; c < C; ++c) acc[c] = acc[c] - h * x[c];
  }
  double nrm = 0.0;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int e = c * NSR_GS_THREADS + threadIdx.x;
    const double2 d = to_d(acc[c]);
    if (base + e < n) w[base + e] = acc[c];
    wt[e] = d;
    nrm += d.x * d.x + d.y * d.y;
  }
  double* part = g_part(A, slot);
  nrm = gs_block_sum(nrm);   // its barriers also publish wt
  if (threadIdx.x == 0) part[(long long)(2 * nv) * nb + blockIdx.x] = nrm;
  gs_dots<TILE>(wt, V, n, nv, [&](int e) -> long long { return min(base + e, n - 1); }, part, nb, blockIdx.x);
  if (gs_arrive(part, nb, 2 * nv + 1, &A.arrive[slot], tot)) g_finish_step(A, S, slot, j, tot);
}

// Back substitution R y = g for the slots that ran a cycle.
__global__ void gk_solve(const __grid_constant__ GArgs A) {
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= A.n_slots) return;
  GSlot& S = A.slots[slot];
  if (S.sys < 0 || S.done || S.used == 0) return;
  const int m = A.m, u = S.used;
  const double2* H = A.H + (long long)slot * (m + 1) * m;
  const double2* gv = A.gv + (long long)slot * (m + 1);
  double2* y = A.y + (long long)slot * m;
  for (int i = u - 1; i >= 0; --i) {
    double2 acc = gv[i];
    for (int k = i + 1; k < u; ++k) acc = acc - H[k * (m + 1) + i] * y[k];
    y[i] = divc(acc, H[i * (m + 1) + i]);
  }
}

// u = V y, forward row FFT into W.
template <bool GEN>
__global__ void __launch_bounds__(256, GEN ? 2 : 4) gk_comb(const __grid_constant__ GArgs A) {
  extern __shared__ float2 sm[];
  const int slot = blockIdx.y;
  const GSlot& S = A.slots[slot];
  if (S.sys < 0 || S.done || S.used == 0) return;
  const Geo& g = A.g;
  const long long n = (long long)g.nz * g.nx;
  const int m = A.m, u = S.used;
  __shared__ float2 yc[NSR_GMRES_MAX_M];
  for (int i = threadIdx.x; i < u; i += blockDim.x) yc[i] = to_f(A.y[(long long)slot * m + i]);
  __syncthreads();
  const int z0 = blockIdx.x * A.rows;
  const int nr = min(A.rows, g.nz - z0);
  const long long off = (long long)z0 * g.nx;
  const float2* __restrict__ V = A.V + (long long)slot * (m + 1) * n + off;
  const GainPair G = gain_pair(A.gains, S.gidx, n, A.adjoint);
  rows_forward<GEN>(sm, nr, A.tab.px, A.W + slot * n + off, [&](auto tag, int k0, int step, float2* v) {
    constexpr int R = decltype(tag)::value;
#pragma unroll
    for (int q = 0; q < R; ++q) v[q] = make_float2(0.f, 0.f);
    for (int i = 0; i < u; ++i) {
      const float2 c = yc[i];
      const float2* __restrict__ Vi = V + i * n;
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = v[q] + c * Vi[k0 + q * step];
    }
    if (G.pre) {
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = gain_mul(G.pre, off + k0 + q * step, G.conj, v[q]);
    }
  });
}

// FP64 true residual.  init = 1: x = x0 (or 0); init = 0: x += M^-1 V y.
template <bool ADJ>
__global__ void __launch_bounds__(NSR_RES_TX) gk_res(const __grid_constant__ GArgs A, int init) {
  __shared__ double tot[2];
  const int slot = blockIdx.y;
  GSlot& S = A.slots[slot];
  if (S.sys < 0 || S.done) return;
  if (!init && S.used == 0) return;
  const Geo& g = A.g;
  const long long n = (long long)g.nz * g.nx;
  const float2* zW = A.W + slot * n;   // M^-1 u after the rinv pass
  const SysScalars sc = S.sc;
  const double2* xo = A.x + (2LL * slot + S.xpar) * n;
  double2* xn = A.x + (2LL * slot + (S.xpar ^ 1)) * n;
  const float2* x0 = (init && A.x0) ? A.x0 + (long long)S.sys * n : nullptr;
  const float2* rhs = A.rhs ? A.rhs + (long long)S.sys * n : nullptr;
  const double st = sin(S.angle);
  float2* r = A.r + slot * n;
  double rr = 0.0, bb = 0.0;
  double* part = g_part(A, slot);
  const int nb = res_tiles(g.nz, g.nx);
  residual_tiles<ADJ>(
      g, A.mat, sc,
      [&](long long id) -> double2 {
        if (init) return x0 ? to_d(x0[id]) : make_double2(0.0, 0.0);
        return xo[id] + to_d(zW[id]);
      },
      [&](long long idx, int i, int jj) { return rhs_at(g, sc.k0, st, rhs, idx, i, jj); },
      [&](long long idx, double2 x, double2 b, double2 res) {
        xn[idx] = x;
        r[idx] = to_f(res);
        rr += res.x * res.x + res.y * res.y;
        bb += b.x * b.x + b.y * b.y;
      },
      [&](int tile) {
        rr = gs_block_sum(rr);
        bb = gs_block_sum(bb);
        if (threadIdx.x == 0) {
          part[tile] = rr;
          part[nb + tile] = bb;
        }
        rr = bb = 0.0;
      });
  if (gs_arrive(part, nb, 2, &A.arrive[slot], tot) && threadIdx.x == 0) {
    rr = tot[0];
    bb = tot[1];
    S.xpar ^= 1;
    if (init) S.bnorm = sqrt(bb);
    const double rn = sqrt(rr);
    const double rel = S.bnorm > 0.0 ? rn / S.bnorm : 0.0;
    S.resid = rel;
    S.used = 0;
    S.stop = 0;
    S.beta = rn;
    if (!(S.bnorm > 0.0)) {
      S.done = 1;
      S.status = isfinite(S.bnorm) ? NSR_CONVERGED : NSR_NONFINITE;
      S.resid = 0.0;
    } else if (!isfinite(rel)) {
      S.done = 1;
      S.status = NSR_NONFINITE;
    } else if (rel < A.tol) {
      S.done = 1;
      S.status = NSR_CONVERGED;
    } else if (S.iters >= A.max_it) {
      S.done = 1;
      S.status = NSR_ITERATION_BUDGET;
    } else {
      double2* gv = A.gv + (long long)slot * (A.m + 1);
      gv[0] = make_double2(rn, 0.0);
    }
    __threadfence();
  }
}

// Outputs of one batch: IQ, residual, iterations, status, fields.
__global__ void gk_emit(const __grid_constant__ GArgs A, double2* iq, const int* rx, int n_rx, double* residual, int* iterations,
                        int* status, void* fields, int fields_fp64) {
  const int slot = blockIdx.y;
  const GSlot& S = A.slots[slot];
  if (S.sys < 0) return;
  const long long n = (long long)A.g.nz * A.g.nx;
  const double2* x = A.x + (2LL * slot + S.xpar) * n;
  const bool zero = !(S.bnorm > 0.0);
  if (blockIdx.x == 0) {
    for (int k = threadIdx.x; k < n_rx; k += blockDim.x) {
      const int idx = rx[k];
      const bool ok = idx >= 0 && (long long)idx < n;
      iq[(long long)S.sys * n_rx + k] = !ok ? make_double2(NAN, NAN) : (zero ? make_double2(0.0, 0.0) : x[idx]);
    }
    if (threadIdx.x == 0) {
      residual[S.sys] = S.resid;
      iterations[S.sys] = S.iters;
      status[S.sys] = S.done ? S.status : NSR_ITERATION_BUDGET;
    }
  }
  if (fields) {
    for (long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
      const double2 v = zero ? make_double2(0.0, 0.0) : x[k];
      if (fields_fp64) ((double2*)fields)[(long long)S.sys * n + k] = v;
      else ((float2*)fields)[(long long)S.sys * n + k] = to_f(v);
    }
  }
}

__global__ void gk_load(const __grid_constant__ GArgs A, int first, int count, const double* freq, const double* angle) {
  const int slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= A.n_slots) return;
  GSlot S;
  memset(&S, 0, sizeof(S));
  if (slot < count) {
    S.sys = first + slot;
    S.gidx = A.gain_index ? A.gain_index[first + slot] : first + slot;
    S.freq = freq[first + slot];
    S.angle = angle ? angle[first + slot] : 0.0;
    S.sc = sys_scalars(A.g, S.freq);
  } else {
    S.sys = -1;
    S.done = 1;
  }
  A.slots[slot] = S;
  A.arrive[slot] = 0;
}

__global__ void gk_count(const __grid_constant__ GArgs A, int* remaining) {
  __shared__ int cnt;
  if (threadIdx.x == 0) cnt = 0;
  __syncthreads();
  for (int s = threadIdx.x; s < A.n_slots; s += blockDim.x)
    if (A.slots[s].sys >= 0 && !A.slots[s].done) atomicAdd(&cnt, 1);
  __syncthreads();
  if (threadIdx.x == 0) *remaining = cnt;
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
struct GLayout {
  size_t tables, slots, arrive, count, partials, H, cs, sn, gv, hc, hc2, y, V, w, W, r, x, total;
  int tz, tile, nb_st, nb_gs, nb_max;   // stencil rows and Gram-Schmidt nodes of a CTA, CTAs per slot
};

static GLayout g_layout(const NsrGrid* g, int n_slots, int m) {
  GLayout L;
  const size_t n = (size_t)g->nz * g->nx;
  // Tall tiles (8 rows, 2,048 nodes) amortise the reductions; a grid of fewer than
  // 64 of them takes 2-row tiles of 512 nodes.  Tiles group the partial sums, so
  // the rule looks at the grid alone and not at the slots of a call.  Cycles of 8
  // steps with 1 / 4 / 11 systems, us, tall against short: 768 x 1024
  // 1003 / 2139 / 4564 and 1161 / 2495 / 5503, 243 x 729 849 / 1192 / 2294 and
  // 856 / 1271 / 2487, 256 x 256 (32 tall tiles) 758 / 784 / 940 and
  // 741 / 779 / 1016, 128 x 192 (16) 711 / 729 / 846 and 690 / 713 / 849.
  const int bx = (g->nx + NSR_GST_TX - 1) / NSR_GST_TX;
  const bool tall = (long long)bx * ((g->nz + 7) / 8) >= 64;
  L.tz = tall ? 8 : 2;
  L.tile = L.tz * NSR_GST_TX;
  L.nb_st = bx * ((g->nz + L.tz - 1) / L.tz);
  L.nb_gs = (int)((n + L.tile - 1) / L.tile);
  L.nb_max = L.nb_st > L.nb_gs ? L.nb_st : L.nb_gs;
  if (res_tiles(g->nz, g->nx) > L.nb_max) L.nb_max = res_tiles(g->nz, g->nx);
  size_t off = 0;
  L.tables = off; off += nsr_align(nsr_prec_table_bytes(g));
  L.slots = off; off += nsr_align(sizeof(GSlot) * n_slots);
  L.arrive = off; off += nsr_align(sizeof(int) * n_slots);
  L.count = off; off += nsr_align(sizeof(int));
  L.partials = off; off += nsr_align(sizeof(double) * (size_t)n_slots * L.nb_max * (2 * (m + 1) + 1));
  L.H = off; off += nsr_align(sizeof(double2) * (size_t)n_slots * (m + 1) * m);
  L.cs = off; off += nsr_align(sizeof(double) * (size_t)n_slots * m);
  L.sn = off; off += nsr_align(sizeof(double2) * (size_t)n_slots * m);
  L.gv = off; off += nsr_align(sizeof(double2) * (size_t)n_slots * (m + 1));
  L.hc = off; off += nsr_align(sizeof(double2) * (size_t)n_slots * (m + 1));
  L.hc2 = off; off += nsr_align(sizeof(double2) * (size_t)n_slots * (m + 1));
  L.y = off; off += nsr_align(sizeof(double2) * (size_t)n_slots * m);
  L.V = off; off += nsr_align(sizeof(float2) * n * (m + 1) * n_slots);
  L.w = off; off += nsr_align(sizeof(float2) * n * n_slots);
  L.W = off; off += nsr_align(sizeof(float2) * n * n_slots);
  L.r = off; off += nsr_align(sizeof(float2) * n * n_slots);
  L.x = off; off += nsr_align(sizeof(double2) * n * 2 * n_slots);
  L.total = off;
  return L;
}

extern "C" size_t nsr_gmres_workspace_size(const NsrGrid* grid, int32_t n_slots, int32_t restart) {
  if (nsr_check_grid(grid, true) || n_slots <= 0 || n_slots > 65535 || restart < 1 || restart > NSR_GMRES_MAX_M)
    return 0;
  return g_layout(grid, n_slots, restart).total;
}

extern "C" int nsr_gmres_batched(const NsrGrid* grid, const void* material, const double* freq_hz,
                                 const double* angle_rad, int32_t n_systems, const float* rhs, const float* x0,
                                 const int32_t* rx_index, int32_t n_rx, const NsrGmresParams* params,
                                 void* workspace, size_t workspace_bytes, double* iq, double* residual,
                                 int32_t* iterations, int32_t* status, void* fields, void* stream) {
  int err = nsr_check_grid(grid, true);
  if (err) return err;
  if (!params || !material || n_systems < 0 || n_rx < 0) return NSR_ERR_ARGUMENT;
  if (n_systems == 0) return 0;   // an empty batch touches no buffer
  if (!freq_hz || (n_rx > 0 && (!rx_index || !iq))) return NSR_ERR_ARGUMENT;
  if (!rhs && !angle_rad) return NSR_ERR_ARGUMENT;
  if (!residual || !iterations || !status || !workspace) return NSR_ERR_ARGUMENT;
  const int m = params->restart, n_slots = params->n_slots;
  if (m < 1 || m > NSR_GMRES_MAX_M || n_slots <= 0 || n_slots > 65535 || !(params->tolerance > 0) ||
      params->max_iterations <= 0 || !(params->shift >= 0))
    return NSR_ERR_ARGUMENT;
  if (params->learned && !params->learned->params) return NSR_ERR_ARGUMENT;
  if (n_systems == 0) return 0;
  const GLayout L = g_layout(grid, n_slots, m);
  if (workspace_bytes < L.total) return NSR_ERR_WORKSPACE;
  const size_t n = (size_t)grid->nz * grid->nx;
  cudaStream_t caller = (cudaStream_t)stream;
  cudaStream_t st = nullptr;
  cudaEvent_t ev_in = nullptr, ev_out = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  int remaining_host = 0;
  cudaError_t ce;
#define NSR_TRY(x) do { ce = (x); if (ce != cudaSuccess) { err = (int)ce; goto cleanup; } } while (0)
  {
    NSR_TRY(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    NSR_TRY(cudaEventCreateWithFlags(&ev_in, cudaEventDisableTiming));
    NSR_TRY(cudaEventCreateWithFlags(&ev_out, cudaEventDisableTiming));
    NSR_TRY(cudaEventRecord(ev_in, caller));
    NSR_TRY(cudaStreamWaitEvent(st, ev_in, 0));
    err = nsr_check_learned(params->learned, n_systems, st);
    if (err) goto cleanup;
    char* ws = (char*)workspace;
    GArgs A;
    memset(&A, 0, sizeof(A));
    A.g = make_geo(*grid);
    err = nsr_prec_setup(grid, &A.tab, ws + L.tables, st);
    if (err) goto cleanup;
    A.mat = nsr_planes(material, (long long)n);
    A.m = m;
    A.n_slots = n_slots;
    A.nb_max = L.nb_max;
    A.rows = nsr_rows_per_cta(grid, n_slots);
    A.tc = nsr_cols_tc(grid, n_slots);
    A.tol = params->tolerance;
    A.shift = params->shift;
    A.max_it = params->max_iterations;
    A.adjoint = params->adjoint ? 1 : 0;
    A.slots = (GSlot*)(ws + L.slots);
    A.arrive = (int*)(ws + L.arrive);
    int* remaining = (int*)(ws + L.count);
    A.partials = (double*)(ws + L.partials);
    A.H = (double2*)(ws + L.H);
    A.cs = (double*)(ws + L.cs);
    A.sn = (double2*)(ws + L.sn);
    A.gv = (double2*)(ws + L.gv);
    A.hc = (double2*)(ws + L.hc);
    A.hc2 = (double2*)(ws + L.hc2);
    A.y = (double2*)(ws + L.y);
    A.V = (float2*)(ws + L.V);
    A.w = (float2*)(ws + L.w);
    A.W = (float2*)(ws + L.W);
    A.r = (float2*)(ws + L.r);
    A.x = (double2*)(ws + L.x);
    A.freq = freq_hz;
    A.angle = rhs ? nullptr : angle_rad;
    A.rhs = (const float2*)rhs;
    A.x0 = (const float2*)x0;
    if (params->learned) {
      A.lp = params->learned->params;
      A.gains = (const float2*)params->learned->gains;
      A.gain_index = params->learned->gain_index;
    }

    const size_t fwd_smem = sizeof(float2) * A.rows * nsr_row_stride(grid->nx);
    const size_t col_smem = sizeof(float2) * (size_t)grid->nz * A.tc;
    const bool gx = !nsr_specialised(grid->nx), gz = !nsr_specialised(grid->nz);
    const auto fwd_fn = gx ? gk_fwd<true> : gk_fwd<false>;
    const auto rinv_fn = gx ? gk_rinv<true> : gk_rinv<false>;
    const auto comb_fn = gx ? gk_comb<true> : gk_comb<false>;
    const auto cols_fn =
        A.lp ? (A.tc == 16 ? (gz ? gk_cols<16, true, true> : gk_cols<16, false, true>)
                           : (gz ? gk_cols<8, true, true> : gk_cols<8, false, true>))
             : (A.tc == 16 ? (gz ? gk_cols<16, true, false> : gk_cols<16, false, false>)
                           : (gz ? gk_cols<8, true, false> : gk_cols<8, false, false>));
    NSR_TRY(cudaFuncSetAttribute((const void*)fwd_fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fwd_smem));
    NSR_TRY(cudaFuncSetAttribute((const void*)comb_fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fwd_smem));
    NSR_TRY(cudaFuncSetAttribute((const void*)cols_fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)col_smem));
    NSR_TRY(cudaFuncSetAttribute((const void*)rinv_fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fwd_smem));

    const dim3 g_rows((grid->nz + A.rows - 1) / A.rows, n_slots);
    const dim3 g_col((grid->nx + A.tc - 1) / A.tc, n_slots);
    const dim3 g_res(res_ctas(grid, n_slots), n_slots);
    const dim3 g_st(L.nb_st, n_slots);
    const dim3 g_gs(L.nb_gs, n_slots);
    const bool tall = L.tz == 8;
    const auto inv_fn = A.adjoint ? (tall ? gk_inv<true, 8> : gk_inv<true, 2>) : (tall ? gk_inv<false, 8> : gk_inv<false, 2>);
    const auto gs_fn = tall ? gk_gs<8 * NSR_GST_TX> : gk_gs<2 * NSR_GST_TX>;
    const size_t gs_smem = sizeof(double2) * L.tile;
    auto cols = [&](int j) {
      cols_fn<<<g_col, nsr_cols_threads(gz), col_smem, st>>>(A, j);
    };
    auto res = [&](int init) {
      if (A.adjoint) gk_res<true><<<g_res, NSR_RES_TX, 0, st>>>(A, init);
      else gk_res<false><<<g_res, NSR_RES_TX, 0, st>>>(A, init);
    };

    // One restart cycle.
    auto cycle = [&]() -> cudaError_t {
      for (int j = 0; j < m; ++j) {
        fwd_fn<<<g_rows, 256, fwd_smem, st>>>(A, j);
        cols(j);
        rinv_fn<<<g_rows, 256, fwd_smem, st>>>(A, j);
        inv_fn<<<g_st, NSR_GS_THREADS, gs_smem, st>>>(A, j);
        gs_fn<<<g_gs, NSR_GS_THREADS, gs_smem, st>>>(A, j);
      }
      gk_solve<<<(n_slots + 127) / 128, 128, 0, st>>>(A);
      comb_fn<<<g_rows, 256, fwd_smem, st>>>(A);
      cols(-1);
      rinv_fn<<<g_rows, 256, fwd_smem, st>>>(A, -1);
      res(0);
      gk_count<<<1, 256, 0, st>>>(A, remaining);
      return cudaGetLastError();
    };

    // The first cycle of the call is launched directly, so that a solve of one
    // cycle (a warm start) never waits for a graph to be built; later ones
    // replay it.
    const int max_cycles = (params->max_iterations + m - 1) / m + 1;
    bool first_cycle = true;
    for (int first = 0; first < n_systems; first += n_slots) {
      const int count = (n_systems - first) < n_slots ? (n_systems - first) : n_slots;
      gk_load<<<(n_slots + 127) / 128, 128, 0, st>>>(A, first, count, freq_hz, A.angle);
      if (A.lp) gk_sym<<<dim3(grid->nz < 256 ? grid->nz : 256, n_slots), 256, 0, st>>>(A);
      NSR_TRY(cudaGetLastError());
      res(1);
      NSR_TRY(cudaGetLastError());
      for (int cyc = 0; cyc < max_cycles; ++cyc) {
        if (first_cycle) {
          NSR_TRY(cycle());
          first_cycle = false;
        } else {
          if (!exec) {
            NSR_TRY(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
            ce = cycle();
            const cudaError_t ce2 = cudaStreamEndCapture(st, &graph);
            if (ce == cudaSuccess) ce = ce2;
            if (ce != cudaSuccess) { err = (int)ce; goto cleanup; }
            NSR_TRY(cudaGraphInstantiate(&exec, graph, 0));
          }
          NSR_TRY(cudaGraphLaunch(exec, st));
        }
        NSR_TRY(cudaMemcpyAsync(&remaining_host, remaining, sizeof(int), cudaMemcpyDeviceToHost, st));
        NSR_TRY(cudaStreamSynchronize(st));
        if (remaining_host == 0) break;
      }
      dim3 g_emit(fields ? 148 : 1, n_slots);
      gk_emit<<<g_emit, 256, 0, st>>>(A, (double2*)iq, rx_index, n_rx, residual, iterations, status, fields,
                                      params->fields_fp64);
      NSR_TRY(cudaGetLastError());
    }
    NSR_TRY(cudaEventRecord(ev_out, st));
    NSR_TRY(cudaStreamWaitEvent(caller, ev_out, 0));
  }
cleanup:
  if (st) cudaStreamSynchronize(st);
  if (exec) cudaGraphExecDestroy(exec);
  if (graph) cudaGraphDestroy(graph);
  if (ev_in) cudaEventDestroy(ev_in);
  if (ev_out) cudaEventDestroy(ev_out);
  if (st) cudaStreamDestroy(st);
#undef NSR_TRY
  return err;
}
