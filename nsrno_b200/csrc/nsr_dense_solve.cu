// Converged solve of the dense path's operator on the device: restarted,
// right-preconditioned GMRES(m) with two classical Gram-Schmidt passes, all
// fields of a frequency (the angles) treated as one vector as the reference's
// solver does (nsrno/wave_solver.py:9-36 used by solve_system,
// nsrno/dense_wave.py:212-220).
//
// Precision: Krylov vectors are complex64; every inner product, norm, the
// Hessenberg matrix, the Givens rotations and the small triangular solve are
// FP64 on the device; the iterate x is complex128 and each cycle restarts from
// the FP64 true residual b - A x of the complex128 operator -- the mixed FP32
// inverse / FP64 residual refinement of nsrno/dense_wave.py:168-191 folded
// into the restart.
//
// Per Arnoldi step j the host enqueues (no synchronisation):
//   rows  v_j = (w - sum_i h'_i v_i) / ||w|| (the correction of the second
//         Gram-Schmidt pass; r / beta for j = 0), stored, and its row FFT
//   cols, rows   z_j = M v_j, the rest of the fixed shifted Laplacian
//   w   = A z_j                 the dense operator (complex64)
//   h   = V_{0..j}^H w          k_dg_dots     (FP64, last CTA sums)
//   w  -= V h, h' = V^H w, ||w||^2   k_dg_gs; the last CTA takes
//         ||w - V h'||^2 = ||w||^2 - sum |h'_i|^2 (V is orthonormal and h' of
//         rounding size) and forms the Givens rotation
// and per cycle the FP64 residual, the back substitution and x += Z y.  The
// host reads one small state record per cycle to decide whether to go on.  The
// transform tables are built once per solve.  Five fields on 160 x 192, 72
// steps: 13.9 ms with 17 launches a step and dots whose blocks summed one value
// at a time (37 us a launch), 5.9 ms in this form (11.0 with the new transforms
// alone).
#include "nsr_internal.cuh"
#include "nsr_device.cuh"
#include "nsr_gs.cuh"
#include "nsr_dense.cuh"

#include <stdlib.h>
#include <string.h>

#define NSR_DG_MAX_M 64
#define NSR_DG_THREADS 256

struct DgState {
  int done;        // 1: converged / budget / non-finite, status is final
  int status;      // NSR_* status
  int used;        // Arnoldi steps of the current cycle
  int stop;        // happy breakdown: the cycle ends after `used` steps
  int steps;       // Arnoldi steps so far
  int cycles;      // cycles started
  int pad0, pad1;
  double bnorm;    // ||b||
  double beta;     // ||r|| at the start of the cycle, then the norm that normalises the next vector
  double rel;      // true relative residual at the start of the last cycle
};

struct DgArgs {
  long long n;         // complex entries of the whole vector (fields x H x W)
  int m;
  int nb;              // CTAs of the vector kernels
  DgState* st;
  int* arrive;
  double* part;        // [2 (m + 1) + 1][CTAs of the launch]
  double2* H;          // [(m + 1) m], column j at H[j (m + 1) + i]
  double* cs;          // [m]
  double2* sn;         // [m]
  double2* gv;         // [m + 1]
  double2* hc;         // [m + 1] coefficients of the first Gram-Schmidt pass
  double2* hc2;        // [m + 1] and of the second
  double2* y;          // [m]
  float2* V;           // [m + 1][n]
  float2* Z;           // [m][n]
  float2* w;           // [n]
  const double2* b;    // [n]
  double2* x;          // [n]
  const double2* ax;   // [n]  A x of the current iterate
  double tol;
  int max_cycles;
};

// Block sum of `v` over NSR_DG_THREADS threads; thread 0 gets the total.
__device__ __forceinline__ double dg_block_sum(double v, double* red) {
  v = warp_sum(v);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int k = 0; k < NSR_DG_THREADS / 32; ++k) t += red[k];
  return t;
}

// Publishes this CTA's `nv` partials and returns true in the last CTA to
// arrive, after summing every CTA's partials in CTA order into tot[0..nv).
__device__ bool dg_arrive(const DgArgs& A, const double* mine, int nv, double* tot) {
  __shared__ int last;
  __shared__ double red[NSR_DG_THREADS / 32];
  if (threadIdx.x == 0) {
    for (int q = 0; q < nv; ++q) A.part[(long long)blockIdx.x * nv + q] = mine[q];
    __threadfence();
    last = atomicAdd(A.arrive, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  for (int q = 0; q < nv; ++q) {
    double s = 0.0;
    for (int b = threadIdx.x; b < (int)gridDim.x; b += NSR_DG_THREADS)
      s += __ldcg(&A.part[(long long)b * nv + q]);
    s = dg_block_sum(s, red);
    if (threadIdx.x == 0) tot[q] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) *A.arrive = 0;
  return true;
}

// ||b||^2 (once per solve).
__global__ void __launch_bounds__(NSR_DG_THREADS) k_dg_bnorm(const __grid_constant__ DgArgs A) {
  __shared__ double red[NSR_DG_THREADS / 32];
  __shared__ double mine[1], tot[1];
  double s = 0.0;
  for (long long e = blockIdx.x * (long long)NSR_DG_THREADS + threadIdx.x; e < A.n;
       e += (long long)gridDim.x * NSR_DG_THREADS) {
    const double2 v = A.b[e];
    s += v.x * v.x + v.y * v.y;
  }
  s = dg_block_sum(s, red);
  if (threadIdx.x == 0) mine[0] = s;
  if (dg_arrive(A, mine, 1, tot) && threadIdx.x == 0) {
    DgState& S = *A.st;
    S.bnorm = sqrt(tot[0]);
    S.done = 0;
    S.status = NSR_NOT_RUN;
    S.steps = 0;
    S.cycles = 0;
  }
}

// r = b - A x (FP64), v_0 = r in complex64, ||r||^2; the last CTA decides
// whether the solve has converged and sets up the cycle.
__global__ void __launch_bounds__(NSR_DG_THREADS) k_dg_residual(const __grid_constant__ DgArgs A) {
  __shared__ double red[NSR_DG_THREADS / 32];
  __shared__ double mine[1], tot[1];
  if (A.st->done) return;
  double s = 0.0;
  float2* v0 = A.V;
  for (long long e = blockIdx.x * (long long)NSR_DG_THREADS + threadIdx.x; e < A.n;
       e += (long long)gridDim.x * NSR_DG_THREADS) {
    const double2 r = A.b[e] - A.ax[e];
    s += r.x * r.x + r.y * r.y;
    v0[e] = to_f(r);
  }
  s = dg_block_sum(s, red);
  if (threadIdx.x == 0) mine[0] = s;
  if (dg_arrive(A, mine, 1, tot) && threadIdx.x == 0) {
    DgState& S = *A.st;
    const double beta = sqrt(tot[0]);
    const double rel = S.bnorm > 0.0 ? beta / S.bnorm : 0.0;
    S.rel = rel;
    S.beta = beta;
    S.used = 0;
    S.stop = 0;
    if (!isfinite(rel)) {
      S.done = 1;
      S.status = NSR_NONFINITE;
    } else if (rel < A.tol || !(S.bnorm > 0.0)) {
      S.done = 1;
      S.status = NSR_CONVERGED;
    } else if (S.cycles >= A.max_cycles) {
      S.done = 1;
      S.status = NSR_ITERATION_BUDGET;
    } else {
      S.cycles += 1;
      for (int i = 0; i <= A.m; ++i) A.gv[i] = make_double2(0.0, 0.0);
      A.gv[0] = make_double2(beta, 0.0);
    }
  }
}

__device__ __forceinline__ bool dg_skip(const DgState& S) { return S.done || S.stop; }

// hc[i] = <v_i, w> for i <= j of one tile of w.
template <int TILE>
__global__ void __launch_bounds__(NSR_GS_THREADS, 4) k_dg_dots(const __grid_constant__ DgArgs A, int j) {
  __shared__ double2 wt[TILE];
  __shared__ double tot[2 * (NSR_DG_MAX_M + 1)];
  if (dg_skip(*A.st)) return;
  const int nv = j + 1, nb = gridDim.x;
  const long long base = (long long)blockIdx.x * TILE;
#pragma unroll
  for (int e = threadIdx.x; e < TILE; e += NSR_GS_THREADS)
    wt[e] = base + e < A.n ? to_d(A.w[base + e]) : make_double2(0.0, 0.0);
  __syncthreads();
  gs_dots<TILE>(wt, A.V, A.n, nv, [&](int e) -> long long { return min(base + e, A.n - 1); }, A.part, nb,
                blockIdx.x);
  if (gs_arrive(A.part, nb, 2 * nv, A.arrive, tot))
    for (int i = threadIdx.x; i < nv; i += NSR_GS_THREADS) A.hc[i] = make_double2(tot[2 * i], tot[2 * i + 1]);
}

// Column j of the Hessenberg matrix, the Givens rotations and the happy breakdown
// (the last CTA).  Rotations G_i = [[c, s], [-conj(s), c]], c real, act on rows i, i+1.
__device__ __noinline__ void dg_finish_step(const DgArgs& A, int j, const double* tot) {
  __shared__ GsColumn k;
  gs_finish_column(k, j, tot, A.hc, A.hc2, A.H + (long long)j * (A.m + 1), A.cs, A.sn, A.gv,
                   [](double2 a, double hn, double* c, double2* s, double2* d) {
                     const double an = sqrt(a.x * a.x + a.y * a.y);
                     const double den = sqrt(an * an + hn * hn);
                     if (den == 0.0) {
                       *c = 1.0; *s = make_double2(0.0, 0.0);
                     } else if (an == 0.0) {
                       *c = 0.0; *s = make_double2(1.0, 0.0);
                     } else {
                       *c = an / den;
                       const double2 ph = make_double2(a.x / an, a.y / an);
                       *s = (hn / den) * ph;   // s = (a / |a|) hn / den
                     }
                     *d = *c * a + hn * *s;   // = (a / |a|) den
                   });
  if (threadIdx.x != 0) return;
  DgState& S = *A.st;
  S.steps += 1;
  S.used = j + 1;
  if (!isfinite(k.norm)) {
    S.done = 1;
    S.status = NSR_NONFINITE;
  } else if (k.norm < 1e-12) {
    S.stop = 1;   // happy breakdown (nsrno/wave_solver.py:29-31)
  }
  S.beta = k.norm;   // normaliser of v_{j+1}
}

// w -= sum_i hc[i] v_i (FP64), then of the new w the second pass's inner products
// and ||w||^2; the last CTA finishes the step.
template <int TILE>
__global__ void __launch_bounds__(NSR_GS_THREADS, 4) k_dg_gs(const __grid_constant__ DgArgs A, int j) {
  __shared__ double2 wt[TILE];
  __shared__ double tot[2 * (NSR_DG_MAX_M + 1) + 1];
  __shared__ double2 h[NSR_DG_MAX_M + 1];
  if (dg_skip(*A.st)) return;
  const int nv = j + 1, nb = gridDim.x;
  for (int i = threadIdx.x; i < nv; i += NSR_GS_THREADS) h[i] = A.hc[i];
  __syncthreads();
  const long long base = (long long)blockIdx.x * TILE;
  constexpr int C = TILE / NSR_GS_THREADS;
  const float2 zero = make_float2(0.f, 0.f);
  double2 acc[C];
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const long long k = base + c * NSR_GS_THREADS + threadIdx.x;
    acc[c] = to_d(k < A.n ? A.w[k] : zero);
  }
  constexpr int B = C >= 8 ? 1 : 8 / C;   // vectors whose loads are in flight together
  for (int i0 = 0; i0 < nv; i0 += B) {
    float2 x[B][C];
#pragma unroll
    for (int b = 0; b < B; ++b)
#pragma unroll
      for (int c = 0; c < C; ++c)
        x[b][c] = A.V[min(i0 + b, nv - 1) * A.n + min(base + c * NSR_GS_THREADS + threadIdx.x, A.n - 1)];
#pragma unroll
    for (int b = 0; b < B; ++b)
      if (i0 + b < nv) {
        const double2 hi = h[i0 + b];
#pragma unroll
        for (int c = 0; c < C; ++c) acc[c] = acc[c] - hi * to_d(x[b][c]);
      }
  }
#pragma unroll
  for (int c = 0; c < C; ++c)   // nodes past the end hold what their clamped loads gave
    if (base + c * NSR_GS_THREADS + threadIdx.x >= A.n) acc[c] = make_double2(0.0, 0.0);
  double nrm = 0.0;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const int e = c * NSR_GS_THREADS + threadIdx.x;
    const float2 f = to_f(acc[c]);
    const double2 d = to_d(f);
    if (base + e < A.n) A.w[base + e] = f;
    wt[e] = d;
    nrm += d.x * d.x + d.y * d.y;
  }
  nrm = gs_block_sum(nrm);   // its barriers also publish wt
  if (threadIdx.x == 0) A.part[(long long)(2 * nv) * nb + blockIdx.x] = nrm;
  gs_dots<TILE>(wt, A.V, A.n, nv, [&](int e) -> long long { return min(base + e, A.n - 1); }, A.part, nb,
                blockIdx.x);
  if (gs_arrive(A.part, nb, 2 * nv + 1, A.arrive, tot)) dg_finish_step(A, j, tot);
}

// v_j and its row transform: the elementwise work runs inside the transform's
// first stage.
template <bool GEN>
__global__ void __launch_bounds__(256, GEN ? 2 : 3) k_dg_rows(const __grid_constant__ DgArgs A, int nz, int nx, PrecTables t,
                                                              float2* __restrict__ W, int rows, int j) {
  extern __shared__ float2 sm[];
  __shared__ double2 c2[NSR_DG_MAX_M];
  const DgState& S = *A.st;
  if (dg_skip(S)) return;
  for (int i = threadIdx.x; i < j; i += blockDim.x) c2[i] = A.hc2[i];
  __syncthreads();
  const float inv = (float)(1.0 / S.beta);
  const int z0 = blockIdx.x * rows;
  const long long off = blockIdx.y * (long long)nz * nx + (long long)z0 * nx;
  // k_dg_residual leaves r in v_0, so for j = 0 src and vj are one buffer
  const float2* src = (j == 0 ? A.V : A.w) + off;
  float2* vj = A.V + (long long)j * A.n + off;
  const float2* __restrict__ V = A.V + off;
  rows_forward<GEN>(sm, min(rows, nz - z0), t.px, W + off, [&](auto tag, int k0, int step, float2* v) {
    constexpr int R = decltype(tag)::value;
    if (j == 0) {
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = inv * src[k0 + q * step];
    } else {
      constexpr int CH = R <= 4 ? R : 1;
#pragma unroll
      for (int c = 0; c < R; c += CH) {
        double2 acc[CH];
#pragma unroll
        for (int q = 0; q < CH; ++q) acc[q] = to_d(src[k0 + (c + q) * step]);
        for (int i = 0; i < j; ++i) {
          const double2 h = c2[i];
#pragma unroll
          for (int q = 0; q < CH; ++q) acc[q] = acc[q] - h * to_d(V[(long long)i * A.n + k0 + (c + q) * step]);
        }
#pragma unroll
        for (int q = 0; q < CH; ++q) v[c + q] = inv * to_f(acc[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < R; ++q) vj[k0 + q * step] = v[q];
  });
}

// y = R^-1 g over the steps of the cycle (FP64).
__global__ void k_dg_solve(const __grid_constant__ DgArgs A) {
  // One warp, column by column: once y_i is known every lane takes its share of
  // the rows above it.
  __shared__ double2 g[NSR_DG_MAX_M];
  const DgState& S = *A.st;
  if (S.done) return;
  const int k = S.used;
  const int m1 = A.m + 1;
  for (int i = threadIdx.x; i < k; i += 32) g[i] = A.gv[i];
  __syncwarp();
  for (int i = k - 1; i >= 0; --i) {
    const double2* col = A.H + (long long)i * m1;
    const double2 y = divc(g[i], col[i]);
    __syncwarp();
    if (threadIdx.x == 0) A.y[i] = y;
    for (int l = threadIdx.x; l < i; l += 32) g[l] = g[l] - col[l] * y;
    __syncwarp();
  }
}

// x += sum_j y_j z_j (FP64).
__global__ void __launch_bounds__(NSR_DG_THREADS) k_dg_xupdate(const __grid_constant__ DgArgs A) {
  __shared__ double2 y[NSR_DG_MAX_M];
  const DgState& S = *A.st;
  if (S.done) return;
  const int k = S.used;
  for (int i = threadIdx.x; i < k; i += NSR_DG_THREADS) y[i] = A.y[i];
  __syncthreads();
  for (long long e = blockIdx.x * (long long)NSR_DG_THREADS + threadIdx.x; e < A.n;
       e += (long long)gridDim.x * NSR_DG_THREADS) {
    double2 acc = A.x[e];
    for (int i = 0; i < k; ++i) acc = acc + y[i] * to_d(A.Z[(long long)i * A.n + e]);
    A.x[e] = acc;
  }
}

// Per-field relative residual ||b_f - A x_f|| / ||b_f|| (the reference's
// max_angle_residual, nsrno/dense_wave.py:221-223); grid (chunks, fields).
__global__ void __launch_bounds__(NSR_DG_THREADS) k_dg_field_residual(const double2* __restrict__ b,
                                                                      const double2* __restrict__ ax, long long nf,
                                                                      double* __restrict__ part, int* arrive,
                                                                      double* __restrict__ out) {
  __shared__ double red[NSR_DG_THREADS / 32];
  __shared__ int last;
  const int f = blockIdx.y;
  double rr = 0.0, bb = 0.0;
  for (long long e = blockIdx.x * (long long)NSR_DG_THREADS + threadIdx.x; e < nf;
       e += (long long)gridDim.x * NSR_DG_THREADS) {
    const double2 bv = b[f * nf + e];
    const double2 r = bv - ax[f * nf + e];
    rr += r.x * r.x + r.y * r.y;
    bb += bv.x * bv.x + bv.y * bv.y;
  }
  rr = dg_block_sum(rr, red);
  bb = dg_block_sum(bb, red);
  double* p = part + 2LL * gridDim.x * f;
  if (threadIdx.x == 0) {
    p[2 * blockIdx.x] = rr;
    p[2 * blockIdx.x + 1] = bb;
    __threadfence();
    last = atomicAdd(&arrive[f], 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last || threadIdx.x != 0) return;
  __threadfence();
  double sr = 0.0, sb = 0.0;
  for (int k = 0; k < (int)gridDim.x; ++k) {
    sr += __ldcg(&p[2 * k]);
    sb += __ldcg(&p[2 * k + 1]);
  }
  out[f] = sb > 0.0 ? sqrt(sr / sb) : sqrt(sr);
  arrive[f] = 0;
}

__global__ void k_dg_zero_ints(int* p, int n) {
  for (int k = threadIdx.x; k < n; k += blockDim.x) p[k] = 0;
}

// ---------------------------------------------------------------------------
// Host side.
// ---------------------------------------------------------------------------
struct DgLayout {
  size_t state, arrive, part, small, V, Z, w, ax, prec_ws, total;
  int nb, tile, nb_gs;
};

static int dg_blocks() {
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return 4 * sms;
}

static DgLayout dg_layout(const NsrDenseGrid* g, int n_fields, int m, int nb) {
  DgLayout L;
  const size_t n = (size_t)g->H * g->W * n_fields;
  size_t off = 0;
  L.nb = nb;
  L.state = off; off += nsr_align(sizeof(DgState));
  L.arrive = off; off += nsr_align(sizeof(int) * (1 + (size_t)n_fields));
  // Gram-Schmidt tiles: 2,048 nodes, or 512 where those would be fewer than three per SM.
  L.tile = (n + 2047) / 2048 >= 3 * 148 ? 2048 : 512;
  L.nb_gs = (int)((n + L.tile - 1) / L.tile);
  size_t parts = (size_t)(2 * (m + 1) + 1) * L.nb_gs;
  if (parts < (size_t)2 * nb) parts = (size_t)2 * nb;
  if (parts < (size_t)2 * n_fields * (nb / n_fields > 8 ? nb / n_fields : 8))
    parts = (size_t)2 * n_fields * (nb / n_fields > 8 ? nb / n_fields : 8);
  L.part = off; off += nsr_align(sizeof(double) * parts);
  L.small = off; off += nsr_align(sizeof(double2) * ((size_t)(m + 1) * m + 5 * (m + 1)) + sizeof(double) * m);
  L.V = off; off += nsr_align(sizeof(float2) * n * (m + 1));
  L.Z = off; off += nsr_align(sizeof(float2) * n * m);
  L.w = off; off += nsr_align(sizeof(float2) * n);
  L.ax = off; off += nsr_align(sizeof(double2) * n);
  L.prec_ws = off; off += nsr_align(nsr_dense_precondition_workspace_size(g, n_fields));
  L.total = off;
  return L;
}

extern "C" size_t nsr_dense_solve_workspace_size(const NsrDenseGrid* grid, int32_t n_fields, int32_t restart) {
  if (!grid || n_fields <= 0 || n_fields > 65535 || restart < 1 || restart > NSR_DG_MAX_M) return 0;
  if (nsr_dense_precondition_workspace_size(grid, n_fields) == 0) return 0;
  return dg_layout(grid, n_fields, restart, dg_blocks()).total;
}

extern "C" int nsr_dense_solve(const NsrDenseGrid* grid, const double* coef, const NsrDenseSolveParams* p,
                               int32_t n_fields, const double* rhs, double* x, double* field_residual,
                               NsrDenseSolveInfo* info, void* workspace, size_t workspace_bytes, void* stream) {
  if (!grid || !coef || !p || !rhs || !x || !workspace || n_fields <= 0 || n_fields > 65535) return NSR_ERR_ARGUMENT;
  const int m = p->restart;
  if (m < 1 || m > NSR_DG_MAX_M || p->max_cycles < 1 || !(p->tolerance > 0) || !(p->k0dx2 > 0) || !(p->shift >= 0))
    return NSR_ERR_ARGUMENT;
  if (nsr_dense_precondition_workspace_size(grid, n_fields) == 0) return NSR_ERR_UNSUPPORTED_SIZE;
  if (grid->h < 1 || grid->w < 1 || grid->pz < 0 || grid->px < 0 || grid->pz + grid->h > grid->H ||
      grid->px + grid->w > grid->W || !(grid->dx > 0))
    return NSR_ERR_ARGUMENT;
  const int nb = dg_blocks();
  const DgLayout L = dg_layout(grid, n_fields, m, nb);
  if (workspace_bytes < L.total) return NSR_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  char* ws = (char*)workspace;
  const long long nf = (long long)grid->H * grid->W;
  DgArgs A;
  memset(&A, 0, sizeof(A));
  A.n = nf * n_fields;
  A.m = m;
  A.nb = nb;
  A.st = (DgState*)(ws + L.state);
  A.arrive = (int*)(ws + L.arrive);
  A.part = (double*)(ws + L.part);
  double2* small = (double2*)(ws + L.small);
  A.H = small;
  A.sn = A.H + (size_t)(m + 1) * m;
  A.gv = A.sn + (m + 1);
  A.hc = A.gv + (m + 1);
  A.hc2 = A.hc + (m + 1);
  A.y = A.hc2 + (m + 1);
  A.cs = (double*)(A.y + (m + 1));
  A.V = (float2*)(ws + L.V);
  A.Z = (float2*)(ws + L.Z);
  A.w = (float2*)(ws + L.w);
  A.b = (const double2*)rhs;
  A.x = (double2*)x;
  A.ax = (const double2*)(ws + L.ax);
  A.tol = p->tolerance;
  A.max_cycles = p->max_cycles;
  const int adj = p->adjoint ? 1 : 0;
  int err = 0;
  // Pinned host record of the solve state, one per host thread, kept for the
  // life of the thread (read once per restart cycle).
  static thread_local DgState* host = nullptr;
  if (!host && cudaHostAlloc((void**)&host, sizeof(DgState), cudaHostAllocDefault) != cudaSuccess) {
    host = nullptr;
    return cudaErrorMemoryAllocation;
  }
  DensePrec M;
  err = nsr_dense_prec_setup(grid, p->k0dx2, p->shift, n_fields, adj, ws + L.prec_ws, st, &M);
  if (err) return err;
  const DenseGeo geo = nsr_dense_geo(grid, p->scal_re, p->scal_im);
  const auto rows_fn = M.gx ? k_dg_rows<true> : k_dg_rows<false>;
  const auto dots_fn = L.tile == 2048 ? k_dg_dots<2048> : k_dg_dots<512>;
  const auto gs_fn = L.tile == 2048 ? k_dg_gs<2048> : k_dg_gs<512>;
#define DG_TRY(expr) do { int e_ = (int)(expr); if (e_) { err = e_; goto done; } } while (0)
  k_dg_zero_ints<<<1, 256, 0, st>>>(A.arrive, 1 + n_fields);
  k_dg_bnorm<<<nb, NSR_DG_THREADS, 0, st>>>(A);
  DG_TRY(cudaGetLastError());
  for (;;) {
    DG_TRY(nsr_dense_apply_geo(geo, coef, n_fields, adj, 1, x, (void*)A.ax, st));
    k_dg_residual<<<nb, NSR_DG_THREADS, 0, st>>>(A);
    DG_TRY(cudaGetLastError());
    DG_TRY(cudaMemcpyAsync(host, A.st, sizeof(DgState), cudaMemcpyDeviceToHost, st));
    DG_TRY(cudaStreamSynchronize(st));
    if (host->done) break;
    for (int j = 0; j < m; ++j) {
      rows_fn<<<M.g_rows, 256, M.row_smem, st>>>(A, grid->H, grid->W, M.t, M.w, M.rows, j);
      nsr_dense_prec_finish(M, A.Z + j * A.n, st);
      DG_TRY(nsr_dense_apply_geo(geo, coef, n_fields, adj, 0, A.Z + j * A.n, A.w, st));
      dots_fn<<<L.nb_gs, NSR_GS_THREADS, 0, st>>>(A, j);
      gs_fn<<<L.nb_gs, NSR_GS_THREADS, 0, st>>>(A, j);
      DG_TRY(cudaGetLastError());
    }
    k_dg_solve<<<1, 32, 0, st>>>(A);
    k_dg_xupdate<<<nb, NSR_DG_THREADS, 0, st>>>(A);
    DG_TRY(cudaGetLastError());
  }
  if (field_residual) {
    dim3 gr(nb / n_fields > 8 ? nb / n_fields : 8, n_fields);
    k_dg_field_residual<<<gr, NSR_DG_THREADS, 0, st>>>(A.b, A.ax, nf, A.part, A.arrive + 1, field_residual);
    DG_TRY(cudaGetLastError());
  }
  if (info) {
    info->status = host->status;
    info->steps = host->steps;
    info->cycles = host->cycles;
    info->reserved = 0;
    info->residual = host->rel;
  }
done:
#undef DG_TRY
  return err;
}
