// Device helpers shared by the Krylov solvers: block reductions and the
// 5-point stencil at an explicit neighbourhood.
#pragma once

#include "nsr_common.cuh"
#include "nsr_internal.cuh"

#define NSR_NPART 8

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-reduce NV doubles into red[0..NV) (valid in thread 0 afterwards).
template <int NV>
__device__ __forceinline__ void block_sum(double* vals, double* red) {
  __shared__ double wsum[32][NSR_NPART];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int q = 0; q < NV; ++q) {
    double s = warp_sum(vals[q]);
    if (lane == 0) wsum[wid][q] = s;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int nw = blockDim.x >> 5;
    for (int q = 0; q < NV; ++q) {
      double s = 0.0;
      for (int w = 0; w < nw; ++w) s += wsum[w][q];
      red[q] = s;
    }
  }
}


// Stencil at an explicit 5-point neighbourhood.  Interior nodes (all six
// stretches equal to one) take the real-flux path.
template <bool ADJ>
__device__ __forceinline__ float2 stencil_pts(const Geo& g, const SysScalars& sc, int i, int j, float a_c, float a_e,
                                              float a_w, float a_s, float a_n, float b_c, float t_c, float2 pc,
                                              float2 pe, float2 pw, float2 ps, float2 pn) {
  const bool inner = i > g.n_pml && i < g.nz - 1 - g.n_pml && j > g.n_pml && j < g.nx - 1 - g.n_pml;
  if (inner) {
    const float e = t_c * (float)sc.fpow;
    const float mb = (float)sc.kh2 * b_c;
    const float2 mass = make_float2(mb * (1.0f - e * e), (ADJ ? -2.0f : 2.0f) * mb * e);
    float2 y = mass * pc;
    y = y + (0.5f * (a_c + a_e)) * (pe - pc);
    y = y + (0.5f * (a_c + a_w)) * (pw - pc);
    y = y + (0.5f * (a_c + a_s)) * (ps - pc);
    y = y + (0.5f * (a_c + a_n)) * (pn - pc);
    return y;
  }
  auto P = [&](int i2, int j2) -> float2 {
    if (i2 == i && j2 == j) return pc;
    if (i2 == i) return j2 > j ? pe : pw;
    return i2 > i ? ps : pn;
  };
  auto Aa = [&](int i2, int j2) -> float {
    if (i2 == i && j2 == j) return a_c;
    if (i2 == i) return j2 > j ? a_e : a_w;
    return i2 > i ? a_s : a_n;
  };
  return stencil<float, ADJ>(g, sc, i, j, b_c, t_c, P, Aa);
}


// The PML profile in float, with 1/n_pml given.
__device__ __forceinline__ float pml_profile_f(float pos, int n, int n_pml, float inv_npml) {
  float f = fmaxf((float)n_pml - pos, pos - (float)(n - 1 - n_pml)) * inv_npml;
  f = fminf(fmaxf(f, 0.0f), 1.0f);
  return f * f;
}

// Complex conj(a) * b accumulated in float (short partial sums of the FP64
// inner products).
__device__ __forceinline__ void dot_acc_f(float& re, float& im, float2 a, float2 b) {
  re = fmaf(a.x, b.x, fmaf(a.y, b.y, re));
  im = fmaf(a.x, b.y, fmaf(-a.y, b.x, im));
}

// ---------------------------------------------------------------------------
// Preconditioner passes shared by the Krylov solvers.
// ---------------------------------------------------------------------------
// Column pass on one field w: forward FFT along z, shifted-Laplace multiply in
// the digit-reversed domain, inverse FFT along z.  Columns [c0, c0+TC) in place.
// Learned spectral multiplier of the 5-point path (the conjugate map of
// nsrno/conditioned_wave.py:112-115): with q2 = 4 (s2z + s2x)/(k0 h)^2, the
// angular term 4 s2x / (4 (s2x + s2z) + h^2) and the basis
// (1, q2/(1+q2), angular, angular q2/(1+q2)),
//   m = exp(tanh(mod0)/2 - i tanh(mod1)/2) / (sym + (k0h)^2 (1 + i s)),
// s = clamp(exp(log_shift), 0.01, 1).  `lp` holds spectral[2][4], log_shift.
struct LearnedSpec {
  float sp[8];
  float shift;
};

__device__ __forceinline__ LearnedSpec load_learned_spec(const float* __restrict__ lp) {
  LearnedSpec L;
#pragma unroll
  for (int k = 0; k < 8; ++k) L.sp[k] = __ldg(&lp[k]);
  L.shift = fminf(fmaxf(expf(__ldg(&lp[8])), 0.01f), 1.0f);
  return L;
}

// tanh from the exponential, 1 - 2 / (e^{2x} + 1); exact at both saturations.
__device__ __forceinline__ float fast_tanh(float x) { return 1.0f - __fdividef(2.0f, __expf(2.0f * x) + 1.0f); }

// The column pass evaluates this once per Fourier point and system, so it uses
// the hardware exponential and sine/cosine (relative error near 1e-6 on these
// bounded arguments): the multiplier is still one fixed function of q, which
// is all the Krylov solvers require of a preconditioner.
__device__ __forceinline__ float2 learned_symbol(const LearnedSpec& L, float s2z, float s2x, float kh2, float h2) {
  const float s4 = 4.0f * (s2z + s2x);
  const float q2 = __fdividef(s4, kh2);
  const float rq = __fdividef(q2, 1.0f + q2);
  const float ang = __fdividef(4.0f * s2x, s4 + h2);
  const float mod0 = L.sp[0] + L.sp[1] * rq + (L.sp[2] + L.sp[3] * rq) * ang;
  const float mod1 = L.sp[4] + L.sp[5] * rq + (L.sp[6] + L.sp[7] * rq) * ang;
  const float mag = __expf(0.5f * fast_tanh(mod0));
  float sn, cs;
  __sincosf(0.5f * fast_tanh(mod1), &sn, &cs);
  // E / D with D = (kh2 - s4) + i kh2 shift
  const float dr = kh2 - s4, di = kh2 * L.shift;
  const float inv = __fdividef(mag, dr * dr + di * di);
  const float er = cs * inv, ei = -sn * inv;
  return make_float2(er * dr + ei * di, ei * dr - er * di);
}

// Column pass of the columns [c0, c0 + TC) of a field with a multiplier:
// `mul(c, z)` is the factor of tile column c at digit-reversed z position,
// including the 1/n of the transform pair; columns at or beyond the grid edge
// are never multiplied.  STAGED (specialised sizes only, a launch shape the
// autotuner can choose): load, every stage in shared memory, store.
template <int TC, bool GEN, bool STAGED, typename MUL>
__device__ __forceinline__ void cols_pass_with(float2* sm, const Geo& g, const PrecTables& tab,
                                               float2* __restrict__ ws, int c0, MUL mul) {
  const int ncol = min(TC, g.nx - c0);
  auto m = [&](int c, int z) -> float2 { return c < ncol ? mul(c, z) : make_float2(0.f, 0.f); };
  if constexpr (STAGED) {
    for (int k = threadIdx.x; k < g.nz * TC; k += blockDim.x) {
      const int z = k / TC, c = k - z * TC;
      sm[k] = c < ncol ? ws[(long long)z * g.nx + c0 + c] : make_float2(0.f, 0.f);
    }
    __syncthreads();
    fft_cols_fused<TC>(sm, tab.pz, m);
    for (int k = threadIdx.x; k < g.nz * TC; k += blockDim.x) {
      const int z = k / TC, c = k - z * TC;
      if (c < ncol) ws[(long long)z * g.nx + c0 + c] = sm[k];
    }
  } else {
    cols_multiply<GEN, TC>(sm, tab.pz, ws + c0, g.nx, ncol, m);
  }
}

// Fixed shifted-Laplace multiplier 1 / (n (-4 (s2z + s2x) + (k0 h)^2 (1 + i shift))).
template <int TC, bool GEN>
__device__ __forceinline__ void cols_pass_fixed(float2* sm, const Geo& g, const PrecTables& tab,
                                                float2* __restrict__ ws, double freq, double shift, int adjoint,
                                                int c0) {
  const SysScalars s = sys_scalars(g, freq);
  const float inv_n = 1.0f / (float)((long long)g.nz * g.nx);
  const float2 shiftc = make_float2((float)s.kh2, (float)(s.kh2 * shift));
  cols_pass_with<TC, GEN, false>(sm, g, tab, ws, c0, [&](int c, int z) -> float2 {
    const float sym = -4.0f * (tab.s2z[z] + tab.s2x[c0 + c]);
    const float2 mul = divc(make_float2(inv_n, 0.f), make_float2(sym + shiftc.x, shiftc.y));
    return adjoint ? conjc(mul) : mul;
  });
}

// Learned multiplier times 1/n at digit-reversed position (z, x) of frequency
// `freq`: the value the batched solver's column pass reads from a system's
// multiplier plane.
__device__ __forceinline__ float2 learned_plane_value(const LearnedSpec& L, const Geo& g, const PrecTables& tab,
                                                      float kh2, int z, int x) {
  const float h2 = (float)(g.h * g.h);
  const float inv_n = 1.0f / (float)((long long)g.nz * g.nx);
  return inv_n * learned_symbol(L, tab.s2z[z], tab.s2x[x], kh2, h2);
}

// Column pass with the learned multiplier evaluated on the fly.
template <int TC, bool GEN>
__device__ __forceinline__ void cols_pass_learned(float2* sm, const Geo& g, const PrecTables& tab,
                                                  float2* __restrict__ ws, double freq, int adjoint, int c0,
                                                  const float* __restrict__ lp) {
  // The spectral parameters go through shared memory so that the fused radix
  // stage keeps its registers for the butterfly.
  __shared__ LearnedSpec Ls;
  if (threadIdx.x == 0) Ls = load_learned_spec(lp);
  __syncthreads();
  const float kh2 = (float)sys_scalars(g, freq).kh2;
  cols_pass_with<TC, GEN, false>(sm, g, tab, ws, c0, [&](int c, int z) -> float2 {
    const float2 mul = learned_plane_value(Ls, g, tab, kh2, z, c0 + c);
    return adjoint ? conjc(mul) : mul;
  });
}

// Diagonal gains of the learned preconditioner.  Plane 0 of a gain pair is the
// inner gain (applied before the FFTs), plane 1 the outer one (after them);
// the adjoint applies the conjugated outer gain first and the conjugated
// inner gain last (nsrno/dense_wave.py:163-164).
struct GainPair {
  const float2* pre;    // multiplies the field before the forward FFT (nullptr: none)
  const float2* post;   // multiplies it after the inverse FFT (nullptr: none)
  bool conj;
};

__device__ __forceinline__ GainPair gain_pair(const float2* gains, int gidx, long long n, int adjoint) {
  GainPair G;
  if (!gains) {
    G.pre = G.post = nullptr;
    G.conj = false;
    return G;
  }
  const float2* base = gains + 2LL * gidx * n;
  G.pre = adjoint ? base + n : base;
  G.post = adjoint ? base : base + n;
  G.conj = adjoint != 0;
  return G;
}

__device__ __forceinline__ float2 gain_mul(const float2* plane, long long idx, bool cj, float2 v) {
  float2 gv = __ldg(&plane[idx]);
  if (cj) gv.y = -gv.y;
  return gv * v;
}

// ---------------------------------------------------------------------------
// FP64 residual tiles shared by the Krylov solvers.
// ---------------------------------------------------------------------------
// One thread per column of a NSR_RES_TZ x NSR_RES_TX tile walks down its rows
// with the north/centre/south values of x and a in registers; the east and west
// neighbours come from the adjacent lanes, the PML factors from the separable
// form of stencil_sep (no division per node).
#define NSR_RES_TZ 8      // rows of one tile: 384 tiles of one 768 x 1024 system
#define NSR_RES_TX 256    // threads of a block
#define NSR_RES_CTAS 1184 // CTAs of one launch over all its slots (8 per SM): most launches find no slot to
                          // serve, and 4,224 idle CTAs cost 8 us more than 1,184
__host__ __device__ inline int res_tiles(int nz, int nx) {
  return ((nz + NSR_RES_TZ - 1) / NSR_RES_TZ) * ((nx + NSR_RES_TX - 1) / NSR_RES_TX);
}
// CTAs per slot of a launch over ns slots.
inline int res_ctas(const NsrGrid* g, int ns) {
  const int tiles = res_tiles(g->nz, g->nx), share = NSR_RES_CTAS / ns > 1 ? NSR_RES_CTAS / ns : 1;
  return tiles < share ? tiles : share;
}

// Tiles blockIdx.x, blockIdx.x + gridDim.x, ... : `P(id)` is x at node id,
// `b_at(idx, i, j)` the h^2-scaled right-hand side, `out(idx, x, b, r)` takes
// each node's x, b and r = b - A x, and `end(tile)` closes a tile.  Sums are
// published by tile: how many CTAs a launch spreads the tiles over follows from
// the slots beside this one, and must not regroup them.
template <bool ADJ, typename XF, typename BF, typename OUT, typename END>
__device__ __forceinline__ void residual_tiles(const Geo& g, const MatPlanes& mat, const SysScalars& sc, XF P,
                                               BF b_at, OUT out, END end) {
  __shared__ RowFactors<double> rowf[NSR_RES_TZ];
  const int nx = g.nx;
  const int nbx = (nx + NSR_RES_TX - 1) / NSR_RES_TX;
  const int n_tiles = res_tiles(g.nz, nx);
  const int lane = threadIdx.x & 31;
  const double2 zero = make_double2(0.0, 0.0);
  for (int tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
    const int rb = tile / nbx, cb = tile - rb * nbx;
    const int z0 = rb * NSR_RES_TZ, z1 = min(z0 + NSR_RES_TZ, g.nz);
    const int j = cb * NSR_RES_TX + threadIdx.x;
    const bool own = j < nx;
    __syncthreads();   // rowf of the tile before has been read
    if (threadIdx.x < z1 - z0) rowf[threadIdx.x] = row_factors<double>(g, sc, z0 + threadIdx.x);
    __syncthreads();
    const ColFactors<double> cf = col_factors<double>(g, sc, j);
    const bool edge_w = lane == 0, edge_e = lane == 31 || j + 1 >= nx;
    // Loads take clamped addresses and are selected afterwards; the south values
    // are loaded one row ahead of their use.
    const int jc = min(j, nx - 1);
    auto row = [&](int i) -> long long { return (long long)min(i, g.nz - 1) * nx + jc; };
    long long idx = row(z0);
    double2 pn = P(z0 > 0 ? idx - nx : idx), pc = P(idx), ps_next = P(row(z0 + 1));
    double an = __ldg(&mat.a64[z0 > 0 ? idx - nx : idx]), ac = __ldg(&mat.a64[idx]);
    double as_next = __ldg(&mat.a64[row(z0 + 1)]);
    if (z0 == 0) { pn = zero; an = 1.0; }
    for (int i = z0; i < z1; ++i, idx += nx) {
      double2 ps = ps_next;
      double as = as_next;
      const long long ahead = row(min(i + 2, z1));
      ps_next = P(ahead);
      as_next = __ldg(&mat.a64[ahead]);
      const double b_c = __ldg(&mat.b64[idx]), t_c = __ldg(&mat.t64[idx]);
      if (i + 1 >= g.nz) { ps = zero; as = 1.0; }
      double2 pw = make_double2(__shfl_up_sync(0xffffffffu, pc.x, 1), __shfl_up_sync(0xffffffffu, pc.y, 1));
      double2 pe = make_double2(__shfl_down_sync(0xffffffffu, pc.x, 1), __shfl_down_sync(0xffffffffu, pc.y, 1));
      double aw = __shfl_up_sync(0xffffffffu, ac, 1), ae = __shfl_down_sync(0xffffffffu, ac, 1);
      if (own && edge_w) {
        pw = j > 0 ? P(idx - 1) : zero;
        aw = j > 0 ? __ldg(&mat.a64[idx - 1]) : 1.0;
      }
      if (own && edge_e) {
        pe = j + 1 < nx ? P(idx + 1) : zero;
        ae = j + 1 < nx ? __ldg(&mat.a64[idx + 1]) : 1.0;
      }
      if (own) {
        const double2 b = b_at(idx, i, j);
        const double2 ax = stencil_sep<double, ADJ>(sc.kh2, sc.fpow, rowf[i - z0], cf, ac, ae, aw, as, an,
                                                    b_c, t_c, pc, pe, pw, ps, pn);
        out(idx, pc, b, b - ax);
      }
      pn = pc;
      pc = ps;
      an = ac;
      ac = as;
    }
    end(tile);
  }
}

// h^2-scaled right-hand side at a node: the given SI field, or the plane-wave
// source on the array row.
__device__ __forceinline__ double2 rhs_at(const Geo& g, double k0, double sin_theta, const float2* rhs, long long idx,
                                          int i, int j) {
  if (rhs) return (g.h * g.h) * to_d(rhs[idx]);
  if (i != g.face) return make_double2(0.0, 0.0);
  const double2 l = source_line(g, k0, sin_theta, j);
  return make_double2(-l.x, -l.y);
}
