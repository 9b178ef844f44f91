// The dense path's operator (nsrno/conditioned_wave.py:52-80, projected as in
// nsrno/dense_wave.py:66-68) and its analytic adjoint (nsrno/dense_wave.py:70-82),
// evaluated as a direct radius-4 staggered stencil instead of 11 FFTs.
//
// The reference evaluates the 8th-order staggered derivative D (forward, at
// n + 1/2) and its negative adjoint (divergence) by FFT on a padded grid.  The
// field is masked to the native region and the padding is at least 8 nodes
// wide, so the periodic FFT evaluation equals the direct stencil with zero
// values outside the grid:
//   (D p)[n]     = (1/dx) sum_k a_k (p[n+1+k] - p[n-k])
//   (-D^H f)[n]  = (1/dx) sum_k a_k (f[n+k]   - f[n-1-k])
// with a = (1225/1024, -245/3072, 49/5120, -5/7168).
// One kernel forms the staggered fluxes of a tile in shared memory and takes
// their divergence.
#include "nsr_dense.cuh"

#include <string.h>

struct DenseCoef {
  // planes [H][W]
  const double* ax;
  const double* az;
  const double2* mass;
  // profiles along x [W] and z [H]
  const double2 *svx, *gvx, *lx, *rx;
  const double2 *svz, *gvz, *lz, *rz;
};

__host__ __device__ inline size_t dense_coef_doubles(int H, int W) { return (size_t)H * W * 4 + 8 * (size_t)W + 8 * (size_t)H; }

__host__ __device__ inline DenseCoef dense_unpack(const double* c, int H, int W) {
  DenseCoef d;
  const size_t n = (size_t)H * W;
  d.ax = c;
  d.az = c + n;
  d.mass = (const double2*)(c + 2 * n);
  const double2* px = (const double2*)(c + 4 * n);
  d.svx = px; d.gvx = px + W; d.lx = px + 2 * W; d.rx = px + 3 * W;
  const double2* pz = px + 4 * W;
  d.svz = pz; d.gvz = pz + H; d.lz = pz + 2 * H; d.rz = pz + 3 * H;
  return d;
}

template <typename T> struct DC;
template <> struct DC<float> { typedef float2 C; static __device__ C from(double2 a) { return make_float2((float)a.x, (float)a.y); } };
template <> struct DC<double> { typedef double2 C; static __device__ C from(double2 a) { return a; } };

__device__ __forceinline__ bool dense_inside(const DenseGeo& g, int i, int j) {
  return i >= g.pz && i < g.pz + g.h && j >= g.px && j < g.px + g.w;
}

// One pass over a TZ x DA_TX tile.  The x part of a node needs p along its row
// only and the z part along its column only, 7 nodes each way: the tile of
// mask p with those halos is staged in shared memory, the staggered fluxes of
// the tile (3 or 4 nodes beyond it) are formed there, and their divergence is
// taken from there, so that HBM carries p, y and the coefficients once.  (Two
// passes with four flux planes through memory moved 80 B per node and field.)
//   Forward: X = ax svx D_x(mask p), likewise Z;
//            y = mask (scal (lx div X + rx div(gvx X) + lz div Z + rz div(gvz Z)) + mass p) + (1 - mask) p.
//   Adjoint: w = conj(scal) mask p;
//            X = conj(ax svx) (-D_x(conj(lx) w) - conj(gvx) D_x(conj(rx) w)), likewise Z;
//            y = mask (-div X - div Z + conj(mass) p) + (1 - mask) p.
// Off the PML gv = sv = 1, the left factor is zero and the right one is one
// constant: a tile all of whose profiles say so takes a shorter form.
// Eleven complex64 fields on 1056 x 1216: 695 us in two passes, 316 us here,
// bound by its shared-memory reads (about 33 a node).
#define DA_TX 64
#define DA_THREADS 256
#define DA_R 7    // reach of the two staggered stencils

template <typename T, int TZ>
struct DenseTile {
  typedef typename DC<T>::C C;
  C p[TZ + 2 * DA_R][DA_TX + 2 * DA_R];   // mask p; rows and columns start at (z0 - 7, c0 - 7)
  C x[TZ][DA_TX + 7];                     // X at columns c0 - 4 .. c0 + DA_TX + 2
  C z[TZ + 7][DA_TX];                     // Z at rows z0 - 4 .. z0 + TZ + 2
  C prx[4][DA_TX + 2 * DA_R];             // sv, gv, l, r of the columns
  C prz[4][TZ + 2 * DA_R];                // and of the rows
};

template <typename C>
__device__ __forceinline__ bool is_real(C v, double re) { return v.x == (decltype(v.x))re && v.y == 0; }

template <typename T, bool ADJ, int TZ>
__global__ void __launch_bounds__(DA_THREADS) k_dense_apply(DenseGeo g, const double* __restrict__ coef,
                                                            const typename DC<T>::C* __restrict__ p,
                                                            typename DC<T>::C* __restrict__ y, int nf) {
  typedef typename DC<T>::C C;
  extern __shared__ __align__(16) unsigned char da_smem[];
  DenseTile<T, TZ>& t = *reinterpret_cast<DenseTile<T, TZ>*>(da_smem);
  const DenseCoef dc = dense_unpack(coef, g.H, g.W);
  const long long n = (long long)g.H * g.W;
  // The fields run fastest, so the coefficients of a tile come from L2 after
  // the first field.
  const int f = blockIdx.x % nf, tile = blockIdx.x / nf;
  const int nbx = (g.W + DA_TX - 1) / DA_TX;
  const int z0 = (tile / nbx) * TZ, c0 = (tile % nbx) * DA_TX;
  const C* pf = p + (long long)f * n;
  C* yf = y + (long long)f * n;
  const C zero = cx<C>(T(0), T(0));
  const int tid = threadIdx.x;
  // A tile with no node of the native region copies.
  const bool touched = z0 < g.pz + g.h && z0 + TZ > g.pz && c0 < g.px + g.w && c0 + DA_TX > g.px;
  if (!touched) {
    for (int k = tid; k < TZ * DA_TX; k += DA_THREADS) {
      const int i = z0 + k / DA_TX, j = c0 + k % DA_TX;
      if (i < g.H && j < g.W) yf[(long long)i * g.W + j] = pf[(long long)i * g.W + j];
    }
    return;
  }
  constexpr int PW = DA_TX + 2 * DA_R, PH = TZ + 2 * DA_R;
  // The corners of the halo are never read.
  for (int k = tid; k < PW * PH; k += DA_THREADS) {
    const int r = k / PW, c = k - r * PW;
    const int i = z0 - DA_R + r, j = c0 - DA_R + c;
    const bool cross = (r >= DA_R && r < DA_R + TZ) || (c >= DA_R && c < DA_R + DA_TX);
    if (cross) t.p[r][c] = i >= 0 && i < g.H && j >= 0 && j < g.W && dense_inside(g, i, j)
                               ? pf[(long long)i * g.W + j] : zero;
  }
  bool plain_x = true, plain_z = true;
  C r0x = zero, r0z = zero;   // the right factors of the first column and row
  {
    const int jm = min(max(c0, 0), g.W - 1), im = min(max(z0, 0), g.H - 1);
    r0x = DC<T>::from(dc.rx[jm]);
    r0z = DC<T>::from(dc.rz[im]);
  }
  for (int c = tid; c < PW; c += DA_THREADS) {
    const int j = c0 - DA_R + c;
    const bool in = j >= 0 && j < g.W;
    const C sv = in ? DC<T>::from(dc.svx[j]) : zero, gv = in ? DC<T>::from(dc.gvx[j]) : zero;
    const C l = in ? DC<T>::from(dc.lx[j]) : zero, r = in ? DC<T>::from(dc.rx[j]) : zero;
    t.prx[0][c] = sv; t.prx[1][c] = gv; t.prx[2][c] = l; t.prx[3][c] = r;
    plain_x = plain_x && is_real(sv, 1.0) && is_real(gv, 1.0) && is_real(l, 0.0) && r.x == r0x.x && r.y == r0x.y;
  }
  for (int c = tid; c < PH; c += DA_THREADS) {
    const int i = z0 - DA_R + c;
    const bool in = i >= 0 && i < g.H;
    const C sv = in ? DC<T>::from(dc.svz[i]) : zero, gv = in ? DC<T>::from(dc.gvz[i]) : zero;
    const C l = in ? DC<T>::from(dc.lz[i]) : zero, r = in ? DC<T>::from(dc.rz[i]) : zero;
    t.prz[0][c] = sv; t.prz[1][c] = gv; t.prz[2][c] = l; t.prz[3][c] = r;
    plain_z = plain_z && is_real(sv, 1.0) && is_real(gv, 1.0) && is_real(l, 0.0) && r.x == r0z.x && r.y == r0z.y;
  }
  plain_x = __syncthreads_and(plain_x) != 0;
  plain_z = __syncthreads_and(plain_z) != 0;
  const T a4[4] = {(T)nsr_dense_stencil(0), (T)nsr_dense_stencil(1), (T)nsr_dense_stencil(2), (T)nsr_dense_stencil(3)};
  const T inv_dx = (T)(1.0 / g.dx);
  const C scal = DC<T>::from(g.scal);
  // D along a line of stride s: sum a_q (p[+1+q] - p[-q])
  auto grad = [&](const C* q, int s) -> C {
    C v = a4[0] * (q[s] - q[0]);
#pragma unroll
    for (int k = 1; k < 4; ++k) v = v + a4[k] * (q[(1 + k) * s] - q[-k * s]);
    return v;
  };
  // divergence: sum a_q (f[+q] - f[-1-q])
  auto div = [&](const C* q, int s) -> C {
    C v = a4[0] * (q[0] - q[-s]);
#pragma unroll
    for (int k = 1; k < 4; ++k) v = v + a4[k] * (q[k * s] - q[-(1 + k) * s]);
    return v;
  };
  // D of (conj(factor) p) with a factor per node of the line
  auto grad_of = [&](const C* q, int s, const C* fac) -> C {
    C v = zero;
#pragma unroll
    for (int k = 0; k < 4; ++k) v = v + a4[k] * (conjc(fac[1 + k]) * q[(1 + k) * s] - conjc(fac[-k]) * q[-k * s]);
    return v;
  };
  auto div_of = [&](const C* q, int s, const C* fac) -> C {
    C v = zero;
#pragma unroll
    for (int k = 0; k < 4; ++k) v = v + a4[k] * (fac[k] * q[k * s] - fac[-1 - k] * q[-(1 + k) * s]);
    return v;
  };
  // fluxes along x: node (z0 + r, c0 - 4 + c)
  for (int k = tid; k < TZ * (DA_TX + 7); k += DA_THREADS) {
    const int r = k / (DA_TX + 7), c = k - r * (DA_TX + 7);
    const int i = z0 + r, j = c0 - 4 + c;
    C v = zero;
    if (i < g.H && j >= 0 && j < g.W) {
      const C* q = &t.p[r + DA_R][c + 3];
      const T ax = (T)dc.ax[(long long)i * g.W + j];
      if (!ADJ) {
        const C gx = grad(q, 1);
        v = plain_x ? (inv_dx * ax) * gx : (inv_dx * ax) * (t.prx[0][c + 3] * gx);
      } else if (plain_x) {
        v = (T(-1) * inv_dx * ax) * (conjc(scal * r0x) * grad(q, 1));
      } else {
        const C fl = grad_of(q, 1, &t.prx[2][c + 3]), fr = grad_of(q, 1, &t.prx[3][c + 3]);
        v = (T(-1) * inv_dx * ax) * (conjc(t.prx[0][c + 3] * scal) * (fl + conjc(t.prx[1][c + 3]) * fr));
      }
    }
    t.x[r][c] = v;
  }
  // fluxes along z: node (z0 - 4 + r, c0 + c)
  for (int k = tid; k < (TZ + 7) * DA_TX; k += DA_THREADS) {
    const int r = k / DA_TX, c = k - r * DA_TX;
    const int i = z0 - 4 + r, j = c0 + c;
    C v = zero;
    if (i >= 0 && i < g.H && j < g.W) {
      const C* q = &t.p[r + 3][c + DA_R];
      const T az = (T)dc.az[(long long)i * g.W + j];
      if (!ADJ) {
        const C gz = grad(q, PW);
        v = plain_z ? (inv_dx * az) * gz : (inv_dx * az) * (t.prz[0][r + 3] * gz);
      } else if (plain_z) {
        v = (T(-1) * inv_dx * az) * (conjc(scal * r0z) * grad(q, PW));
      } else {
        const C fl = grad_of(q, PW, &t.prz[2][r + 3]), fr = grad_of(q, PW, &t.prz[3][r + 3]);
        v = (T(-1) * inv_dx * az) * (conjc(t.prz[0][r + 3] * scal) * (fl + conjc(t.prz[1][r + 3]) * fr));
      }
    }
    t.z[r][c] = v;
  }
  __syncthreads();
  for (int k = tid; k < TZ * DA_TX; k += DA_THREADS) {
    const int r = k / DA_TX, c = k - r * DA_TX;
    const int i = z0 + r, j = c0 + c;
    if (i >= g.H || j >= g.W) continue;
    const long long id = (long long)i * g.W + j;
    if (!dense_inside(g, i, j)) { yf[id] = pf[id]; continue; }
    const C* qx = &t.x[r][c + 4];
    const C* qz = &t.z[r + 4][c];
    const C pk = t.p[r + DA_R][c + DA_R];
    const C mass = DC<T>::from(dc.mass[id]);
    if (!ADJ) {
      C part;
      const C dX = div(qx, 1), dZ = div(qz, DA_TX);
      part = plain_x ? r0x * dX
                     : t.prx[2][c + DA_R] * dX + t.prx[3][c + DA_R] * div_of(qx, 1, &t.prx[1][c + DA_R]);
      part = part + (plain_z ? r0z * dZ
                             : t.prz[2][r + DA_R] * dZ + t.prz[3][r + DA_R] * div_of(qz, DA_TX, &t.prz[1][r + DA_R]));
      yf[id] = scal * (inv_dx * part) + mass * pk;
    } else {
      yf[id] = (T(-1) * inv_dx) * (div(qx, 1) + div(qz, DA_TX)) + conjc(mass) * pk;
    }
  }
}

template <typename T, bool ADJ, int TZ>
static cudaError_t launch_dense_apply(const DenseGeo& g, const double* coef, int nf, const void* x, void* y,
                                      cudaStream_t st) {
  typedef typename DC<T>::C C;
  const int smem = (int)sizeof(DenseTile<T, TZ>);
  const cudaError_t ce = cudaFuncSetAttribute(k_dense_apply<T, ADJ, TZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (ce != cudaSuccess) return ce;
  const long long tiles = (long long)((g.W + DA_TX - 1) / DA_TX) * ((g.H + TZ - 1) / TZ);
  k_dense_apply<T, ADJ, TZ><<<(unsigned)(tiles * nf), DA_THREADS, smem, st>>>(g, coef, (const C*)x, (C*)y, nf);
  return cudaGetLastError();
}

// Tile height: tall tiles form the fewest fluxes twice (23 rows for 16); grids
// whose 16-row tiles are fewer than three per SM take 8-row ones.
template <typename T, bool ADJ>
static cudaError_t dense_apply_t(const DenseGeo& g, const double* coef, int nf, const void* x, void* y,
                                 cudaStream_t st) {
  const long long tiles = (long long)((g.W + DA_TX - 1) / DA_TX) * ((g.H + 15) / 16) * nf;
  return tiles >= 3 * 148 ? launch_dense_apply<T, ADJ, 16>(g, coef, nf, x, y, st)
                          : launch_dense_apply<T, ADJ, 8>(g, coef, nf, x, y, st);
}

extern "C" size_t nsr_dense_coef_bytes(const NsrDenseGrid* g) {
  if (!g || g->H <= 0 || g->W <= 0) return 0;
  return sizeof(double) * dense_coef_doubles(g->H, g->W);
}

extern "C" size_t nsr_dense_workspace_size(const NsrDenseGrid* g, int32_t n_fields, int32_t precision) {
  if (!g || g->H <= 0 || g->W <= 0 || n_fields < 0 || (precision != 0 && precision != 1)) return 0;
  return n_fields > 0 ? 256 : 0;   // the fluxes live in shared memory
}

DenseGeo nsr_dense_geo(const NsrDenseGrid* grid, double scal_re, double scal_im) {
  DenseGeo g;
  g.H = grid->H; g.W = grid->W; g.pz = grid->pz; g.px = grid->px; g.h = grid->h; g.w = grid->w; g.dx = grid->dx;
  g.scal = make_double2(scal_re, scal_im);
  return g;
}

int nsr_dense_apply_geo(const DenseGeo& g, const double* coef, int n_fields, int adjoint, int precision,
                        const void* x, void* y, cudaStream_t st) {
  const cudaError_t e =
      precision == 0 ? (adjoint ? dense_apply_t<float, true>(g, coef, n_fields, x, y, st)
                                : dense_apply_t<float, false>(g, coef, n_fields, x, y, st))
                     : (adjoint ? dense_apply_t<double, true>(g, coef, n_fields, x, y, st)
                                : dense_apply_t<double, false>(g, coef, n_fields, x, y, st));
  return e == cudaSuccess ? 0 : (int)e;
}

extern "C" int nsr_dense_apply(const NsrDenseGrid* grid, const double* coef, double scal_re, double scal_im,
                               int32_t n_fields, int32_t adjoint, int32_t precision, const void* x, void* y,
                               void* workspace, size_t workspace_bytes, void* stream) {
  if (!grid || !coef || !x || !y || n_fields < 0 || n_fields > 65535) return NSR_ERR_ARGUMENT;
  if (grid->H < 3 || grid->W < 3 || grid->h < 1 || grid->w < 1 || grid->pz < 0 || grid->px < 0 ||
      grid->pz + grid->h > grid->H || grid->px + grid->w > grid->W || !(grid->dx > 0))
    return NSR_ERR_ARGUMENT;
  if (precision != 0 && precision != 1) return NSR_ERR_ARGUMENT;
  if (n_fields == 0) return 0;
  if (!workspace || workspace_bytes < nsr_dense_workspace_size(grid, n_fields, precision)) return NSR_ERR_WORKSPACE;
  return nsr_dense_apply_geo(nsr_dense_geo(grid, scal_re, scal_im), coef, n_fields, adjoint, precision, x, y,
                             (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// Implicit gradient of the dense operator: cotangents of its coefficient
// planes for the bilinear form
//   L = -Re sum_f sum_n conj(lam_f[n]) mask[n] (A(m) (mask u_f))[n]
// that ImplicitChannels.backward differentiates (nsrno/dense_wave.py:250-255).
// A depends on the medium only through ax, az (the face coefficients) and the
// mass term, and L is linear in each, so
//   dL/dax[k]   = -Re sum_f svx[j] gx_f[k] Qx_f[k],   gx = D_x(mask u) / dx,
//   Qx = Div^T(mu lx) + gvx Div^T(mu rx),   mu = conj(lam) mask scal,
//   (Div^T v)[k] = (1/dx) sum_q a_q (v[k-q] - v[k+1+q]),
// likewise along z, and with w = conj(lam) mask u:
//   dL/dRe(mass) = -Re w,  dL/dIm(mass) = Im w.
// One thread per node sums the fields in order (deterministic).
// ---------------------------------------------------------------------------
__global__ void k_dense_grad(DenseGeo g, const double* __restrict__ coef, const double2* __restrict__ u,
                             const double2* __restrict__ lam, int nf, double* __restrict__ g_ax,
                             double* __restrict__ g_az, double* __restrict__ g_mass) {
  const DenseCoef dc = dense_unpack(coef, g.H, g.W);
  const long long n = (long long)g.H * g.W;
  const double inv_dx = 1.0 / g.dx;
  const double2 zero = make_double2(0.0, 0.0);
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k / g.W), j = (int)(k - (long long)i * g.W);
    double sax = 0.0, saz = 0.0, smr = 0.0, smi = 0.0;
    for (int f = 0; f < nf; ++f) {
      const double2* uf = u + (long long)f * n;
      const double2* lf = lam + (long long)f * n;
      // masked field and mu = conj(lam) mask scal at (i2, j2); zero outside the grid
      auto U = [&](int i2, int j2) -> double2 {
        if (i2 < 0 || i2 >= g.H || j2 < 0 || j2 >= g.W || !dense_inside(g, i2, j2)) return zero;
        return uf[(long long)i2 * g.W + j2];
      };
      auto MU = [&](int i2, int j2) -> double2 {
        if (i2 < 0 || i2 >= g.H || j2 < 0 || j2 >= g.W || !dense_inside(g, i2, j2)) return zero;
        return conjc(lf[(long long)i2 * g.W + j2]) * g.scal;
      };
      double2 gx = zero, gz = zero, qxl = zero, qxr = zero, qzl = zero, qzr = zero;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double a = nsr_dense_stencil(q);
        gx = gx + a * (U(i, j + 1 + q) - U(i, j - q));
        gz = gz + a * (U(i + 1 + q, j) - U(i - q, j));
        const int jw = j - q, je = j + 1 + q, in_ = i - q, is = i + 1 + q;
        const double2 mw = MU(i, jw), me = MU(i, je), mn = MU(in_, j), ms = MU(is, j);
        const double2 lxw = jw >= 0 ? dc.lx[jw] : zero, lxe = je < g.W ? dc.lx[je] : zero;
        const double2 rxw = jw >= 0 ? dc.rx[jw] : zero, rxe = je < g.W ? dc.rx[je] : zero;
        const double2 lzn = in_ >= 0 ? dc.lz[in_] : zero, lzs = is < g.H ? dc.lz[is] : zero;
        const double2 rzn = in_ >= 0 ? dc.rz[in_] : zero, rzs = is < g.H ? dc.rz[is] : zero;
        qxl = qxl + a * (mw * lxw - me * lxe);
        qxr = qxr + a * (mw * rxw - me * rxe);
        qzl = qzl + a * (mn * lzn - ms * lzs);
        qzr = qzr + a * (mn * rzn - ms * rzs);
      }
      const double2 Qx = inv_dx * (qxl + dc.gvx[j] * qxr);
      const double2 Qz = inv_dx * (qzl + dc.gvz[i] * qzr);
      sax -= (dc.svx[j] * (inv_dx * gx) * Qx).x;
      saz -= (dc.svz[i] * (inv_dx * gz) * Qz).x;
      if (dense_inside(g, i, j)) {
        const double2 w = conjc(lf[k]) * uf[k];
        smr -= w.x;
        smi += w.y;
      }
    }
    g_ax[k] = sax;
    g_az[k] = saz;
    g_mass[k] = smr;
    g_mass[n + k] = smi;
  }
}

extern "C" int nsr_dense_grad(const NsrDenseGrid* grid, const double* coef, double scal_re, double scal_im,
                              int32_t n_fields, const double* u, const double* lam, double* g_ax, double* g_az,
                              double* g_mass, void* stream) {
  if (!grid || !coef || !u || !lam || !g_ax || !g_az || !g_mass || n_fields < 0 || n_fields > 65535)
    return NSR_ERR_ARGUMENT;
  if (grid->H < 3 || grid->W < 3 || grid->h < 1 || grid->w < 1 || grid->pz < 0 || grid->px < 0 ||
      grid->pz + grid->h > grid->H || grid->px + grid->w > grid->W || !(grid->dx > 0))
    return NSR_ERR_ARGUMENT;
  const DenseGeo g = nsr_dense_geo(grid, scal_re, scal_im);
  const long long n = (long long)g.H * g.W;
  int bx = (int)((n + 255) / 256);
  if (bx > 4096) bx = 4096;
  k_dense_grad<<<bx, 256, 0, (cudaStream_t)stream>>>(g, coef, (const double2*)u, (const double2*)lam, n_fields,
                                                     g_ax, g_az, g_mass);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

// ---------------------------------------------------------------------------
// Fixed preconditioner of the dense path (nsrno/conditioned_wave.py:90-92,
// nsrno/dense_wave.py:194-196):
//   M r = mask * IFFT((1 + lap/k0^2 - i shift)^-1 FFT(r)),
// lap = -(|Dx|^2 + |Dz|^2) with the 8th-order staggered symbols
// |D(q)|^2 = (2 sum_k a_k sin((k + 1/2) q))^2 / dx^2 (conditioned_wave.py:24-27).
// The transforms are the solver's row and column FFTs (sizes 8..2048 whose
// prime factors are at most 61, e.g. the 1056 x 1216 padding of the reference).
// ---------------------------------------------------------------------------
// Eleven 1056 x 1216 fields (radices 11 3 2 16 and 19 4 16): 1,365 us with the
// prime radices as loops over local arrays and unpadded rows, 490 us with
// register butterflies and the ends of the transforms fused.
template <bool GEN>
__global__ void __launch_bounds__(256, GEN ? 2 : 4) k_dense_rows_fwd(int nz, int nx, PrecTables t,
                                                                     const float2* __restrict__ x,
                                                                     float2* __restrict__ w, int rows) {
  extern __shared__ float2 sm[];
  const int z0 = blockIdx.x * rows;
  const long long off = blockIdx.y * (long long)nz * nx + (long long)z0 * nx;
  const float2* __restrict__ xs = x + off;
  rows_forward<GEN>(sm, min(rows, nz - z0), t.px, w + off, [&](auto tag, int k0, int step, float2* v) {
#pragma unroll
    for (int q = 0; q < decltype(tag)::value; ++q) v[q] = xs[k0 + q * step];
  });
}

template <int TC, bool GEN>
__global__ void __launch_bounds__(GEN ? 256 : 512, 2) k_dense_cols(int nz, int nx, PrecTables t,
                                                                   const float* __restrict__ d2z,
                                                                   const float* __restrict__ d2x,
                                                                   float2* __restrict__ w, float inv_k0dx2,
                                                                   float shift, int adjoint) {
  extern __shared__ float2 sm[];
  const long long n = (long long)nz * nx;
  const int c0 = blockIdx.x * TC;
  const int ncol = min(TC, nx - c0);
  const float inv_n = 1.0f / (float)n;
  cols_multiply<GEN, TC>(sm, t.pz, w + blockIdx.y * n + c0, nx, ncol, [&](int c, int z) -> float2 {
    if (c >= ncol) return make_float2(0.f, 0.f);
    const float re = 1.0f - (d2z[z] + d2x[c0 + c]) * inv_k0dx2;
    const float2 mul = divc(make_float2(inv_n, 0.f), make_float2(re, -shift));
    return adjoint ? conjc(mul) : mul;
  });
}

// Inverse rows, masked to the native region: a tile of rows outside it is zero
// without a transform.
template <bool GEN>
__global__ void __launch_bounds__(256, GEN ? 2 : 4) k_dense_rows_inv(DenseGeo g, PrecTables t,
                                                                     const float2* __restrict__ w,
                                                                     float2* __restrict__ y, int rows) {
  extern __shared__ float2 sm[];
  const int nz = g.H, nx = g.W, z0 = blockIdx.x * rows, nr = min(rows, nz - z0);
  const long long off = blockIdx.y * (long long)nz * nx + (long long)z0 * nx;
  float2* __restrict__ ys = y + off;
  if (z0 >= g.pz + g.h || z0 + nr <= g.pz) {
    for (int k = threadIdx.x; k < nr * nx; k += blockDim.x) ys[k] = make_float2(0.f, 0.f);
    return;
  }
  rows_inverse<GEN>(sm, nr, t.px, w + off, [&](int k, float2 v, int l, int c) {
    ys[k] = dense_inside(g, z0 + l, c) ? v : make_float2(0.f, 0.f);
  });
}

static NsrGrid dense_fft_grid(const NsrDenseGrid* g) {
  NsrGrid q;
  memset(&q, 0, sizeof(q));
  q.nz = g->H;
  q.nx = g->W;
  q.h = g->dx;
  q.c0 = 1540.0;      // only the transform sizes of this grid are used
  q.rho0 = 1000.0;
  return q;
}

extern "C" size_t nsr_dense_precondition_workspace_size(const NsrDenseGrid* g, int32_t n_fields) {
  if (!g || n_fields <= 0 || n_fields > 65535) return 0;
  NsrGrid q = dense_fft_grid(g);
  if (nsr_check_grid(&q, true)) return 0;
  return nsr_align(nsr_prec_table_bytes(&q)) + nsr_align(sizeof(float) * (g->H + g->W)) +
         nsr_align(sizeof(float2) * (size_t)g->H * g->W * n_fields);
}

extern "C" int nsr_dense_precondition(const NsrDenseGrid* grid, double k0dx2, double shift, int32_t n_fields,
                                      int32_t adjoint, const float* x, float* y, void* workspace,
                                      size_t workspace_bytes, void* stream) {
  if (!grid || !x || !y || !workspace || n_fields < 0 || n_fields > 65535 || !(k0dx2 > 0) || !(shift >= 0))
    return NSR_ERR_ARGUMENT;
  if (grid->pz < 0 || grid->px < 0 || grid->pz + grid->h > grid->H || grid->px + grid->w > grid->W)
    return NSR_ERR_ARGUMENT;
  if (n_fields == 0) return 0;
  const size_t need = nsr_dense_precondition_workspace_size(grid, n_fields);
  if (need == 0) return NSR_ERR_UNSUPPORTED_SIZE;
  if (workspace_bytes < need) return NSR_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  DensePrec M;
  const int err = nsr_dense_prec_setup(grid, k0dx2, shift, n_fields, adjoint, workspace, st, &M);
  if (err) return err;
  const auto fwd = M.gx ? k_dense_rows_fwd<true> : k_dense_rows_fwd<false>;
  fwd<<<M.g_rows, 256, M.row_smem, st>>>(grid->H, grid->W, M.t, (const float2*)x, M.w, M.rows);
  nsr_dense_prec_finish(M, (float2*)y, st);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

int nsr_dense_prec_setup(const NsrDenseGrid* grid, double k0dx2, double shift, int n_fields, int adjoint,
                         void* workspace, cudaStream_t st, DensePrec* M) {
  NsrGrid q = dense_fft_grid(grid);
  char* ws = (char*)workspace;
  M->geo = nsr_dense_geo(grid, 0.0, 0.0);
  M->d2x = (float*)(ws + nsr_align(nsr_prec_table_bytes(&q)));
  M->d2z = M->d2x + grid->W;
  M->w = (float2*)(ws + nsr_align(nsr_prec_table_bytes(&q)) + nsr_align(sizeof(float) * (grid->H + grid->W)));
  const int err = nsr_prec_setup(&q, &M->t, ws, st, M->d2x, M->d2z);
  if (err) return err;
  M->inv_k0dx2 = (float)(1.0 / k0dx2);
  M->shift = (float)shift;
  M->adjoint = adjoint;
  M->rows = nsr_rows_per_cta(&q, n_fields);
  M->tc = nsr_cols_tc(&q, n_fields);
  M->gx = !nsr_specialised(grid->W);
  M->gz = !nsr_specialised(grid->H);
  M->g_rows = dim3((grid->H + M->rows - 1) / M->rows, n_fields);
  M->g_cols = dim3((grid->W + M->tc - 1) / M->tc, n_fields);
  M->row_smem = sizeof(float2) * (size_t)M->rows * nsr_row_stride(grid->W);
  M->col_smem = sizeof(float2) * (size_t)grid->H * M->tc;
  return 0;
}

void nsr_dense_prec_finish(const DensePrec& M, float2* y, cudaStream_t st) {
  const auto cols = M.tc == 16 ? (M.gz ? k_dense_cols<16, true> : k_dense_cols<16, false>)
                               : (M.gz ? k_dense_cols<8, true> : k_dense_cols<8, false>);
  cudaFuncSetAttribute((const void*)cols, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)M.col_smem);
  cols<<<M.g_cols, nsr_cols_threads(M.gz), M.col_smem, st>>>(M.geo.H, M.geo.W, M.t, M.d2z, M.d2x, M.w, M.inv_k0dx2,
                                                             M.shift, M.adjoint);
  const auto inv = M.gx ? k_dense_rows_inv<true> : k_dense_rows_inv<false>;
  inv<<<M.g_rows, 256, M.row_smem, st>>>(M.geo, M.t, M.w, y, M.rows);
}
