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
#include <type_traits>

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

// The same operator as a walk down the rows, for grids that fill the chip with
// bands of rows.  A thread owns CPT adjacent columns of a strip and keeps the
// last eight rows of mask p and of Z in registers, so the z part reads no shared
// memory at all; the x part writes a row of p (and then of X) once and reads ten
// neighbours of two columns as five 16-byte loads.  A step takes in row q, forms
// Z of row q - 4 and finishes row q - 7; the strip's halo columns and the next
// rows are in flight meanwhile.  A strip yields all but its four outermost columns
// on each side, whose X lacks neighbours.
// Eleven complex64 fields on 1056 x 1216: 260 us (tiles 316, two passes 695);
// bound by instruction issue at three CTAs per SM.
#define DS_THREADS 128
#define DS_ROWS 64     // most rows of a band
#define DS_UNROLL 2

template <typename T, int CPT>
struct __align__(16) DenseRowsSmem {
  typedef typename DC<T>::C C;
  static constexpr int N = DS_THREADS * CPT + 8;   // columns b0 - 4 .. b0 + strip + 3
  C a[2][N], b[2][N];                              // p, or conj(l) p and conj(r) p (adjoint in the PML)
  C x[N], gx[N];                                   // X, gvx X (forward in the PML)
  C halo[8][8];                                    // p at columns b0 - 3 .. b0 - 1 and the four after the strip
  C prz[4][DS_ROWS + 16];                          // sv, gv, l, r of rows z0 - 8 ..
};

__device__ __forceinline__ void ds_cp_async(float2* dst, const float2* src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(live ? 8 : 0) : "memory");
}
__device__ __forceinline__ void ds_cp_async(double2* dst, const double2* src, bool live) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(live ? 16 : 0) : "memory");
}

// CPT adjacent values, as one 16-byte access where CPT is 2.
template <int CPT>
__device__ __forceinline__ void ds_vec(const float2* p, float2* v) {
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = make_float2(t.x, t.y);
  v[1] = make_float2(t.z, t.w);
}
template <int CPT>
__device__ __forceinline__ void ds_vec(const double2* p, double2* v) { v[0] = *p; }
template <int CPT>
__device__ __forceinline__ void ds_vec(const double* p, double* v) {
  if constexpr (CPT == 2) {
    const double2 t = __ldg(reinterpret_cast<const double2*>(p));
    v[0] = t.x;
    v[1] = t.y;
  } else {
    v[0] = __ldg(p);
  }
}
template <int CPT>
__device__ __forceinline__ void ds_store(float2* p, const float2* v) {
  *reinterpret_cast<float4*>(p) = make_float4(v[0].x, v[0].y, v[1].x, v[1].y);
}
template <int CPT>
__device__ __forceinline__ void ds_store(double2* p, const double2* v) { *p = v[0]; }

// CPT + 8 consecutive row entries, from an entry that is a multiple of CPT.
template <int CPT>
__device__ __forceinline__ void ds_load(const float2* row, float2 (&v)[CPT + 8]) {
  static_assert(CPT == 2, "pairs");
#pragma unroll
  for (int q = 0; q < (CPT + 8) / 2; ++q) {
    const float4 t = reinterpret_cast<const float4*>(row)[q];
    v[2 * q] = make_float2(t.x, t.y);
    v[2 * q + 1] = make_float2(t.z, t.w);
  }
}
template <int CPT>
__device__ __forceinline__ void ds_load(const double2* row, double2 (&v)[CPT + 8]) {
#pragma unroll
  for (int q = 0; q < CPT + 8; ++q) v[q] = row[q];
}

template <typename T, bool ADJ, int CPT>
__global__ void __launch_bounds__(DS_THREADS, sizeof(T) == 4 ? 3 : 2)
    k_dense_stream(DenseGeo g, const double* __restrict__ coef, const typename DC<T>::C* __restrict__ p,
                   typename DC<T>::C* __restrict__ y, int nf, int rows) {
  typedef typename DC<T>::C C;
  typedef DenseRowsSmem<T, CPT> Smem;
  extern __shared__ __align__(16) unsigned char da_smem[];
  Smem& sm = *reinterpret_cast<Smem*>(da_smem);
  constexpr int STRIP = DS_THREADS * CPT, OUT = STRIP - 8;
  const DenseCoef dc = dense_unpack(coef, g.H, g.W);
  const long long n = (long long)g.H * g.W;
  const int f = blockIdx.x % nf, tile = blockIdx.x / nf;
  const int nbx = (g.W + OUT - 1) / OUT;
  const int z0 = (tile / nbx) * rows, z1 = min(z0 + rows, g.H);
  const int c0 = (tile % nbx) * OUT, b0 = c0 - 4;   // outputs c0 .. c0 + OUT - 1
  const C* __restrict__ pf = p + (long long)f * n;
  C* __restrict__ yf = y + (long long)f * n;
  const C zero = cx<C>(T(0), T(0));
  const int tid = threadIdx.x, jt = b0 + CPT * tid;
  const int j0 = min(max(jt, 0), g.W - CPT);   // W is a multiple of CPT and jt too: a thread's columns are in or out together
  if (!(z0 < g.pz + g.h && z1 > g.pz && c0 < g.px + g.w && c0 + OUT > g.px)) {   // no native node: copy
    for (int i = z0; i < z1; ++i)
      for (int j = c0 + tid; j < min(c0 + OUT, g.W); j += DS_THREADS) yf[(long long)i * g.W + j] = pf[(long long)i * g.W + j];
    return;
  }
  C rxc[CPT], lxc[CPT], svc[CPT], gvc[CPT];
#pragma unroll
  for (int c = 0; c < CPT; ++c) {
    svc[c] = DC<T>::from(dc.svx[j0 + c]);
    gvc[c] = DC<T>::from(dc.gvx[j0 + c]);
    lxc[c] = DC<T>::from(dc.lx[j0 + c]);
    rxc[c] = DC<T>::from(dc.rx[j0 + c]);
  }
  // Whether every column (row) the block touches is off the PML, with one right factor.
  const C r0x = DC<T>::from(dc.rx[min(c0, g.W - 1)]), r0z = DC<T>::from(dc.rz[z0]);
  bool px = true, pz = true;
  for (int e = tid; e < STRIP + 8; e += DS_THREADS) {
    const int j = min(max(b0 - 4 + e, 0), g.W - 1);
    const C r = DC<T>::from(dc.rx[j]);
    px = px && is_real(DC<T>::from(dc.svx[j]), 1.0) && is_real(DC<T>::from(dc.gvx[j]), 1.0) &&
         is_real(DC<T>::from(dc.lx[j]), 0.0) && r.x == r0x.x && r.y == r0x.y;
  }
  for (int e = tid; e < rows + 16; e += DS_THREADS) {
    const int i = z0 - 8 + e;
    const bool in = i >= 0 && i < g.H;
    const C sv = in ? DC<T>::from(dc.svz[i]) : zero, gv = in ? DC<T>::from(dc.gvz[i]) : zero;
    const C l = in ? DC<T>::from(dc.lz[i]) : zero, r = in ? DC<T>::from(dc.rz[i]) : zero;
    sm.prz[0][e] = sv; sm.prz[1][e] = gv; sm.prz[2][e] = l; sm.prz[3][e] = r;
    pz = pz && is_real(sv, 1.0) && is_real(gv, 1.0) && is_real(l, 0.0) && r.x == r0z.x && r.y == r0z.y;
  }
  const bool plain_x = __syncthreads_and(px) != 0, plain_z = __syncthreads_and(pz) != 0;
  const T a4[4] = {(T)nsr_dense_stencil(0), (T)nsr_dense_stencil(1), (T)nsr_dense_stencil(2), (T)nsr_dense_stencil(3)};
  const T inv_dx = (T)(1.0 / g.dx), sgn = ADJ ? T(-1) * inv_dx : inv_dx;
  const C scal = DC<T>::from(g.scal);
  const C adj_x = conjc(scal * r0x), adj_z = conjc(scal * r0z);
  bool col_in[CPT], col_out[CPT];
#pragma unroll
  for (int c = 0; c < CPT; ++c) {
    col_in[c] = jt + c >= g.px && jt + c < g.px + g.w;
    col_out[c] = jt + c >= c0 && jt + c < min(c0 + OUT, g.W);
  }
  const bool live_cols = jt >= 0 && jt < g.W;
  const C* __restrict__ pcol = pf + j0;
  const double* __restrict__ axt = dc.ax + j0;
  const double* __restrict__ azt = dc.az + j0;
  const double2* __restrict__ mt = dc.mass + j0;
  auto load_p = [&](int i, C* v) {   // mask p of row i at the thread's columns
    C t[CPT];
    ds_vec<CPT>(pcol + (long long)min(max(i, 0), g.H - 1) * g.W, t);
    const bool row_in = i >= g.pz && i < g.pz + g.h;
#pragma unroll
    for (int c = 0; c < CPT; ++c) v[c] = row_in && col_in[c] ? t[c] : zero;
  };
  // halo entry of this thread (the first seven)
  const int hj = tid < 3 ? b0 - 3 + tid : b0 + STRIP + tid - 3;
  const int he = tid < 3 ? 1 + tid : STRIP + 4 + tid - 3;   // its entry in a row
  const bool h_in = hj >= g.px && hj < g.px + g.w;
  const int hjc = min(max(hj, 0), g.W - 1);
  const C hl = ADJ ? conjc(DC<T>::from(dc.lx[hjc])) : zero, hr = ADJ ? conjc(DC<T>::from(dc.rx[hjc])) : zero;

  // Windows of mask p and of Z: entry 8 + k takes the row of step k of a group of
  // DS_UNROLL, entries 0 .. 7 hold the eight before.  (A ring of eight without the
  // shift needs eight copies of the step, which missed the instruction cache: 327
  // us where this form takes 260.)
  C pw[8 + DS_UNROLL][CPT], zw[8 + DS_UNROLL][CPT];
#pragma unroll
  for (int k = 0; k < 8 + DS_UNROLL; ++k)
#pragma unroll
    for (int c = 0; c < CPT; ++c) pw[k][c] = zw[k][c] = zero;
  C pn[2][CPT];   // rows q + 1, q + 2 in flight
  load_p(z0 - 7, pn[0]);
  load_p(z0 - 6, pn[1]);
  double raw_az[CPT], raw_ax[CPT];
  double2 raw_m[CPT];
  auto load_coef = [&](int q) {   // az of row q - 4, ax and mass of row q - 7
    const long long rz = (long long)min(max(q - 4, 0), g.H - 1) * g.W, ri = (long long)min(max(q - 7, 0), g.H - 1) * g.W;
    ds_vec<CPT>(azt + rz, raw_az);
    ds_vec<CPT>(axt + ri, raw_ax);
#pragma unroll
    for (int c = 0; c < CPT; ++c) raw_m[c] = __ldg(mt + ri + c);
  };
  load_coef(z0 - 7);
  const int steps = z1 - z0 + 14;
  // One copy of the loop per kind of block: with every case in one body it did
  // not fit the instruction cache.
  auto walk = [&](auto tag_x, auto tag_z) {
  constexpr bool plain_x = decltype(tag_x)::value, plain_z = decltype(tag_z)::value;
#pragma unroll 1
  for (int s0 = 0; s0 < steps; s0 += DS_UNROLL) {
#pragma unroll
    for (int k = 0; k < DS_UNROLL; ++k) {
      const int s = s0 + k;
      if (s >= steps) break;
      const int q = z0 - 7 + s;
      if (tid < 7) {
        const bool live = h_in && q >= g.pz && q < g.pz + g.h;
        ds_cp_async(&sm.halo[s & 7][tid], pf + (live ? (long long)q * g.W + hjc : 0), live);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
      const int zr = q - 4, i = q - 7;
      // this step's coefficients (loaded during the step before), then the next's
      T caz[CPT], cax[CPT];
      C cm[CPT];
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        caz[c] = (T)raw_az[c];
        cax[c] = (T)raw_ax[c];
        cm[c] = DC<T>::from(raw_m[c]);
      }
      load_coef(q + 1);
#pragma unroll
      for (int c = 0; c < CPT; ++c) pw[8 + k][c] = pn[k & 1][c];
      load_p(q + 2, pn[k & 1]);
      // Z of row q - 4 from rows q - 7 .. q
      if (s >= 7) {
        const bool live = zr >= 0 && zr < g.H;
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          C v;
          const T az = live ? sgn * caz[c] : T(0);
          if (!ADJ || plain_z) {
            C d = zero;
#pragma unroll
            for (int t = 0; t < 4; ++t) d = d + a4[t] * (pw[k + 5 + t][c] - pw[k + 4 - t][c]);
            v = plain_z ? (ADJ ? az * (adj_z * d) : az * d) : az * (sm.prz[0][zr - z0 + 8] * d);
          } else {
            C fl = zero, fr = zero;
            const int e = zr - z0 + 8;
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              const C ps = pw[k + 5 + t][c], pm = pw[k + 4 - t][c];
              fl = fl + a4[t] * (conjc(sm.prz[2][e + 1 + t]) * ps - conjc(sm.prz[2][e - t]) * pm);
              fr = fr + a4[t] * (conjc(sm.prz[3][e + 1 + t]) * ps - conjc(sm.prz[3][e - t]) * pm);
            }
            v = az * (conjc(sm.prz[0][e] * scal) * (fl + conjc(sm.prz[1][e]) * fr));
          }
          zw[8 + k][c] = v;
        }
      }
      if (s < 14) continue;
      // finish row i = q - 7, whose p is the oldest row of the window
      const C* pi = pw[k + 1];
      C* ra = sm.a[s & 1];
      C* rb = sm.b[s & 1];
      asm volatile("cp.async.wait_group 7;" ::: "memory");
      if (tid < 7) {
        const C h = sm.halo[(s + 1) & 7][tid];
        ra[he] = !ADJ || plain_x ? h : hl * h;
        if (ADJ && !plain_x) rb[he] = hr * h;
      }
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        ra[4 + CPT * tid + c] = !ADJ || plain_x ? pi[c] : conjc(lxc[c]) * pi[c];
        if (ADJ && !plain_x) rb[4 + CPT * tid + c] = conjc(rxc[c]) * pi[c];
      }
      __syncthreads();
      {
        C v[CPT + 8], d[CPT];
        auto grad = [&](int c) -> C {   // D at the thread's column c
          C u = zero;
#pragma unroll
          for (int t = 0; t < 4; ++t) u = u + a4[t] * (v[c + 5 + t] - v[c + 4 - t]);
          return u;
        };
        ds_load<CPT>(ra + CPT * tid, v);
#pragma unroll
        for (int c = 0; c < CPT; ++c) d[c] = grad(c);
        if (ADJ && !plain_x) {
          ds_load<CPT>(rb + CPT * tid, v);
#pragma unroll
          for (int c = 0; c < CPT; ++c) d[c] = d[c] + conjc(gvc[c]) * grad(c);
        }
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          const T ax = live_cols ? sgn * cax[c] : T(0);
          const C x = ax * (plain_x ? (ADJ ? adj_x * d[c] : d[c]) : (ADJ ? conjc(svc[c] * scal) : svc[c]) * d[c]);
          sm.x[4 + CPT * tid + c] = x;
          if (!ADJ && !plain_x) sm.gx[4 + CPT * tid + c] = gvc[c] * x;
        }
      }
      __syncthreads();
      {
        C v[CPT + 8], part[CPT];
        auto div = [&](int c) -> C {   // sum a (X[c + t] - X[c - 1 - t])
          C u = zero;
#pragma unroll
          for (int t = 0; t < 4; ++t) u = u + a4[t] * (v[c + 4 + t] - v[c + 3 - t]);
          return u;
        };
        ds_load<CPT>(sm.x + CPT * tid, v);
#pragma unroll
        for (int c = 0; c < CPT; ++c) part[c] = ADJ ? div(c) : (plain_x ? rxc[c] : lxc[c]) * div(c);
        if (!ADJ && !plain_x) {
          ds_load<CPT>(sm.gx + CPT * tid, v);
#pragma unroll
          for (int c = 0; c < CPT; ++c) part[c] = part[c] + rxc[c] * div(c);
        }
        const bool row_in = i >= g.pz && i < g.pz + g.h;
        C res[CPT];
        bool all = row_in;
#pragma unroll
        for (int c = 0; c < CPT; ++c) {
          C dz = zero, dg = zero;
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const C zs = zw[k + 5 + t][c], zm = zw[k + 4 - t][c];
            dz = dz + a4[t] * (zs - zm);
            if (!ADJ && !plain_z) dg = dg + a4[t] * (sm.prz[1][i - z0 + 8 + t] * zs - sm.prz[1][i - z0 + 7 - t] * zm);
          }
          if (ADJ) {
            res[c] = sgn * (part[c] + dz) + conjc(cm[c]) * pi[c];
          } else {
            const C sum = part[c] + (plain_z ? r0z * dz : sm.prz[2][i - z0 + 8] * dz + sm.prz[3][i - z0 + 8] * dg);
            res[c] = scal * (inv_dx * sum) + cm[c] * pi[c];
          }
          all = all && col_out[c] && col_in[c];
        }
        const long long id = (long long)i * g.W + jt;
        if (all) {
          ds_store<CPT>(yf + id, res);
        } else {
#pragma unroll
          for (int c = 0; c < CPT; ++c)
            if (col_out[c]) yf[id + c] = row_in && col_in[c] ? res[c] : pf[id + c];
        }
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e)
#pragma unroll
      for (int c = 0; c < CPT; ++c) {
        pw[e][c] = pw[e + DS_UNROLL][c];
        zw[e][c] = zw[e + DS_UNROLL][c];
      }
  }
  };
  if (plain_x) {
    if (plain_z) walk(std::true_type{}, std::true_type{});
    else walk(std::true_type{}, std::false_type{});
  } else {
    if (plain_z) walk(std::false_type{}, std::true_type{});
    else walk(std::false_type{}, std::false_type{});
  }
}

// Launch: the walk where it is the faster one and, for complex64, even widths and
// 16-byte aligned buffers let it read pairs; else the tiles, 16 rows high (23 rows
// of fluxes for 16) or, where those are fewer than three per SM, 8.
// The walk's time goes by the columns of its strips, filled or not, the tiles' by
// the nodes, more of it once the fields pass the L2.  us, walk against tiles
// (forward, complex64, then complex128): 11 of 480 x 480 (2.5 M nodes, strips
// filled to 0.97 and 1.0) 52 / 54, 105 / 98; 11 of 672 x 576 (4.3 M, 0.77 and 0.96)
// 113 / 102, 187 / 182; 2 of 1056 x 1216 (2.6 M, 0.98 and 0.92) 52 / 70, 118 / 126;
// 3 of 768 x 992 (2.3 M, 1.0 and 0.92) 61 / 54, 106 / 107; 11 of them (8.4 M)
// 166 / 239, 305 / 352; 60 of 128 x 128 (1.0 M, 0.52 and 0.53) 44 / 23, 78 / 27.
template <typename T, bool ADJ>
static cudaError_t dense_apply_t(const DenseGeo& g, const double* coef, int nf, const void* x, void* y,
                                 cudaStream_t st) {
  typedef typename DC<T>::C C;
  constexpr int CPT = sizeof(T) == 4 ? 2 : 1, OUT = DS_THREADS * CPT - 8;
  constexpr int RESIDENT = 148 * (sizeof(T) == 4 ? 3 : 2);
  const long long across = (g.W + OUT - 1) / OUT, strips = across * nf, nodes = (long long)nf * g.H * g.W;
  const bool walk = (nodes >= 2500000 && 8LL * g.W >= 7 * across * OUT) ||
                    (nodes >= 6000000 && 4LL * g.W >= 3 * across * OUT);
  const bool pairs = CPT == 1 || (g.W % 2 == 0 && (((uintptr_t)coef | (uintptr_t)x | (uintptr_t)y) & 15) == 0);
  if (walk && pairs) {
    // Band height: a band walks 14 rows more than it yields, and the last wave of
    // blocks should be full, so take the height with the fewest row steps over
    // all waves (1056 rows of eleven fields: 44 rows, 262 us at 32).
    int rows = 32;
    long long best = -1;
    for (int r = 16; r <= DS_ROWS; ++r) {
      const long long waves = (strips * ((g.H + r - 1) / r) + RESIDENT - 1) / RESIDENT, cost = waves * (r + 14);
      if (best < 0 || cost < best) { best = cost; rows = r; }
    }
    const long long bands = strips * ((g.H + rows - 1) / rows);
    const int smem = (int)sizeof(DenseRowsSmem<T, CPT>);
    const cudaError_t ce = cudaFuncSetAttribute(k_dense_stream<T, ADJ, CPT>,
                                                cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (ce != cudaSuccess) return ce;
    k_dense_stream<T, ADJ, CPT><<<(unsigned)bands, DS_THREADS, smem, st>>>(g, coef, (const C*)x, (C*)y, nf, rows);
    return cudaGetLastError();
  }
  const long long tiles = (long long)((g.W + DA_TX - 1) / DA_TX) * ((g.H + 15) / 16) * nf;
  return tiles >= 3 * 148 ? launch_dense_apply<T, ADJ, 16>(g, coef, nf, x, y, st)
                          : launch_dense_apply<T, ADJ, 8>(g, coef, nf, x, y, st);
}

extern "C" size_t nsr_dense_coef_bytes(const NsrDenseGrid* g) {
  if (!g || g->H <= 0 || g->W <= 0) return 0;
  return sizeof(double) * dense_coef_doubles(g->H, g->W);
}

// The fluxes live in shared memory: separate buffers need no workspace to speak
// of.  A call in place copies its fields there first, because tiles read the
// halos of their neighbours' nodes.
#define NSR_DENSE_WORKSPACE_MIN 256
extern "C" size_t nsr_dense_workspace_size(const NsrDenseGrid* g, int32_t n_fields, int32_t precision) {
  if (!g || g->H <= 0 || g->W <= 0 || n_fields < 0 || (precision != 0 && precision != 1)) return 0;
  if (n_fields == 0) return 0;
  return NSR_DENSE_WORKSPACE_MIN + (size_t)g->H * g->W * n_fields * (precision ? 16 : 8);
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
  const size_t full = nsr_dense_workspace_size(grid, n_fields, precision);
  if (!workspace || workspace_bytes < (x == y ? full : NSR_DENSE_WORKSPACE_MIN)) return NSR_ERR_WORKSPACE;
  if (x == y) {
    const cudaError_t ce = cudaMemcpyAsync(workspace, x, full - NSR_DENSE_WORKSPACE_MIN, cudaMemcpyDeviceToDevice,
                                           (cudaStream_t)stream);
    if (ce != cudaSuccess) return (int)ce;
    x = workspace;
  }
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
// prime radices as loops over local arrays and unpadded rows, 420 us with
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
  M->gx = nsr_rows_generic(grid->W, M->w);
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
