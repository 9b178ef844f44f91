// Stand-alone operators of the nsrno_b200 C ABI: material planes, the 5-point
// operator apply, the FFT shifted-Laplace preconditioner, plane-wave
// right-hand sides and the adjoint-state material gradient.
#include "nsr_common.cuh"
#include "nsr_internal.cuh"
#include "nsr_device.cuh"

#include <string.h>

// ---------------------------------------------------------------------------
// Error strings and argument checks.
// ---------------------------------------------------------------------------
extern "C" int nsr_version(void) { return 100; }

extern "C" const char* nsr_error_string(int code) {
  switch (code) {
    case 0: return "ok";
    case NSR_ERR_ARGUMENT: return "nsrno_b200: invalid argument";
    case NSR_ERR_UNSUPPORTED_SIZE: return "nsrno_b200: nz and nx must be between 8 and 2048 with no prime factor above 61";
    case NSR_ERR_WORKSPACE: return "nsrno_b200: workspace too small";
    case NSR_ERR_INTERNAL: return "nsrno_b200: solver queue did not drain";
    case NSR_ERR_CAPACITY: return "nsrno_b200: request exceeds the fixed capacity";
    case NSR_ERR_TIMEOUT: return "nsrno_b200: a kernel timed out waiting for its shared-memory copies";
    default: break;
  }
  if (code > 0 && code < 1000) return cudaGetErrorString((cudaError_t)code);
  return "nsrno_b200: unknown error";
}

int nsr_check_grid(const NsrGrid* g, bool need_fft) {
  if (!g) return NSR_ERR_ARGUMENT;
  if (g->nz < 3 || g->nx < 3 || g->n_pml < 0 || 2 * g->n_pml >= g->nz || 2 * g->n_pml >= g->nx) return NSR_ERR_ARGUMENT;
  if (!(g->h > 0) || !(g->c0 > 0) || !(g->rho0 > 0) || !(g->pml_strength >= 0)) return NSR_ERR_ARGUMENT;
  if (g->face < 0 || g->face >= g->nz) return NSR_ERR_ARGUMENT;
  if ((long long)g->nz * g->nx > (1LL << 30)) return NSR_ERR_ARGUMENT;
  if (need_fft) {
    int r[NSR_MAX_RADIX_STAGES], k;
    if (!nsr_make_radices(g->nz, r, &k) || !nsr_make_radices(g->nx, r, &k)) return NSR_ERR_UNSUPPORTED_SIZE;
  }
  return 0;
}

static inline int last_error() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : (int)e;
}

// ---------------------------------------------------------------------------
// Material planes.
// ---------------------------------------------------------------------------
__global__ void k_setup_material(Geo g, const float* __restrict__ c, const float* __restrict__ rho,
                                 const float* __restrict__ alpha, void* __restrict__ mat, long long n) {
  const double neper = 100.0 * 2.302585092994045684 / 20.0;  // dB/cm -> Np/m
  float* f = (float*)mat;
  double* d = (double*)((char*)mat + nsr_material_off64(n));
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const double cc = c[k], rr = rho[k], al = alpha[k];
    const double a = g.rho0 / rr;
    const double b = g.rho0 * g.c0 * g.c0 / (rr * cc * cc);
    const double t = al * neper * cc / (2.0 * NSR_PI * 1e6);
    d[k] = a; d[n + k] = b; d[2 * n + k] = t;
    f[k] = (float)a; f[n + k] = (float)b; f[2 * n + k] = (float)t;
  }
}

extern "C" size_t nsr_material_bytes(const NsrGrid* grid) {
  if (nsr_check_grid(grid, false)) return 0;
  return nsr_material_size((long long)grid->nz * grid->nx);
}

extern "C" int nsr_setup_material(const NsrGrid* grid, const float* c, const float* rho,
                                  const float* alpha_db, void* material, void* stream) {
  int err = nsr_check_grid(grid, false);
  if (err) return err;
  if (!c || !rho || !alpha_db || !material) return NSR_ERR_ARGUMENT;
  long long n = (long long)grid->nz * grid->nx;
  int blocks = (int)((n + 255) / 256);
  if (blocks > 148 * 32) blocks = 148 * 32;
  k_setup_material<<<blocks, 256, 0, (cudaStream_t)stream>>>(make_geo(*grid), c, rho, alpha_db, material, n);
  return last_error();
}

// ---------------------------------------------------------------------------
// Operator apply (one thread per node; used for checks and true residuals).
// ---------------------------------------------------------------------------
template <typename T> struct PlaneOf;
template <> struct PlaneOf<float> {
  static __device__ __forceinline__ const float* a(const MatPlanes& m) { return m.a32; }
  static __device__ __forceinline__ const float* b(const MatPlanes& m) { return m.b32; }
  static __device__ __forceinline__ const float* t(const MatPlanes& m) { return m.t32; }
};
template <> struct PlaneOf<double> {
  static __device__ __forceinline__ const double* a(const MatPlanes& m) { return m.a64; }
  static __device__ __forceinline__ const double* b(const MatPlanes& m) { return m.b64; }
  static __device__ __forceinline__ const double* t(const MatPlanes& m) { return m.t64; }
};

// FP32 fields use the float planes, FP64 fields the double planes.  A thread
// walks down one column of a TZ-row tile: the north and centre values are
// carried, east and west come from the adjacent lanes, and the PML factors are
// formed once per column and row (stencil_sep).  Bound by HBM for large batches
// and by launch latency for one small field.  Six complex128 243 x 729 fields,
// adjoint: 42 us with one thread per node and four complex divisions each,
// 19 us in this form.
template <typename T, bool ADJ, int TZ, int TX>
__global__ void __launch_bounds__(TX) k_apply(Geo g, const void* __restrict__ mat, const double* __restrict__ freq,
                                              const typename CxT<T>::type* __restrict__ x,
                                              typename CxT<T>::type* __restrict__ y) {
  typedef typename CxT<T>::type C;
  __shared__ SysScalars sc;
  __shared__ RowFactors<T> rowf[TZ];
  const long long n = (long long)g.nz * g.nx;
  const int nx = g.nx, nz = g.nz;
  const int nbx = (nx + TX - 1) / TX;
  const int z0 = (blockIdx.x / nbx) * TZ;
  const int j = (blockIdx.x % nbx) * TX + threadIdx.x;
  const int lane = threadIdx.x & 31;
  const bool own = j < nx;
  const C* __restrict__ xs = x + blockIdx.y * n;
  C* __restrict__ ys = y + blockIdx.y * n;
  const MatPlanes mp = nsr_planes(mat, n);
  const T* __restrict__ ca = PlaneOf<T>::a(mp);
  const T* __restrict__ cb = PlaneOf<T>::b(mp);
  const T* __restrict__ ct = PlaneOf<T>::t(mp);
  const C zero = cx<C>(T(0), T(0));
  long long idx = (long long)z0 * nx + (own ? j : nx - 1);
  C pn = z0 > 0 ? xs[idx - nx] : zero, pc = xs[idx];
  T an = z0 > 0 ? ca[idx - nx] : T(1), ac = ca[idx];
  if (threadIdx.x == 0) sc = sys_scalars(g, freq[blockIdx.y]);
  __syncthreads();
  if (threadIdx.x < TZ) rowf[threadIdx.x] = row_factors<T>(g, sc, z0 + threadIdx.x);
  const ColFactors<T> cf = col_factors<T>(g, sc, j);
  const T kh2 = (T)sc.kh2, fpow = (T)sc.fpow;
  __syncthreads();
  const bool edge_w = lane == 0 && j > 0, edge_e = lane == 31 && j + 1 < nx;
#pragma unroll
  for (int r = 0; r < TZ; ++r) {
    const int i = z0 + r;
    if (i >= nz) break;
    const bool has_s = i + 1 < nz;
    const C ps = has_s ? xs[idx + nx] : zero;
    const T as = has_s ? ca[idx + nx] : T(1);
    C pe, pw;
    pe.x = __shfl_down_sync(0xffffffffu, pc.x, 1);
    pe.y = __shfl_down_sync(0xffffffffu, pc.y, 1);
    pw.x = __shfl_up_sync(0xffffffffu, pc.x, 1);
    pw.y = __shfl_up_sync(0xffffffffu, pc.y, 1);
    T ae = __shfl_down_sync(0xffffffffu, ac, 1), aw = __shfl_up_sync(0xffffffffu, ac, 1);
    if (edge_e) { pe = xs[idx + 1]; ae = ca[idx + 1]; }
    if (edge_w) { pw = xs[idx - 1]; aw = ca[idx - 1]; }
    if (j + 1 >= nx) { pe = zero; ae = T(1); }
    if (j == 0) { pw = zero; aw = T(1); }
    const C v = stencil_sep<T, ADJ>(kh2, fpow, rowf[r], cf, ac, ae, aw, as, an, cb[idx], ct[idx], pc, pe, pw, ps, pn);
    if (own) ys[idx] = v;
    pn = pc;
    pc = ps;
    an = ac;
    ac = as;
    idx += nx;
  }
}

// One thread per node, for grids so narrow that a warp of columns would be half
// empty or more.
template <typename T, bool ADJ>
__global__ void __launch_bounds__(256) k_apply_nodes(Geo g, const void* __restrict__ mat,
                                                     const double* __restrict__ freq,
                                                     const typename CxT<T>::type* __restrict__ x,
                                                     typename CxT<T>::type* __restrict__ y) {
  typedef typename CxT<T>::type C;
  const long long n = (long long)g.nz * g.nx, k = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const SysScalars s = sys_scalars(g, freq[blockIdx.y]);
  const MatPlanes mp = nsr_planes(mat, n);
  const T* __restrict__ ca = PlaneOf<T>::a(mp);
  const C* __restrict__ xs = x + blockIdx.y * n;
  auto inside = [&](int i, int j) { return i >= 0 && i < g.nz && j >= 0 && j < g.nx; };
  auto P = [&](int i, int j) -> C { return inside(i, j) ? xs[(long long)i * g.nx + j] : cx<C>(T(0), T(0)); };
  auto A = [&](int i, int j) -> T { return inside(i, j) ? ca[(long long)i * g.nx + j] : T(1); };
  const int i = (int)(k / g.nx), j = (int)(k - (long long)i * g.nx);
  y[blockIdx.y * n + k] = stencil<T, ADJ>(g, s, i, j, PlaneOf<T>::b(mp)[k], PlaneOf<T>::t(mp)[k], P, A);
}

template <typename T, bool ADJ, int TX>
static void launch_apply_tx(const Geo& g, const void* coef, const double* freq, int ns, const void* x, void* y,
                            cudaStream_t st) {
  typedef typename CxT<T>::type C;
  // 8-row tiles read 10 rows for 8; small grids take 2-row tiles so that every
  // SM gets a few blocks.
  const int bx = (g.nx + TX - 1) / TX;
  if ((long long)bx * ((g.nz + 7) / 8) * ns * TX >= 8 * 148 * 128)
    k_apply<T, ADJ, 8, TX><<<dim3(bx * ((g.nz + 7) / 8), ns), TX, 0, st>>>(g, coef, freq, (const C*)x, (C*)y);
  else
    k_apply<T, ADJ, 2, TX><<<dim3(bx * ((g.nz + 1) / 2), ns), TX, 0, st>>>(g, coef, freq, (const C*)x, (C*)y);
}
// Columns of a block: 128, one warp's where 128 would be largely empty, a thread
// per node where a warp would.  Us a call, 22 complex64 fields of 2048 x 8: 45 with
// 128 columns, 19 with 32, 15 by nodes; of 2048 x 16: 45 and 23 by nodes; six of
// 2048 x 60: 17.6 with 128, 18.7 with 32.
template <typename T, bool ADJ>
static void launch_apply(const Geo& g, const void* coef, const double* freq, int ns, const void* x, void* y,
                         cudaStream_t st) {
  typedef typename CxT<T>::type C;
  if (g.nx <= 16)
    k_apply_nodes<T, ADJ><<<dim3((unsigned)(((long long)g.nz * g.nx + 255) / 256), ns), 256, 0, st>>>(g, coef, freq,
                                                                                                      (const C*)x, (C*)y);
  else if (g.nx <= 48) launch_apply_tx<T, ADJ, 32>(g, coef, freq, ns, x, y, st);
  else launch_apply_tx<T, ADJ, 128>(g, coef, freq, ns, x, y, st);
}

extern "C" int nsr_apply(const NsrGrid* grid, const void* coef, const double* freq_hz,
                         int32_t n_systems, int32_t adjoint, int32_t precision,
                         const void* x, void* y, void* stream) {
  int err = nsr_check_grid(grid, false);
  if (err) return err;
  if (!coef || !freq_hz || !x || !y || n_systems < 0 || n_systems > 65535) return NSR_ERR_ARGUMENT;
  if (n_systems == 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  const Geo g = make_geo(*grid);
  if (precision == 0) {
    if (adjoint) launch_apply<float, true>(g, coef, freq_hz, n_systems, x, y, st);
    else launch_apply<float, false>(g, coef, freq_hz, n_systems, x, y, st);
  } else if (precision == 1) {
    if (adjoint) launch_apply<double, true>(g, coef, freq_hz, n_systems, x, y, st);
    else launch_apply<double, false>(g, coef, freq_hz, n_systems, x, y, st);
  } else {
    return NSR_ERR_ARGUMENT;
  }
  return last_error();
}

// ---------------------------------------------------------------------------
// Preconditioner tables and passes (shared with the solver).
// ---------------------------------------------------------------------------
// Twiddle tw[k] and symbols of output position k of a line of n points:
// s2 = sin^2(pi f / n) of its frequency f, and (dense path) d2 = |D|^2 dx^2 of
// the 8th-order staggered derivative.
__device__ void table_entry(int n, const FftPlan& plan, int k, float2* tw, float* s2, float* d2) {
  double sn, cs;
  sincospi(-2.0 * k / n, &sn, &cs);
  tw[k] = make_float2((float)cs, (float)sn);
  const int f = nsr_digit_reverse(k, n, plan.radix, plan.nst);
  const double sp = sinpi((double)f / n);
  s2[k] = (float)(sp * sp);
  if (d2) {
    const double q = 2.0 * NSR_PI * f / n;
    double s = 0.0;
    for (int j = 0; j < 4; ++j) s += nsr_dense_stencil(j) * sin((j + 0.5) * q);
    d2[k] = (float)(4.0 * s * s);
  }
}

// Entry e of the per-stage twiddle rows (layout: FftPlan::tws), with the same
// rounding of the same angles as tw.
__device__ void stage_twiddle_entry(int n, const FftPlan& plan, int e, float2* tws) {
  int l = n, off = 0;
  for (int st = 0; st < plan.nst; ++st) {
    const int r = plan.radix[st], m = l / r;
    if (m > 1) {
      if (e < off + m * (r - 1)) {
        const int k = (e - off) / m + 1, j = (e - off) % m;
        double sn, cs;
        sincospi(-2.0 * (j * k * (n / l)) / n, &sn, &cs);
        tws[e] = make_float2((float)cs, (float)sn);
        break;
      }
      off += m * (r - 1);
    }
    l = m;
  }
}

// Every table of a grid in one launch (four to six small launches before, about
// 2.5 us each in front of every preconditioner call).
struct TableOut {
  float2 *twx, *twz, *twsx, *twsz;
  float *s2x, *s2z, *d2x, *d2z;
  int nwx, nwz;
};
__global__ void __launch_bounds__(128) k_fft_tables(FftPlan px, FftPlan pz, TableOut o) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < px.n) { table_entry(px.n, px, k, o.twx, o.s2x, o.d2x); return; }
  k -= px.n;
  if (k < pz.n) { table_entry(pz.n, pz, k, o.twz, o.s2z, o.d2z); return; }
  k -= pz.n;
  if (k < o.nwx) { stage_twiddle_entry(px.n, px, k, o.twsx); return; }
  k -= o.nwx;
  if (k < o.nwz) stage_twiddle_entry(pz.n, pz, k, o.twsz);
}

int nsr_prec_setup(const NsrGrid* g, PrecTables* t, void* table_mem, cudaStream_t st, float* d2x, float* d2z) {
  char* p = (char*)table_mem;
  t->px.n = g->nx;
  t->pz.n = g->nz;
  if (!nsr_make_radices(g->nx, t->px.radix, &t->px.nst)) return NSR_ERR_UNSUPPORTED_SIZE;
  if (!nsr_make_radices(g->nz, t->pz.radix, &t->pz.nst)) return NSR_ERR_UNSUPPORTED_SIZE;
  TableOut o;
  o.twx = (float2*)p; p += nsr_align(sizeof(float2) * g->nx);
  o.twz = (float2*)p; p += nsr_align(sizeof(float2) * g->nz);
  o.s2x = (float*)p; p += nsr_align(sizeof(float) * g->nx);
  o.s2z = (float*)p; p += nsr_align(sizeof(float) * g->nz);
  o.nwx = nsr_twiddle_offset(g->nx, 0);
  o.nwz = nsr_twiddle_offset(g->nz, 0);
  o.twsx = (float2*)p; p += nsr_align(sizeof(float2) * o.nwx);
  o.twsz = (float2*)p; p += nsr_align(sizeof(float2) * o.nwz);
  o.d2x = d2x;
  o.d2z = d2z;
  t->px.tw = o.twx; t->pz.tw = o.twz; t->s2x = o.s2x; t->s2z = o.s2z;
  t->px.tws = o.twsx; t->pz.tws = o.twsz;
  const int total = g->nx + g->nz + o.nwx + o.nwz;
  k_fft_tables<<<(total + 127) / 128, 128, 0, st>>>(t->px, t->pz, o);
  return last_error();
}

size_t nsr_prec_table_bytes(const NsrGrid* g) {
  return nsr_align(sizeof(float2) * g->nx) + nsr_align(sizeof(float2) * g->nz) +
         nsr_align(sizeof(float) * g->nx) + nsr_align(sizeof(float) * g->nz) +
         nsr_align(sizeof(float2) * nsr_twiddle_offset(g->nx, 0)) +
         nsr_align(sizeof(float2) * nsr_twiddle_offset(g->nz, 0));
}

// 16 columns (128-byte row segments) up to 1024 points; 8 for longer columns, and
// for batches of fewer 16-column tiles than SMs.  Two 16-column tiles fit an SM's
// shared memory up to 908 points; between there and 1024, which the solver has
// taken 16 wide from its first version, 8 are faster (22 learned systems of
// 1024 x 1536: 0.233 ms a launch against 0.309) and the autotuner's cols_width
// finds them.
int nsr_cols_tc(const NsrGrid* g, int ns) {
  return g->nz <= 1024 && (long long)ns * ((g->nx + 15) / 16) >= 148 ? 16 : 8;
}

// Stand-alone passes of nsr_precondition.  The ends of the transforms run
// between registers and global memory (rows_forward, cols_multiply,
// rows_inverse); each pass reads and writes a field once.  Eleven 768 x 1024
// fields, rows / columns / rows: 75 / 113 / 58 us staged through shared memory,
// 46 / 67 / 38 us in this form (21 us each at the copy rate).
template <bool GEN>
__global__ void __launch_bounds__(256, GEN ? 2 : 4) k_prec_rows_fwd(Geo g, PrecTables t, const float2* __restrict__ x,
                                                                    float2* __restrict__ w, int rows) {
  extern __shared__ float2 sm[];
  const long long n = (long long)g.nz * g.nx;
  const int z0 = blockIdx.x * rows;
  const long long off = blockIdx.y * n + (long long)z0 * g.nx;
  const float2* __restrict__ xs = x + off;
  rows_forward<GEN>(sm, min(rows, g.nz - z0), t.px, w + off, [&](auto tag, int k0, int step, float2* v) {
#pragma unroll
    for (int q = 0; q < decltype(tag)::value; ++q) v[q] = xs[k0 + q * step];
  });
}

template <int TC, bool GEN>
__global__ void __launch_bounds__(GEN ? 256 : 512, 2) k_prec_cols(Geo g, PrecTables t, const double* __restrict__ freq,
                                                                  float2* __restrict__ w, double shift, int adjoint) {
  extern __shared__ float2 sm[];
  const long long n = (long long)g.nz * g.nx;
  cols_pass_fixed<TC, GEN>(sm, g, t, w + blockIdx.y * n, freq[blockIdx.y], shift, adjoint, blockIdx.x * TC);
}

template <bool GEN>
__global__ void __launch_bounds__(256, GEN ? 2 : 4) k_prec_rows_inv(Geo g, PrecTables t, const float2* __restrict__ w,
                                                                    float2* __restrict__ y, int rows) {
  extern __shared__ float2 sm[];
  const long long n = (long long)g.nz * g.nx;
  const int z0 = blockIdx.x * rows;
  const long long off = blockIdx.y * n + (long long)z0 * g.nx;
  float2* __restrict__ ys = y + off;
  rows_inverse<GEN>(sm, min(rows, g.nz - z0), t.px, w + off, [&](int k, float2 v, int, int) { ys[k] = v; });
}

extern "C" size_t nsr_precondition_workspace_size(const NsrGrid* grid, int32_t n_systems) {
  if (nsr_check_grid(grid, true) || n_systems < 0) return 0;
  return nsr_prec_table_bytes(grid) + nsr_align(sizeof(float2) * (size_t)grid->nz * grid->nx * n_systems);
}

extern "C" int nsr_precondition(const NsrGrid* grid, const double* freq_hz, int32_t n_systems,
                                double shift, int32_t adjoint, const float* x, float* y,
                                void* workspace, size_t workspace_bytes, void* stream) {
  int err = nsr_check_grid(grid, true);
  if (err) return err;
  if (!freq_hz || !x || !y || !workspace || n_systems < 0 || n_systems > 65535) return NSR_ERR_ARGUMENT;
  if (n_systems == 0) return 0;
  if (workspace_bytes < nsr_precondition_workspace_size(grid, n_systems)) return NSR_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  PrecTables t;
  err = nsr_prec_setup(grid, &t, workspace, st);
  if (err) return err;
  float2* w = (float2*)((char*)workspace + nsr_prec_table_bytes(grid));
  Geo g = make_geo(*grid);
  const int rows = nsr_rows_per_cta(grid, n_systems);
  const size_t row_smem = sizeof(float2) * (size_t)rows * nsr_row_stride(grid->nx);
  dim3 gr((grid->nz + rows - 1) / rows, n_systems);
  const bool gx = nsr_rows_generic(grid->nx, w);
  if (!gx) k_prec_rows_fwd<false><<<gr, 256, row_smem, st>>>(g, t, (const float2*)x, w, rows);
  else k_prec_rows_fwd<true><<<gr, 256, row_smem, st>>>(g, t, (const float2*)x, w, rows);
  const int tc = nsr_cols_tc(grid, n_systems);
  const bool gen = !nsr_specialised(grid->nz);
  const dim3 gc((grid->nx + tc - 1) / tc, n_systems);
  const size_t csm = sizeof(float2) * (size_t)grid->nz * tc;
  const auto cols = tc == 16 ? (gen ? k_prec_cols<16, true> : k_prec_cols<16, false>)
                             : (gen ? k_prec_cols<8, true> : k_prec_cols<8, false>);
  cudaFuncSetAttribute((const void*)cols, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)csm);
  cols<<<gc, nsr_cols_threads(gen), csm, st>>>(g, t, freq_hz, w, shift, adjoint);
  if (!gx) k_prec_rows_inv<false><<<gr, 256, row_smem, st>>>(g, t, w, (float2*)y, rows);
  else k_prec_rows_inv<true><<<gr, 256, row_smem, st>>>(g, t, w, (float2*)y, rows);
  return last_error();
}

// Row tiles near 32 KB of shared memory (40 KB where the transform's first radix
// may be a large prime: four rows of 1216 give all 256 threads a butterfly, 107 ->
// 96 us for eleven 1056 x 1216 fields, the one width it was measured at), at most
// 8 rows; half or a quarter of that
// for batches of fewer than four such tiles for three SMs (solves of three 256 x
// 256 and six 256 x 384 systems take 4% less with the tile rules).
int nsr_rows_per_cta(const NsrGrid* g, int ns) {
  int rows = (int)((nsr_specialised(g->nx) ? 4096 : 5120) / g->nx);
  if (rows < 1) rows = 1;
  if (rows > 8) rows = 8;
  while (rows > 2 && 3LL * ns * ((g->nz + rows - 1) / rows) < 4 * 148) rows = (rows + 1) / 2;
  return rows;
}

// ---------------------------------------------------------------------------
// Plane-wave right-hand side (SI units, c128).
// ---------------------------------------------------------------------------
__global__ void k_plane_wave_rhs(Geo g, const double* __restrict__ freq, const double* __restrict__ angle,
                                 double2* __restrict__ b) {
  const long long n = (long long)g.nz * g.nx;
  const int sysi = blockIdx.y;
  const SysScalars s = sys_scalars(g, freq[sysi]);
  const double st = sin(angle[sysi]);
  const double inv_h2 = 1.0 / (g.h * g.h);
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k / g.nx), j = (int)(k - (long long)i * g.nx);
    double2 v = make_double2(0.0, 0.0);
    if (i == g.face) {
      double2 l = source_line(g, s.k0, st, j);
      v = make_double2(-l.x * inv_h2, -l.y * inv_h2);
    }
    b[sysi * n + k] = v;
  }
}

extern "C" int nsr_plane_wave_rhs(const NsrGrid* grid, const double* freq_hz, const double* angle_rad,
                                  int32_t n_systems, void* b, void* stream) {
  int err = nsr_check_grid(grid, false);
  if (err) return err;
  if (!freq_hz || !angle_rad || !b || n_systems < 0 || n_systems > 65535) return NSR_ERR_ARGUMENT;
  if (n_systems == 0) return 0;
  long long n = (long long)grid->nz * grid->nx;
  int bx = (int)((n + 255) / 256);
  if (bx > 4096) bx = 4096;
  k_plane_wave_rhs<<<dim3(bx, n_systems), 256, 0, (cudaStream_t)stream>>>(make_geo(*grid), freq_hz, angle_rad,
                                                                           (double2*)b);
  return last_error();
}

// ---------------------------------------------------------------------------
// Material gradient: -Re(lambda^H dA/dm u) for m = log c, log rho.
// d mass / d log c  = -2 k0^2 sx sz b (1 + i e)
// d mass / d log rho = -mass
// each edge e=(i,j): d(lam^H A u)/d log rho_i = a_i w_e conj(lam_j - lam_i)(u_j - u_i),
// w_e = stretch_e / (2 h^2).
// ---------------------------------------------------------------------------
//
// A thread owns one column of a TZ-row tile and keeps its nodes' sums in
// registers while the systems go by; the tile of u and lam of the next system is
// copied into shared memory (cp.async) while the present one is summed.  The edge term is the same product at both
// ends of an edge, so each south edge is formed once and carried to the next
// row, each east edge once and handed to the next lane.  With c = (k0 h)^2 sx sz and onepie = 1 + i e the sums are kept without
// b and a:  acc_c = 2 sum Re(conj(lam) u c onepie),  acc_r = sum Re(conj(lam) u
// c onepie^2),  acc_e = sum Re(edges); everything is FP64 as before.  Bound by
// FP64 issue and conversions (about 40 FP64 operations and 8 conversions per
// node and system).  22 systems of 1024 x 1536: 1,152 us with one thread per
// node, a pow and six PML profiles per node and system; 270 us with the x edges formed at both ends, 251 us in this form.
// TX threads of a block take one column each.  Columns a block yields: a warp's
// first lane only forms the east edge its neighbour needs, and the last lane of a
// one-warp block has no east neighbour in the tile.
__host__ __device__ constexpr int grad_own(int TX) { return TX == 32 ? 30 : 31 * (TX / 32); }
#define NSR_GRAD_CHUNK 64    // systems whose scalars are staged in shared memory at a time

__device__ __forceinline__ void cp_async_zfill(float2* dst, const float2* src, bool live) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(live ? 8 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_zfill(double2* dst, const double2* src, bool live) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory"); }

// Columns c0 .. c0 + TX - 1 of the rows z0 - 1 .. z0 + TZ of a field (zero outside
// the grid).
template <typename CT, int TZ, int TX>
struct GradTile {
  CT u[TZ + 2][TX], l[TZ + 2][TX];
};
template <typename CT, int TZ, int TX>
__device__ __forceinline__ void grad_fetch(GradTile<CT, TZ, TX>& t, const Geo& g, const CT* us, const CT* ls, int z0,
                                           int c0) {
#pragma unroll
  for (int r = 0; r < TZ + 2; ++r) {
    const int i = z0 - 1 + r;
    const bool row = i >= 0 && i < g.nz;
    const int j = c0 + threadIdx.x;
    const bool live = row && j >= 0 && j < g.nx;
    const long long id = live ? (long long)i * g.nx + j : 0;
    cp_async_zfill(&t.u[r][threadIdx.x], us + id, live);
    cp_async_zfill(&t.l[r][threadIdx.x], ls + id, live);
  }
  cp_async_commit();
}

template <typename CT, int TZ, int TX>
__global__ void __launch_bounds__(TX, TX == 32 ? 16 : 5) k_grad(Geo g, const void* __restrict__ mat,
                                                         const double* __restrict__ freq, int ns,
                                                         const CT* __restrict__ u, const CT* __restrict__ lam,
                                                         double* __restrict__ gc, double* __restrict__ gr) {
  __shared__ SysScalars scs[NSR_GRAD_CHUNK];
  extern __shared__ __align__(16) unsigned char grad_smem[];
  GradTile<CT, TZ, TX>* tiles = reinterpret_cast<GradTile<CT, TZ, TX>*>(grad_smem);   // two: one in use, one in flight
  const long long n = (long long)g.nz * g.nx;
  const int nx = g.nx, nz = g.nz;
  // Tile column tx is grid column c0 + tx; warp w takes 32 of them from 31 w on, and
  // its lanes 1 .. 31 own theirs.
  constexpr int OWN = grad_own(TX);
  const int nbx = (nx + OWN - 1) / OWN;
  const int c0 = (blockIdx.x % nbx) * OWN - 1;
  const int lane = threadIdx.x & 31, tx = 31 * (threadIdx.x >> 5) + lane;
  const int j = c0 + tx;
  const int z0 = (blockIdx.x / nbx) * TZ;
  // The east neighbour; a one-warp block's last lane has none.
  const int te = TX == 32 ? min(tx + 1, TX - 1) : tx + 1;
  const bool own = lane > 0 && (TX > 32 || lane < 31) && j < nx;
  const int jc = min(max(j, 0), nx - 1);
  const MatPlanes mp = nsr_planes(mat, n);
  grad_fetch(tiles[0], g, u, lam, z0, c0);
  const bool col_plain = j > g.n_pml && j < nx - 1 - g.n_pml;
  // PML profiles of the column at j and j + 1/2 (zero off the PML)
  const double px = col_plain ? 0.0 : pml_profile<double>((double)j, nx, g.n_pml);
  const double pxe = col_plain ? 0.0 : pml_profile<double>(j + 0.5, nx, g.n_pml);
  const bool warp_plain = __all_sync(0xffffffffu, col_plain || j >= nx);
  double acc_c[TZ], acc_r[TZ], acc_e[TZ];
  double t64[TZ];
#pragma unroll
  for (int q = 0; q < TZ; ++q) {
    acc_c[q] = acc_r[q] = acc_e[q] = 0.0;
    t64[q] = z0 + q < nz ? __ldg(&mp.t64[(long long)(z0 + q) * nx + jc]) : 0.0;
  }
  auto D = [](CT v) { return make_double2((double)v.x, (double)v.y); };
  // conj(dl) du
  auto prod = [](double2 dl, double2 du) {
    return make_double2(dl.x * du.x + dl.y * du.y, dl.x * du.y - dl.y * du.x);
  };
  for (int s0 = 0; s0 < ns; s0 += NSR_GRAD_CHUNK) {
    const int cnt = min(NSR_GRAD_CHUNK, ns - s0);
    __syncthreads();
    for (int q = threadIdx.x; q < cnt; q += TX) scs[q] = sys_scalars(g, freq[s0 + q]);
    for (int q = 0; q < cnt; ++q) {
      const int sys = s0 + q;
      __syncthreads();   // the tile about to be refilled has been read
      if (sys + 1 < ns) {
        grad_fetch(tiles[(sys + 1) & 1], g, u + (long long)(sys + 1) * n, lam + (long long)(sys + 1) * n, z0, c0);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      const GradTile<CT, TZ, TX>& t = tiles[sys & 1];
      const SysScalars s = scs[q];
      // 1 / (1 + i sig p) of the column's east half node
      double2 ie = make_double2(1.0, 0.0);
      if (!warp_plain) ie = inv_stretch(s.sig * pxe);
      const double2 sx = make_double2(1.0, s.sig * px);
      double2 uc = D(t.u[1][tx]), lc = D(t.l[1][tx]);
      double north;   // Re(w conj(dl) du) of the edge to the row above
      {
        const double2 p = prod(D(t.l[0][tx]) - lc, D(t.u[0][tx]) - uc);
        north = p.x;
        if (!(warp_plain && z0 > g.n_pml && z0 <= nz - 1 - g.n_pml)) {
          const double2 w = sx * inv_stretch(s.sig * pml_profile<double>(z0 - 0.5, nz, g.n_pml));
          north = w.x * p.x - w.y * p.y;
        }
      }
#pragma unroll
      for (int r = 0; r < TZ; ++r) {
        const int i = z0 + r;
        const double2 un = D(t.u[r + 2][tx]), ln = D(t.l[r + 2][tx]);
        const double2 due = D(t.u[r + 1][te]) - uc, dle = D(t.l[r + 1][te]) - lc;
        const double2 dus = un - uc, dls = ln - lc;
        const double2 lu = prod(lc, uc);
        const double e = t64[r] * s.fpow;
        const bool row_plain = i > g.n_pml && i < nz - 1 - g.n_pml;
        if (row_plain && warp_plain) {
          const double south = dls.x * dus.x + dls.y * dus.y;
          const double east = dle.x * due.x + dle.y * due.y;
          const double west = __shfl_up_sync(0xffffffffu, east, 1);
          acc_e[r] += 0.5 * (east + west + south + north);
          north = south;
          const double ei = e * lu.y;
          acc_c[r] += s.kh2 * (lu.x - ei);
          acc_r[r] += s.kh2 * (lu.x * (1.0 - e * e) - 2.0 * ei);
        } else {
          const double2 pe = prod(dle, due), ps = prod(dls, dus);
          const double2 sz = make_double2(1.0, s.sig * pml_profile<double>((double)i, nz, g.n_pml));
          const double2 we = sz * ie;
          const double2 ws = sx * inv_stretch(s.sig * pml_profile<double>(i + 0.5, nz, g.n_pml));
          const double south = ws.x * ps.x - ws.y * ps.y;
          const double east = we.x * pe.x - we.y * pe.y;
          const double west = __shfl_up_sync(0xffffffffu, east, 1);
          acc_e[r] += 0.5 * (east + west + south + north);
          north = south;
          const double2 cell = sx * sz;
          const double2 c1 = cell * make_double2(1.0, e), c2 = cell * make_double2(1.0 - e * e, 2.0 * e);
          acc_c[r] += s.kh2 * (lu.x * c1.x - lu.y * c1.y);
          acc_r[r] += s.kh2 * (lu.x * c2.x - lu.y * c2.y);
        }
        uc = un;
        lc = ln;
      }
    }
  }
  if (!own) return;
  const double inv_h2 = 1.0 / (g.h * g.h);
#pragma unroll
  for (int r = 0; r < TZ; ++r) {
    if (z0 + r >= nz) break;
    const long long k = (long long)(z0 + r) * nx + j;
    const double b = mp.b64[k], a = mp.a64[k];
    gc[k] += 2.0 * b * acc_c[r] * inv_h2;
    gr[k] += (b * acc_r[r] - a * acc_e[r]) * inv_h2;
  }
}

template <typename CT, int TX>
static cudaError_t launch_grad_tx(const Geo& g, const void* coef, const double* freq, int ns, const void* u,
                                  const void* lam, double* gc, double* gr, cudaStream_t st) {
  // 4-row tiles read 6 rows for 4, from L2; a grid whose 4-row tiles would
  // leave SMs without sixteen warps takes 2-row tiles.
  const int bx = (g.nx + grad_own(TX) - 1) / grad_own(TX);
  const CT *pu = (const CT*)u, *pl = (const CT*)lam;
  cudaError_t ce;
  if ((long long)bx * ((g.nz + 3) / 4) * TX >= 4 * 148 * 128) {
    const int smem = 2 * (int)sizeof(GradTile<CT, 4, TX>);
    ce = cudaFuncSetAttribute(k_grad<CT, 4, TX>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (ce != cudaSuccess) return ce;
    k_grad<CT, 4, TX><<<bx * ((g.nz + 3) / 4), TX, smem, st>>>(g, coef, freq, ns, pu, pl, gc, gr);
  } else {
    const int smem = 2 * (int)sizeof(GradTile<CT, 2, TX>);
    k_grad<CT, 2, TX><<<bx * ((g.nz + 1) / 2), TX, smem, st>>>(g, coef, freq, ns, pu, pl, gc, gr);
  }
  return cudaGetLastError();
}
// One-warp blocks where a block of 128 columns would be half empty or more (22
// fields of 2048 x 8: 58 us a call with 128 columns, 30 us with 32).
template <typename CT>
static cudaError_t launch_grad(const Geo& g, const void* coef, const double* freq, int ns, const void* u,
                               const void* lam, double* gc, double* gr, cudaStream_t st) {
  return g.nx <= 60 ? launch_grad_tx<CT, 32>(g, coef, freq, ns, u, lam, gc, gr, st)
                    : launch_grad_tx<CT, 128>(g, coef, freq, ns, u, lam, gc, gr, st);
}

extern "C" int nsr_grad_accum(const NsrGrid* grid, const void* coef, const double* freq_hz,
                              int32_t n_systems, int32_t precision, const void* u, const void* lam,
                              double* g_logc, double* g_logrho, void* stream) {
  int err = nsr_check_grid(grid, false);
  if (err) return err;
  if (!coef || !freq_hz || !u || !lam || !g_logc || !g_logrho || n_systems < 0) return NSR_ERR_ARGUMENT;
  if (precision != 0 && precision != 1) return NSR_ERR_ARGUMENT;
  if (n_systems == 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  const Geo g = make_geo(*grid);
  const cudaError_t ce = precision == 0 ? launch_grad<float2>(g, coef, freq_hz, n_systems, u, lam, g_logc, g_logrho, st)
                                        : launch_grad<double2>(g, coef, freq_hz, n_systems, u, lam, g_logc, g_logrho, st);
  return ce == cudaSuccess ? 0 : (int)ce;
}

// ---------------------------------------------------------------------------
// Tangent right-hand side -dA[dm] u (the Born perturbation of
// theranostic/wave.py:280-329 for a direction dm = (dlog c, dlog rho)).
// The flux part is the stencil evaluated with a' = -a dlogrho and zero ghost
// contrast (the fluxes are linear in a); the mass part is
// -2 k0^2 sx sz b (1+ie) dlogc - k0^2 sx sz b (1+ie)^2 dlogrho.  Output in SI
// units, the units of the solver's right-hand side.
// ---------------------------------------------------------------------------
template <typename CT>
__global__ void k_tangent(Geo g, const void* __restrict__ mat, const double* __restrict__ freq,
                          const CT* __restrict__ u, const double* __restrict__ dlogc,
                          const double* __restrict__ dlogrho, CT* __restrict__ rhs) {
  const long long n = (long long)g.nz * g.nx;
  const int sidx = blockIdx.y;
  const SysScalars s = sys_scalars(g, freq[sidx]);
  const MatPlanes mp = nsr_planes(mat, n);
  const CT* us = u + sidx * n;
  const double inv_h2 = 1.0 / (g.h * g.h);
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k / g.nx), j = (int)(k - (long long)i * g.nx);
    auto U = [&](int i2, int j2) -> double2 {
      if (i2 < 0 || i2 >= g.nz || j2 < 0 || j2 >= g.nx) return make_double2(0.0, 0.0);
      const CT q = us[(long long)i2 * g.nx + j2];
      return make_double2((double)q.x, (double)q.y);
    };
    auto DA = [&](int i2, int j2) -> double {
      if (i2 < 0 || i2 >= g.nz || j2 < 0 || j2 >= g.nx) return 0.0;
      const long long id = (long long)i2 * g.nx + j2;
      return -mp.a64[id] * dlogrho[id];
    };
    const double2 flux = stencil<double, false>(g, s, i, j, 0.0, mp.t64[k], U, DA);
    const double sig = s.sig;
    const double2 sx = make_double2(1.0, sig * pml_profile<double>((double)j, g.nx, g.n_pml));
    const double2 sz = make_double2(1.0, sig * pml_profile<double>((double)i, g.nz, g.n_pml));
    const double2 onepie = make_double2(1.0, mp.t64[k] * s.fpow);
    const double2 cell = (s.kh2 * mp.b64[k]) * (sx * sz);
    const double2 dmass = (-2.0 * dlogc[k]) * (cell * onepie) + (-dlogrho[k]) * (cell * (onepie * onepie));
    const double2 d = flux + dmass * U(i, j);
    const double2 r = (-inv_h2) * d;
    CT o;
    o.x = r.x;
    o.y = r.y;
    rhs[sidx * n + k] = o;
  }
}

extern "C" int nsr_tangent_rhs(const NsrGrid* grid, const void* coef, const double* freq_hz, int32_t n_systems,
                               int32_t precision, const void* u, const double* dlogc, const double* dlogrho,
                               void* rhs, void* stream) {
  int err = nsr_check_grid(grid, false);
  if (err) return err;
  if (!coef || !freq_hz || !u || !dlogc || !dlogrho || !rhs || n_systems < 0 || n_systems > 65535)
    return NSR_ERR_ARGUMENT;
  if (precision != 0 && precision != 1) return NSR_ERR_ARGUMENT;
  if (n_systems == 0) return 0;
  long long n = (long long)grid->nz * grid->nx;
  int bx = (int)((n + 255) / 256);
  if (bx > 148 * 8) bx = 148 * 8;
  dim3 gd(bx, n_systems);
  cudaStream_t st = (cudaStream_t)stream;
  if (precision == 0)
    k_tangent<float2><<<gd, 256, 0, st>>>(make_geo(*grid), coef, freq_hz, (const float2*)u, dlogc, dlogrho,
                                          (float2*)rhs);
  else
    k_tangent<double2><<<gd, 256, 0, st>>>(make_geo(*grid), coef, freq_hz, (const double2*)u, dlogc, dlogrho,
                                           (double2*)rhs);
  return last_error();
}

// ---------------------------------------------------------------------------
// Band-limited RF traces from receiver spectra (predict_band_rf,
// nsrno/wave_operator.py:169-180): the inverse real DFT with 'forward'
// normalisation of a spectrum that is zero except on the given positive bins,
//   x[t] = sum_b 2 Re(S[b] exp(2 pi i k_b t / n)),   0 < k_b < n/2.
// The phase k_b t is reduced modulo n in integers, so every term is exact to
// double rounding whatever the trace length.
// ---------------------------------------------------------------------------
__global__ void k_band_rf(int n_ch, int n_bins, int n, const double2* __restrict__ spec,
                          const int* __restrict__ bins, double* __restrict__ out) {
  const int ch = blockIdx.y;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    double acc = 0.0;
    for (int b = 0; b < n_bins; ++b) {
      const long long m = ((long long)bins[b] * t) % n;
      double sn, cs;
      sincospi(2.0 * (double)m / (double)n, &sn, &cs);
      const double2 s = spec[(long long)ch * n_bins + b];
      acc += 2.0 * (s.x * cs - s.y * sn);
    }
    out[(long long)ch * n + t] = acc;
  }
}

extern "C" int nsr_band_rf(int32_t n_channels, int32_t n_bins, int32_t n_samples, const double* spectrum,
                           const int32_t* bins, double* rf, void* stream) {
  if (n_channels < 0 || n_bins < 0 || n_samples <= 0 || n_channels > 65535 || !rf ||
      (n_bins > 0 && (!spectrum || !bins)))
    return NSR_ERR_ARGUMENT;
  if (n_channels == 0) return 0;
  cudaStream_t st = (cudaStream_t)stream;
  if (n_bins == 0) {
    cudaError_t e = cudaMemsetAsync(rf, 0, sizeof(double) * (size_t)n_channels * n_samples, st);
    return e == cudaSuccess ? 0 : (int)e;
  }
  const int bx = (n_samples + 255) / 256;
  k_band_rf<<<dim3(bx, n_channels), 256, 0, st>>>(n_channels, n_bins, n_samples, (const double2*)spectrum, bins, rf);
  return last_error();
}

// ---------------------------------------------------------------------------
// FP64 true relative residual ||b - A x|| / ||b|| of n_systems fields
// (the acceptance check of nsrno/dense_wave.py:146-147,221-225 and
// theranostic/wave.py:320-323).  b is the given SI right-hand side or, when
// rhs is null, the plane-wave source of (freq, angle).  Per-CTA partials are
// summed in CTA order by a second kernel, so the result is deterministic.
// ---------------------------------------------------------------------------
#define NSR_TR_BLOCKS 256
__global__ void __launch_bounds__(256) k_true_residual(Geo g, const void* __restrict__ mat,
                                                       const double* __restrict__ freq,
                                                       const double* __restrict__ angle,
                                                       const double2* __restrict__ x, const double2* __restrict__ rhs,
                                                       int adjoint, double* __restrict__ partials) {
  const long long n = (long long)g.nz * g.nx;
  const int sidx = blockIdx.y;
  const SysScalars s = sys_scalars(g, freq[sidx]);
  const MatPlanes mp = nsr_planes(mat, n);
  const double2* xs = x + sidx * n;
  const double st = angle ? sin(angle[sidx]) : 0.0;
  const double h2 = g.h * g.h;
  double rr = 0.0, bb = 0.0;
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n; k += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(k / g.nx), j = (int)(k - (long long)i * g.nx);
    auto P = [&](int i2, int j2) -> double2 {
      if (i2 < 0 || i2 >= g.nz || j2 < 0 || j2 >= g.nx) return make_double2(0.0, 0.0);
      return xs[(long long)i2 * g.nx + j2];
    };
    auto Aa = [&](int i2, int j2) -> double {
      if (i2 < 0 || i2 >= g.nz || j2 < 0 || j2 >= g.nx) return 1.0;
      return mp.a64[(long long)i2 * g.nx + j2];
    };
    double2 b;
    if (rhs) {
      b = h2 * rhs[sidx * n + k];
    } else if (i == g.face) {
      const double2 l = source_line(g, s.k0, st, j);
      b = make_double2(-l.x, -l.y);
    } else {
      b = make_double2(0.0, 0.0);
    }
    const double2 ax = adjoint ? stencil<double, true>(g, s, i, j, mp.b64[k], mp.t64[k], P, Aa)
                               : stencil<double, false>(g, s, i, j, mp.b64[k], mp.t64[k], P, Aa);
    const double2 r = b - ax;
    rr += r.x * r.x + r.y * r.y;
    bb += b.x * b.x + b.y * b.y;
  }
  __shared__ double wr[8], wb[8];
  for (int o = 16; o > 0; o >>= 1) {
    rr += __shfl_xor_sync(0xffffffffu, rr, o);
    bb += __shfl_xor_sync(0xffffffffu, bb, o);
  }
  if ((threadIdx.x & 31) == 0) { wr[threadIdx.x >> 5] = rr; wb[threadIdx.x >> 5] = bb; }
  __syncthreads();
  if (threadIdx.x == 0) {
    double tr = 0.0, tb = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { tr += wr[w]; tb += wb[w]; }
    partials[((long long)sidx * gridDim.x + blockIdx.x) * 2] = tr;
    partials[((long long)sidx * gridDim.x + blockIdx.x) * 2 + 1] = tb;
  }
}

__global__ void k_true_residual_sum(int n_systems, int nb, const double* __restrict__ partials,
                                    double* __restrict__ residual) {
  const int sidx = blockIdx.x * blockDim.x + threadIdx.x;
  if (sidx >= n_systems) return;
  double rr = 0.0, bb = 0.0;
  for (int b = 0; b < nb; ++b) {
    rr += partials[((long long)sidx * nb + b) * 2];
    bb += partials[((long long)sidx * nb + b) * 2 + 1];
  }
  residual[sidx] = bb > 0.0 ? sqrt(rr / bb) : sqrt(rr);
}

extern "C" size_t nsr_true_residual_workspace_size(const NsrGrid* grid, int32_t n_systems) {
  if (nsr_check_grid(grid, false) || n_systems <= 0 || n_systems > 65535) return 0;
  return nsr_align(sizeof(double) * 2 * NSR_TR_BLOCKS * (size_t)n_systems);
}

extern "C" int nsr_true_residual(const NsrGrid* grid, const void* coef, const double* freq_hz,
                                 const double* angle_rad, int32_t n_systems, int32_t adjoint, const double* x,
                                 const double* rhs, double* residual, void* workspace, size_t workspace_bytes,
                                 void* stream) {
  int err = nsr_check_grid(grid, false);
  if (err) return err;
  if (!coef || !freq_hz || !x || !residual || !workspace || n_systems < 0 || n_systems > 65535) return NSR_ERR_ARGUMENT;
  if (!rhs && !angle_rad) return NSR_ERR_ARGUMENT;
  if (n_systems == 0) return 0;
  if (workspace_bytes < nsr_true_residual_workspace_size(grid, n_systems)) return NSR_ERR_WORKSPACE;
  cudaStream_t st = (cudaStream_t)stream;
  double* partials = (double*)workspace;
  k_true_residual<<<dim3(NSR_TR_BLOCKS, n_systems), 256, 0, st>>>(make_geo(*grid), coef, freq_hz,
                                                                   rhs ? nullptr : angle_rad, (const double2*)x,
                                                                   (const double2*)rhs, adjoint ? 1 : 0, partials);
  k_true_residual_sum<<<(n_systems + 127) / 128, 128, 0, st>>>(n_systems, NSR_TR_BLOCKS, partials, residual);
  return last_error();
}
