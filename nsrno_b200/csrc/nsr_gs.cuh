// Gram-Schmidt building blocks of the two GMRES solvers (the 5-point batch and
// the dense path): FP64 inner products of a tile of w with the basis, and the
// sum of the tiles' partials by the last block to arrive.
//
// A block holds a tile of w in shared memory, already converted to double, and
// its warps take the basis vectors in turn: a warp streams one vector's tile,
// so an inner product costs one warp reduction per tile and no block barrier.
// (One thread per few nodes looping over the vectors needed a local array of
// partials and two block barriers per value: 228 us for 5 vectors of eleven
// 768 x 1024 systems.)
#pragma once

#include "nsr_device.cuh"

#define NSR_GS_THREADS 256

// part[q * nb + block] = partial of value q: re, im of <v_i, w> for i < nv.
// `at(e)` is the global index of tile element e; outside the vector it is any
// index inside it, and tile[e] is zero (a condition around the loads kept them
// from being issued together).  With fewer vectors than warps, several warps share a
// vector's tile.  Called by the whole block.
template <int U, typename AT>
__device__ __forceinline__ void gs_warp_dot(const double2* tile, const float2* __restrict__ v, int first, int last,
                                            AT at, double& re, double& im) {
  for (int e0 = first; e0 < last; e0 += 32 * U) {   // U loads in flight per lane
    float2 x[U];
#pragma unroll
    for (int u = 0; u < U; ++u) x[u] = v[at(e0 + 32 * u)];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double2 w = tile[e0 + 32 * u];
      const double a = x[u].x, b = x[u].y;
      re += a * w.x + b * w.y;
      im += a * w.y - b * w.x;
    }
  }
}

template <int TILE, typename AT>
__device__ __forceinline__ void gs_dots(const double2* tile, const float2* __restrict__ V, long long stride, int nv,
                                        AT at, double* part, int nb, int block) {
  constexpr int NW = NSR_GS_THREADS / 32;
  constexpr int U = TILE / (32 * NW) < 8 ? TILE / (32 * NW) : 8;   // where all warps share one vector
  __shared__ double piece[NW][2];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int log_p = 0;   // 2^log_p warps per vector
  while ((nv << (log_p + 1)) <= NW) ++log_p;
  const int span = TILE >> log_p;
  for (int q = wid; q < (nv << log_p); q += NW) {
    const int i = q >> log_p, first = (q & ((1 << log_p) - 1)) * span;
    const float2* __restrict__ v = V + i * stride;
    double re = 0.0, im = 0.0;
    if (span >= 256) gs_warp_dot<8>(tile, v, first + lane, first + span, at, re, im);
    else gs_warp_dot<U>(tile, v, first + lane, first + span, at, re, im);
    re = warp_sum(re);
    im = warp_sum(im);
    if (lane == 0) {
      if (log_p == 0) {
        part[(long long)(2 * i) * nb + block] = re;
        part[(long long)(2 * i + 1) * nb + block] = im;
      } else {
        piece[q][0] = re;
        piece[q][1] = im;
      }
    }
  }
  if (log_p == 0) return;
  __syncthreads();
  if (threadIdx.x < 2 * nv) {
    const int i = threadIdx.x >> 1, c = threadIdx.x & 1;
    double s = 0.0;
    for (int k = 0; k < (1 << log_p); ++k) s += piece[(i << log_p) + k][c];
    part[(long long)threadIdx.x * nb + block] = s;
  }
}

// Sum over a block of one double per thread (valid in thread 0).
__device__ __forceinline__ double gs_block_sum(double v) {
  __shared__ double wsum[NSR_GS_THREADS / 32];
  v = warp_sum(v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int k = 0; k < NSR_GS_THREADS / 32; ++k) t += wsum[k];
  return t;
}

// Counts this block in; in the last block of the launch's row returns true with
// the sums of the `nv` columns of `nb` partials (in order within each lane, then
// over the lanes: the same on every run) in tot.
__device__ __forceinline__ bool gs_arrive(double* part, int nb, int nv, int* arrive, double* tot) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(arrive, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // Four columns a warp at a time, so that their loads are in flight together: the
  // last block works alone here.
  for (int q0 = 4 * wid; q0 < nv; q0 += 4 * (NSR_GS_THREADS / 32)) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
    for (int b = lane; b < nb; b += 32)
#pragma unroll
      for (int u = 0; u < 4; ++u) s[u] += __ldcg(&part[(long long)min(q0 + u, nv - 1) * nb + b]);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      s[u] = warp_sum(s[u]);
      if (lane == 0 && q0 + u < nv) tot[q0 + u] = s[u];
    }
  }
  if (threadIdx.x == 0) *arrive = 0;
  __syncthreads();
  return true;
}

// Column j of the Hessenberg matrix (h + h', then the next norm) and the Givens
// rotations, in shared memory: one thread applies the rotations, and every global
// value is read and written by the block at once.  (One thread walking global
// memory paid an L2 latency per entry.)
struct GsColumn {
  double2 h[66], sn[65];
  double cs[65];
  double norm;      // h_{j+1,j}
  double2 g0, g1;   // gv[j], gv[j + 1] after the new rotation
};
// `rotate` computes the new rotation from (a, norm): c, s and the new diagonal.
template <typename ROT>
__device__ __forceinline__ void gs_finish_column(GsColumn& k, int j, const double* tot, const double2* hc, double2* hc2,
                                                 double2* col, double* cs, double2* sn, double2* gv, ROT rotate) {
  for (int i = threadIdx.x; i <= j; i += NSR_GS_THREADS) {
    const double2 h2 = make_double2(tot[2 * i], tot[2 * i + 1]);
    hc2[i] = h2;
    k.h[i] = hc[i] + h2;
    if (i < j) {
      k.cs[i] = cs[i];
      k.sn[i] = sn[i];
    }
  }
  if (threadIdx.x == 0) k.g0 = gv[j];
  __syncthreads();
  if (threadIdx.x == 0) {
    double nrm = tot[2 * (j + 1)];
    for (int i = 0; i <= j; ++i) nrm -= tot[2 * i] * tot[2 * i] + tot[2 * i + 1] * tot[2 * i + 1];
    k.norm = nrm > 0.0 ? sqrt(nrm) : (nrm <= 0.0 ? 0.0 : nrm);   // a NaN stays one
    double2 a = k.h[0];
    for (int i = 0; i < j; ++i) {
      const double2 b = k.h[i + 1];
      k.h[i] = k.cs[i] * a + k.sn[i] * b;
      a = k.cs[i] * b - conjc(k.sn[i]) * a;
    }
    double c;
    double2 s, d;
    rotate(a, k.norm, &c, &s, &d);
    k.h[j] = d;
    k.h[j + 1] = make_double2(0.0, 0.0);
    cs[j] = c;
    sn[j] = s;
    const double2 g = k.g0;
    k.g0 = c * g;
    k.g1 = make_double2(0.0, 0.0) - conjc(s) * g;
    gv[j] = k.g0;
    gv[j + 1] = k.g1;
  }
  __syncthreads();
  for (int i = threadIdx.x; i <= j + 1; i += NSR_GS_THREADS) col[i] = k.h[i];
}
