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
template <int TILE, typename AT>
__device__ __forceinline__ void gs_dots(const double2* tile, const float2* __restrict__ V, long long stride, int nv,
                                        AT at, double* part, int nb, int block) {
  constexpr int NW = NSR_GS_THREADS / 32;
  constexpr int U = TILE / (32 * NW) < 8 ? TILE / (32 * NW) : 8;   // loads in flight per lane
  __shared__ double piece[NW][2];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int log_p = 0;   // 2^log_p warps per vector
  while ((nv << (log_p + 1)) <= NW) ++log_p;
  const int span = TILE >> log_p;
  for (int q = wid; q < (nv << log_p); q += NW) {
    const int i = q >> log_p, first = (q & ((1 << log_p) - 1)) * span;
    const float2* __restrict__ v = V + i * stride;
    double re = 0.0, im = 0.0;
    for (int e0 = first + lane; e0 < first + span; e0 += 32 * U) {
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

// Counts this block in; in the last of `nb` blocks returns true with the sums
// of the `nv` partial columns (in block order within each lane, then over the
// lanes: the same on every run) in tot.
__device__ __forceinline__ bool gs_arrive(double* part, int nb, int nv, int* arrive, double* tot) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(arrive, 1) == nb - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int q = wid; q < nv; q += NSR_GS_THREADS / 32) {
    double s = 0.0;
#pragma unroll 4
    for (int b = lane; b < nb; b += 32) s += __ldcg(&part[(long long)q * nb + b]);
    s = warp_sum(s);
    if (lane == 0) tot[q] = s;
  }
  if (threadIdx.x == 0) *arrive = 0;
  __syncthreads();
  return true;
}
