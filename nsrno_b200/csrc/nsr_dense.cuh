// Pieces of the dense path shared by its entry points and its solver.
#pragma once

#include "nsr_internal.cuh"

struct DenseGeo {
  int H, W, pz, px, h, w;
  double dx;
  double2 scal;   // (D - 1) / (D k0^2)
};

// The fixed preconditioner of one call or solve: tables and the transformed
// fields in the caller's workspace, and its launch shapes.
struct DensePrec {
  DenseGeo geo;
  PrecTables t;
  float *d2x, *d2z;
  float2* w;
  float inv_k0dx2, shift;
  int adjoint, rows, tc;
  bool gx, gz;            // run-time transforms along x, z
  dim3 g_rows, g_cols;
  size_t row_smem, col_smem;
};

DenseGeo nsr_dense_geo(const NsrDenseGrid* grid, double scal_re, double scal_im);
// y = A x or A^H x of checked arguments; 0 or a CUDA error.
int nsr_dense_apply_geo(const DenseGeo& g, const double* coef, int n_fields, int adjoint, int precision,
                        const void* x, void* y, cudaStream_t st);
// Tables (one launch) and shapes; the workspace is that of nsr_dense_precondition.
int nsr_dense_prec_setup(const NsrDenseGrid* grid, double k0dx2, double shift, int n_fields, int adjoint,
                         void* workspace, cudaStream_t st, DensePrec* M);
// The column pass on M.w and the masked inverse row pass into y, after a
// forward row pass has filled M.w.
void nsr_dense_prec_finish(const DensePrec& M, float2* y, cudaStream_t st);
