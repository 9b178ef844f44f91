// Declarations shared between the translation units of the nsrno_b200 library.
#pragma once

#include "nsr_common.cuh"

// FFT plans and digit-reversed symbol tables of one grid.
struct PrecTables {
  FftPlan px, pz;      // along x (rows) and z (columns)
  const float* s2x;    // sin^2(pi kx / nx) at digit-reversed x positions
  const float* s2z;    // sin^2(pi kz / nz) at digit-reversed z positions
};

inline size_t nsr_align(size_t b) { return (b + 255) & ~(size_t)255; }

int nsr_check_grid(const NsrGrid* g, bool need_fft);
// Tables of a grid, one launch; d2x, d2z (optional): the dense path's symbols.
int nsr_prec_setup(const NsrGrid* g, PrecTables* t, void* table_mem, cudaStream_t st, float* d2x = nullptr,
                   float* d2z = nullptr);
size_t nsr_prec_table_bytes(const NsrGrid* g);
// Columns and rows per CTA of the transform passes over ns fields.
int nsr_cols_tc(const NsrGrid* g, int ns);
int nsr_rows_per_cta(const NsrGrid* g, int ns);

// Threads of a column-pass CTA: the run-time transforms take half as many
// (their butterflies hold up to 19 points in registers).
inline int nsr_cols_threads(bool gen) { return gen ? 256 : 512; }

// Whether a row pass between caller's fields and the work field `w` runs the
// run-time stages: the specialised transforms read and write w in 16-byte pairs,
// which a workspace that is only 8-byte aligned does not allow.
inline bool nsr_rows_generic(int nx, const void* w) { return !nsr_specialised(nx) || ((uintptr_t)w & 15) != 0; }

int nsr_check_learned(const NsrLearned* L, int n_systems, cudaStream_t st);
