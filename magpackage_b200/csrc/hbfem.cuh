// Harmonic-balance assembly (hbfem.cu).
#pragma once

#include <cuda_runtime.h>

#include "common.cuh"

namespace mag {

constexpr int kMaxHarm = 16;  // harmonics per call

// Whether the constant-curl kernel serves this call (it can also hand back the time-averaged
// reluctivity, from which the DC block is one stiffness assembly). dc: the DC block is wanted.
bool hbfem_constant_curls(const QuadParams &qp, int K, int N, int64_t ne, bool dc);

// Residual (and, when vals is given, the DC block) of one harmonic field. rscr: [Ne][6][2K]
// workspace. nu_dc [Ne], only with hbfem_constant_curls: receives the time-averaged
// reluctivity; the caller then assembles the DC block from it. NULL: the DC block goes
// through scratch and the row reduction.
int launch_hbfem(const ElemData &m, const RowPlan &rp, int max_row, const double *sr, const double *si, int K,
                 const double *dr, const double *di, const double *pr, const double *pi, int N,
                 const QuadParams &qp, const MaterialParams &mp, double *scratch, double *rscr, double *nu_dc,
                 double *vals, double *out_re, double *out_im, cudaStream_t s);

}  // namespace mag
