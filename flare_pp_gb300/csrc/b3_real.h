// The real-arithmetic FP32 form of the B3 coupling (b3_real.cu).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <vector>

#include "b2_kernels.h"

namespace fpp {

// Whether the mixed form of a B3 descriptor with nr radial channels runs in it
// (lmax 1..3, a block's shared memory holds an atom).
bool b3_real_fits(int lmax, int nr);

// Its operand columns: for each, the descriptor column it holds (triples in order,
// the triangles with even l1 + l2 + l3), -1 for the padding to a multiple of four.
std::vector<int> b3_real_columns(int lmax, int n_tri);

// From the single-bond coefficients c (noa x nr x H): |p| (float-float in 8-byte
// slots) and the rows of the centred split operand, nd columns.
int launch_b3_couple(const B2Args &a, int nd, const int *species, const int *row_of_atom,
                     const float *c_in, double *norm_out, __half *phat_hi, __half *phat_lo,
                     int ldp, const float *pbar, cudaStream_t stream);
// The mixed power-2 adjoint, part 1: atom energies and u = dE/dc.
int launch_b3_adjoint(const B2Args &a, int nd, const AdjArgs &g, const int *species,
                      const int *row_of_atom, const float *c_in, const double *norm_in,
                      double *atom_e, float *u_out, cudaStream_t stream);

}  // namespace fpp
