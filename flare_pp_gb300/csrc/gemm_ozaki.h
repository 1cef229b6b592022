// FP64-accurate C = A B^T from exact fp16 digit planes on the tcgen05 tensor
// cores (gemm_ozaki.cu).  Row-major A (M x K), B (N x K), C (M x N).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstddef>

#include "common.cuh"

namespace fpp {

constexpr int kOzakiDigits = 8;  // balanced digits per operand entry
constexpr int kOzakiBits = 7;    // bits per digit (|digit| <= 64)
constexpr int kOzakiMaxGroups = 8;

// Padded shape of one operand's digit planes: rows to a multiple of 128,
// K to a multiple of 64; plane_bytes covers all kOzakiDigits planes.
struct OzakiShape {
  int rows_pad, k_pad;
  size_t plane_bytes;
};
OzakiShape ozaki_shape(int rows, int K);

// Digit planes (kOzakiDigits x rows_pad x k_pad fp16, zero padded) and the
// exponent e of each row (max |row| < 2^e; kOzakiNanRow if the row holds a
// non-finite entry) of X (rows x K, row stride ldx, device memory).
constexpr int kOzakiNanRow = -(1 << 30);
// Powers of two by which the columns are scaled before the split, exactly: column k of the
// rows from row0[g] on (up to the next group's) by 2^(sign shift[g][k]), where shift[g] (device,
// 16-byte aligned, K entries padded to a multiple of four) is not null.  With 2^shift on one
// operand and 2^-shift on the other the product is the same, but what counts as a row's
// largest entry is not.
struct OzakiColumns {
  const int *shift[kOzakiMaxGroups] = {};
  int row0[kOzakiMaxGroups] = {};
  int n = 0, sign = 1;
};
// row_ptr (device): where each row starts, instead of X and ldx.
int launch_ozaki_split(int rows, int K, const double *X, long long ldx, __half *planes,
                       int *exps, cudaStream_t stream, const double *const *row_ptr = nullptr,
                       const OzakiColumns *cols = nullptr);
// Such powers of two for a symmetric matrix (finite, n x n, row stride lda): the largest
// |a_ij| 2^(-shift_i - shift_j) of every row about 1.  tmp: scratch of the same size.
int launch_equilibrate(int n, const double *a, int lda, int *shift, int *tmp,
                       cudaStream_t stream);

// An operand split by launch_ozaki_split.
struct OzakiMat {
  const __half *planes;
  const int *exps;
  int rows, K;
};

// One product of a grouped launch: C (M x N, row stride ldc) = A B^T with rows
// a_row0 .. a_row0 + M of operand a and rows b_row0 .. b_row0 + N of operand b.  C need not
// be initialised.  b_lower: B is lower triangular (B[n][k] = 0 for k > n; an
// L^-1, or an R^-1 transposed), and the K blocks above each column tile's last
// row are skipped.  Rows or columns with a non-finite operand come out NaN.
struct OzakiProblem {
  OzakiMat a, b;
  int a_row0, M, N;
  double *C;
  long long ldc;
  bool b_lower;
  int b_row0 = 0;
};
// Up to kOzakiMaxGroups products in one persistent launch (their tiles share
// the SMs).  n_levels: 8, or 9 where the dropped digit pairs must stay below the
// operands' rounding (43 pairs instead of 36).  0 on success.
int launch_ozaki_gemm(const OzakiProblem *probs, int n_probs, DeviceStatus *status,
                      cudaStream_t stream, int n_levels = 8);

}  // namespace fpp
