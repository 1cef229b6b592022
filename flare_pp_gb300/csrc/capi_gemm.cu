// C ABI and host helper of the FP64-accurate tensor-core GEMM (gemm_ozaki.cu).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>

#include "capi_state.h"
#include "gemm_ozaki.h"
#include "internal.h"

namespace fpp {

int ozaki_split(OzakiOperand &op, int rows, int K, const double *X, long long ldx,
                cudaStream_t st, const OzakiColumns *cols) {
  const OzakiShape sh = ozaki_shape(rows, K);
  // one allocation: the planes, then the row exponents
  FPP_TRY(op.buf.reserve(sh.plane_bytes + sizeof(int) * (size_t)std::max(rows, 1)));
  op.rows = rows;
  op.K = K;
  op.exps_at = sh.plane_bytes;
  if (launch_ozaki_split(rows, K, X, ldx, op.planes(), op.exps(), st, nullptr, cols) != 0)
    return fail(FPP_ERR_CUDA, "digit-plane split launch failed");
  return FPP_OK;
}

int ozaki_const(OzakiOperand &op, int rows, int K, const double *X, long long ldx,
                cudaStream_t st, const OzakiColumns *cols) {
  if (op.ready && op.rows == rows && op.K == K) return FPP_OK;
  op.ready = false;
  FPP_TRY(ozaki_split(op, rows, K, X, ldx, st, cols));
  FPP_CUDA(cudaStreamSynchronize(st));  // later calls may run on other streams
  op.ready = true;
  return FPP_OK;
}

OzakiMat ozaki_mat(const OzakiOperand &op) {
  return OzakiMat{op.planes(), op.exps(), op.rows, op.K};
}

int ozaki_run(const OzakiProblem *probs, int n, DeviceStatus *status, cudaStream_t st,
              int n_levels) {
  const int rc = launch_ozaki_gemm(probs, n, status, st, n_levels);
  if (rc != 0) return fail(FPP_ERR_CUDA, "tensor-core FP64 GEMM launch failed (" +
                                             std::to_string(rc) + ")");
  return FPP_OK;
}

int ozaki_status(OzakiWork &w, cudaStream_t st, DeviceStatus **out) {
  if (w.status.bytes < sizeof(DeviceStatus)) {  // cleared once, then by each check
    FPP_TRY(w.status.reserve(sizeof(DeviceStatus)));
    FPP_CUDA(cudaMemsetAsync(w.status.ptr, 0, sizeof(DeviceStatus), st));
  }
  *out = w.status.as<DeviceStatus>();
  return FPP_OK;
}

int ozaki_dgemm_nt(int M, int N, int K, const double *A, long long lda, const double *B,
                   long long ldb, double *C, long long ldc, OzakiWork &w, cudaStream_t st,
                   bool b_lower) {
  if (M <= 0 || N <= 0) return FPP_OK;
  if (K <= 0) return fail(FPP_ERR_INVALID, "GEMM with K <= 0");
  DeviceStatus *status;
  FPP_TRY(ozaki_status(w, st, &status));
  FPP_TRY(ozaki_split(w.a, M, K, A, lda, st));
  FPP_TRY(ozaki_split(w.b, N, K, B, ldb, st));
  const OzakiProblem q{ozaki_mat(w.a), ozaki_mat(w.b), 0, M, N, C, ldc, b_lower};
  return ozaki_run(&q, 1, status, st);
}

int ozaki_check_status(OzakiWork &w, cudaStream_t st) {
  if (w.status.bytes < sizeof(DeviceStatus)) return FPP_OK;  // nothing ran
  DeviceStatus h;
  FPP_CUDA(cudaMemcpyAsync(&h, w.status.ptr, sizeof(h), cudaMemcpyDeviceToHost, st));
  FPP_CUDA(cudaStreamSynchronize(st));
  if (h.code != 0) FPP_CUDA(cudaMemsetAsync(w.status.ptr, 0, sizeof(DeviceStatus), st));
  if (h.code != 0)
    return fail(h.code, "tensor-core FP64 GEMM: a bounded wait ran out (site " +
                            std::to_string(h.where) + ")");
  return FPP_OK;
}

}  // namespace fpp

using namespace fpp;

extern "C" int fpp_dgemm_nt(int32_t M, int32_t N, int32_t K, const double *A, int64_t lda,
                            const double *B, int64_t ldb, double *C, int64_t ldc,
                            int32_t on_device, void *stream) {
  if ((M > 0 && N > 0) && (!A || !B || !C)) return fail(FPP_ERR_INVALID, "null argument");
  if (M < 0 || N < 0 || K < 0) return fail(FPP_ERR_INVALID, "negative size");
  if (M == 0 || N == 0) return FPP_OK;
  if (K == 0) {
    if (on_device) {
      FPP_CUDA(cudaMemset2DAsync(C, sizeof(double) * ldc, 0, sizeof(double) * N, M,
                                 (cudaStream_t)stream));
    } else {
      for (int i = 0; i < M; i++) std::fill(C + (size_t)i * ldc, C + (size_t)i * ldc + N, 0.0);
    }
    return FPP_OK;
  }
  if (lda < K || ldb < K || ldc < N) return fail(FPP_ERR_INVALID, "leading dimension too small");
  cudaStream_t st = (cudaStream_t)stream;
  OzakiWork w;
  if (on_device) {
    FPP_TRY(ozaki_dgemm_nt(M, N, K, A, lda, B, ldb, C, ldc, w, st));
    return ozaki_check_status(w, st);
  }
  DevBuf dA, dB, dC;
  FPP_TRY(dA.reserve(sizeof(double) * (size_t)M * K));
  FPP_TRY(dB.reserve(sizeof(double) * (size_t)N * K));
  FPP_TRY(dC.reserve(sizeof(double) * (size_t)M * N));
  FPP_CUDA(cudaMemcpy2DAsync(dA.ptr, sizeof(double) * K, A, sizeof(double) * lda,
                             sizeof(double) * K, M, cudaMemcpyHostToDevice, st));
  FPP_CUDA(cudaMemcpy2DAsync(dB.ptr, sizeof(double) * K, B, sizeof(double) * ldb,
                             sizeof(double) * K, N, cudaMemcpyHostToDevice, st));
  FPP_TRY(ozaki_dgemm_nt(M, N, K, dA.as<double>(), K, dB.as<double>(), K, dC.as<double>(), N,
                         w, st));
  FPP_TRY(ozaki_check_status(w, st));
  FPP_CUDA(cudaMemcpy2DAsync(C, sizeof(double) * ldc, dC.ptr, sizeof(double) * N,
                             sizeof(double) * N, M, cudaMemcpyDeviceToHost, st));
  FPP_CUDA(cudaStreamSynchronize(st));
  return FPP_OK;
}
