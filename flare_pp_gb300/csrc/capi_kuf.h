// Host side of the kernel columns by one GEMM (kuf_gemm.cu).
#pragma once
#include <vector>

#include "capi_state.h"
#include "kuf_gemm.h"

namespace fpp {

// A structure and its label columns: q.col_e, q.col_s and either q.force_col (device)
// or col_f0, the column of atom 0's x force (the other atoms follow; -1: no forces).
struct KufItem {
  fpp_structure *s;
  KufStruc q;
  long long col_f0;
};

// Fewest sparse environments of a species for which fpp_kuf_batched takes this form.  Its
// derivative rows and tiles cost the same for one environment as for tens, the adjoint
// form's time is per environment: 32 cells of 8,460 atoms, N = 8, lmax = 3, two species,
// 4 / 8 / 16 / 32 environments per species: 3.1 / 6.7 / 12.2 / 24.7 ms by the adjoint,
// 7.6 / 8.0 / 8.1 / 8.5 by this form.
constexpr int kKufGemmSparse = 10;
// Largest structure (bytes of its pairs' rows): above it fpp_kuf_batched takes the
// adjoint form, which needs no memory per pair.
constexpr size_t kKufGemmStructure = (size_t)16 << 30;

bool kuf_gemm_fits(const fpp_model *m);
// device memory that n_pairs pairs of one structure take
size_t kuf_gemm_bytes(const fpp_model *m, long long n_pairs);
// Label columns of the items into dK (n_sparse_total x n_labels, row-major; columns that
// are no item's stay as they are).  The structures' FP64 descriptors (forward64) have
// been queued on st.  Queued on st; synchronizes once per slice.
int kuf_gemm(fpp_model *m, KufWork &w, const std::vector<KufItem> &items, double *dK,
             long long n_labels, cudaStream_t st);

}  // namespace fpp
