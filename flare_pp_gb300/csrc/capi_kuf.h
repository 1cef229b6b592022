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
// form's time is per environment.  Where the two meet (adjoint / this form, us):
//  - four structures or more: below 10 environments with 18 to 816 descriptors (24 cells, N = 3,
//    lmax = 2, one species, 10 environments: 2426 / 1962; N = 16, lmax = 5: 18248 / 18226); at
//    13 to 16 above (two species, N = 10, lmax = 4, 12 and 13: 13142 / 15058, 15606 / 15093;
//    N = 12, 14: 19293 / 20120); at 10 to 24 below (one descriptor, four cells of 32 atoms,
//    16 and 24: 240 / 251, 262 / 254);
//  - fewer, where the longer chain of launches shows (one cell of 108 atoms): one species,
//    N = 1, lmax = 0, 48: 197 / 227; N = 4, lmax = 2, 16 and 24: 188 / 238, 243 / 243; two
//    species, N = 8, lmax = 3, 16 and 24: 322 / 340, 445 / 349.
inline int kuf_gemm_sparse(int n_d, int n_structures) {
  if (n_structures < 4) return n_d < 16 ? 64 : n_d < 128 ? 24 : 20;
  return n_d < 16 ? 24 : n_d < 1000 ? 10 : 16;
}
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
