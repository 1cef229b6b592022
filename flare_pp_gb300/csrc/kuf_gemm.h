// Kernel columns of training structures (Kuf, envs_struc) from one GEMM over the
// descriptor pairs' derivative rows.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "b2_kernels.h"

namespace fpp {

// Column of a class's compact descriptor rows: the radial channels n1 (all species)
// and n2 (of the neighbor's species, local), degree l, and the descriptor it is.
struct KufColumn {
  unsigned short n1;
  unsigned char n2, l;
  int d;
};

// A structure of the batch: its tables, and where its pairs, rows and columns lie.
struct KufGemmStruc {
  KufStruc s;
  const int *nbr_i, *rev;
  int noa, n_pairs;
  int pair0;                 // first of its pairs in the batch's pair list
  int chunk;                 // chunk it is evaluated in
  int atom0;                 // first of its atoms in the chunk
  int block0, n_blocks;      // its atom blocks in the chunk
  int want_pairs, want_es;   // force or stress labels; energy or stress labels
  long long col_f0;          // force_col null: column of atom 0 (the rest follow), or -1
  int zbase[kMaxSpecies];    // z row of an atom: zbase[species] + row_of_atom
};

constexpr int kKufAtoms = 8;     // atoms of a gather block (a warp each)

struct KufGemmArgs {
  B2Args a;
  const KufGemmStruc *strucs;
  int n_strucs, n_chunks;
  KufSpecies sp[kMaxSpecies];
  double sig2, power;
  int ldp;
  double *kuf;
  long long n_labels;
  // the batch's pairs ordered by (chunk, central species, neighbor species)
  unsigned int *keys_in, *keys;  // class of a pair; n_chunks n_species^2: left out
  int *vals_in, *vals;           // pair of the batch
  int *start;                    // first place of each class (classes + 1 entries)
  int *place;                    // pair of the batch -> place, or -1
  int n_pairs;
  // rows 3 (place - place0) + component of one unit (a chunk, some species)
  int place0, n_places;
  int s0, s1;                    // species of the unit
  const KufColumn *cols;         // n_species x kc
  int kc, k_same;                // columns; the first k_same have n1 of that species too
  __half *planes;
  int rows_pad, k_pad;
  int *exps;
  double *t;                     // phat . dp of each row
  double *f;                     // rows x ldf: dhat_k . dp
  int ldf;
  double *z, *acoef;             // z rows x ldf: z, and dk/dz / |p|
  double *tsum;                  // per chunk atom: sum t (3), sum t (x) r (6)
  double *partial;               // [block][7][n_sparse_total] energy and virial sums
  const int2 *blocks;            // (structure, first atom) of the chunk's atom blocks
  int n_blocks, struc0, struc1;  // structures of the chunk
  int tiles[kMaxSpecies + 1];    // first sparse tile of each species of the unit
  int n_sparse_total;
};

int upload_kuf_tables(cudaStream_t stream);  // constant memory of kuf_gemm.cu
// shared memory of the derivative rows' kernel and its warps (0: does not fit)
size_t kuf_rows_smem(const B2Args &a, int kc, int *warps);
int launch_kuf_classes(const KufGemmArgs &k, int max_pairs, cudaStream_t st);
int launch_kuf_places(const KufGemmArgs &k, int n_classes, cudaStream_t st);
int launch_kuf_compact(int rows, int kc, const double *const *src, const int *sj,
                       const KufColumn *cols, double *dst, cudaStream_t st);
int launch_kuf_rows(const KufGemmArgs &k, cudaStream_t st);
int launch_kuf_coef(const KufGemmArgs &k, cudaStream_t st);
int launch_kuf_gather(const KufGemmArgs &k, cudaStream_t st);

}  // namespace fpp
