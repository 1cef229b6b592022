// Kernel columns of training structures (Kuf; envs_struc,
// normalized_dot_product.cpp:115-210) by one product over the pairs' derivatives:
//   rows dp[(pair, component)] = d p_i / d r_ij  (FP64, cut into digit planes where
//     they are formed), columns the sparse environments of the central species:
//   f = dp dhat^T, z = phat dhat^T on the tensor cores (gemm_ozaki.cu);
//   dk/dr_ij = a_ik (f - z_ik t),  t = phat_i . dp,  a = sig^2 power z^(power-1) / |p_i|,
// and each atom gathers its own and its reverse pairs (no atomics: every sum runs in a
// fixed order).
//
// Pairs are ordered by (chunk of structures, central species, neighbor species): a
// pair's derivative is zero in the descriptors without a channel of the neighbor's
// species, so a class's rows and its dhat columns leave those out (400 of 544 columns
// with two species of eight channels).
//
// Why: the adjoint form (k_kuf_adjoint, b2_kernels.cu) contracts dk/dc with each pair's
// basis for every sparse environment on the FP64 pipe (2 instructions per clock and
// SM); here the work per (pair, environment) on that pipe is fifteen adds of the
// gather, and the contraction runs at the tensor cores' FP64-equivalent rate.  32 cells of
// 8,460 atoms (354,000 pairs), N = 8, lmax = 3, two species of 150 environments each:
// 76.7 ms by the adjoint; here 10.4 ms: GEMM 3.8, rows 3.6, descriptors 0.9, gather 1.4.
// One cell of 256 atoms (envs_struc; stored derivatives before): 0.50 ms instead of 1.8.
#include <cuda_runtime.h>

#include <algorithm>

#include "basis.cuh"
#include "kuf_gemm.h"
#include "ozaki_split.cuh"

namespace fpp {

__device__ __forceinline__ double kpow(double z, double p) {
  if (p == 2.0) return z * z;
  if (p == 1.0) return z;
  if (p == 0.0) return 1.0;
  return pow(z, p);
}

__device__ __forceinline__ double wsum64(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__global__ void __launch_bounds__(256)
k_kuf_classes(const KufGemmArgs k) {
  const KufGemmStruc &S = k.strucs[blockIdx.y];
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= S.n_pairs) return;
  const int ns = k.a.n_species;
  const int i = S.nbr_i[p], si = S.s.species[i], sj = S.s.nbr_s[p];
  const bool keep = S.want_pairs && k.sp[si].n_sparse > 0 && S.s.norm64[i] >= 1e-8 &&
                    S.s.rel[p].x <= k.a.cutoffs[si * ns + sj];  // b2.cpp:277
  const int none = k.n_chunks * ns * ns;
  k.keys_in[S.pair0 + p] = keep ? (S.chunk * ns + si) * ns + sj : none;
  k.vals_in[S.pair0 + p] = S.pair0 + p;
}

__global__ void __launch_bounds__(256) k_kuf_places(const KufGemmArgs k, int n_classes) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t > k.n_pairs) return;
  // one past the end closes the classes that nothing follows
  const int key = t < k.n_pairs ? min((int)k.keys[t], n_classes) : n_classes;
  const int prev = t > 0 ? min((int)k.keys[t - 1], n_classes) : -1;
  for (int c = prev + 1; c <= key; c++) k.start[c] = t;
  if (t < k.n_pairs) k.place[k.vals[t]] = key < n_classes ? t : -1;
}

// Rows of dhat in a class's columns.
__global__ void __launch_bounds__(128)
k_kuf_compact(int kc, const double *const *__restrict__ src, const int *__restrict__ sj,
              const KufColumn *__restrict__ cols, double *__restrict__ dst) {
  const double *x = src[blockIdx.x];
  const KufColumn *tab = cols + (size_t)sj[blockIdx.x] * kc;
  for (int d = threadIdx.x; d < kc; d += blockDim.x)
    dst[(size_t)blockIdx.x * kc + d] = x[tab[d].d];
}

// ---------------------------------------------------------------------------
// Derivative rows.  A block takes up to 32 consecutive places: one warp evaluates their
// bases, a lane per pair (FP64 instructions cost the same for one lane as for 32),
// then each warp forms the three rows of its pairs from the factored sums
//   alpha[n1, l] = sum_m c[n1, lm] Y[lm],  beta_c[n1, l] = sum_m c[n1, lm] dY[lm]/dr_c:
//   dp_c[(n1, n2), l] = g'_{n2} rhat_c alpha[n1, l] + g_{n2} beta_c[n1, l]
//                       (+ n1 <-> n2 if n1 is of the neighbor's species too),
// six or twelve FP64 instructions for the three components of a column (2 (2 l + 1)
// per component and term with the products of c and dc).  A row waits in shared
// memory for its largest entry, then goes out as digit planes.
//
// Bound by the FP64 pipe (83 % of the active cycles at 41,600 pairs, 592 us; profiles/
// kuf_rows_gather.txt).  On the way there, at 32,000 pairs (484 us): bases by the general
// recurrence 703 us; the split's digits one after the other instead of bit
// fields, and one loop over both kinds of columns, whose branch became predicated FP64
// instructions, 664 us.
// ---------------------------------------------------------------------------
constexpr int kRowPairs = 32, kRowStride = 33;  // most pairs of a block

// channels of a degree's sums, odd: the degrees of a column group in different banks
__host__ __device__ inline int sums_stride(const B2Args &a) {
  return (a.n_species * a.N) | 1;
}
__host__ __device__ inline size_t rows_shared_doubles(const B2Args &a) {
  return (size_t)(2 * a.N + 4 * a.H) * kRowStride + 3 * kRowPairs;
}
// static shared memory of the kernel (m_i, m_sj, m_struc), out of the same limit
constexpr size_t kRowStatic = 3 * sizeof(int) * kRowPairs;
__host__ __device__ inline size_t rows_warp_doubles(const B2Args &a, int kc) {
  return (size_t)6 * sums_stride(a) * (a.lmax + 1) + ((kc + 3) & ~3);
}

// L: lmax (0..4), or -1 for any
template <int L>
__global__ void __launch_bounds__(256) k_kuf_rows(const KufGemmArgs k, int block_pairs) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int m_i[kRowPairs], m_sj[kRowPairs], m_struc[kRowPairs];
  double *sm = reinterpret_cast<double *>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarp = blockDim.x >> 5;
  const B2Args &a = k.a;
  const int N = a.N, H = a.H, ns = a.n_species, L1 = a.lmax + 1, nr = ns * N;
  const int nrs = sums_stride(a), nl = nrs * L1;
  // rows first (16-byte aligned), then the sums, the bases and the unit vectors
  const int kcp = (k.kc + 3) & ~3;
  double *row = sm + (size_t)warp * kcp;
  double *ab = sm + (size_t)nwarp * kcp + (size_t)warp * 6 * nl;
  double *bas = sm + (size_t)nwarp * (kcp + 6 * nl);
  double *unit = bas + (size_t)(2 * N + 4 * H) * kRowStride;  // [3][32]
  const int t0 = blockIdx.x * block_pairs, np = min(block_pairs, k.n_places - t0);
  if (warp == 0 && lane < np) {
    const int gp = k.vals[k.place0 + t0 + lane];
    int lo = 0, hi = k.n_strucs - 1;  // the last structure whose pairs begin at or before gp
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (k.strucs[mid].pair0 <= gp) lo = mid; else hi = mid - 1;
    }
    const KufGemmStruc &S = k.strucs[lo];
    const int p = gp - S.pair0, i = S.nbr_i[p], si = S.s.species[i], sj = S.s.nbr_s[p];
    m_i[lane] = i;
    m_sj[lane] = sj;
    m_struc[lane] = lo;
    const dvec4 rd = S.s.rel[p];
    radial_basis<double>(rd.x, a.r1, a.cutoffs[si * ns + sj], N, a.cutoff_kind, bas + lane,
                         bas + N * kRowStride + lane, kRowStride, a.cinv64_hi[si * ns + sj],
                         a.cinv64_lo[si * ns + sj]);
    const double ir = 1.0 / rd.x, ux = rd.y * ir, uy = rd.z * ir, uz = rd.w * ir;
    double *Y = bas + 2 * N * kRowStride + lane, *dY = Y + H * kRowStride;
    if constexpr (L >= 0)
      harmonics64_grad<L>(ux, uy, uz, ir, Y, dY, kRowStride);
    else
      real_harmonics<double>(rd.y, rd.z, rd.w, a.lmax, Y, dY, kRowStride);
    unit[lane] = ux;
    unit[kRowPairs + lane] = uy;
    unit[2 * kRowPairs + lane] = uz;
  }
  __syncthreads();
  const size_t plane = (size_t)k.rows_pad * k.k_pad;
  for (int pi = warp; pi < np; pi += nwarp) {
    const KufGemmStruc &S = k.strucs[m_struc[pi]];
    const int i = m_i[pi], sj = m_sj[pi];
    const double *c = S.s.c64 + (size_t)i * nr * H;
    const double *phat = S.s.phat64 + (size_t)S.s.row_of_atom[i] * k.ldp;
    const double *g = bas + pi, *dg = bas + N * kRowStride + pi;
    const double *Y = bas + 2 * N * kRowStride + pi, *dY = bas + (2 * N + H) * kRowStride + pi;
    const double u[3] = {unit[pi], unit[kRowPairs + pi], unit[2 * kRowPairs + pi]};
    for (int q = lane; q < nr * L1; q += 32) {
      const int l = q / nr, n1 = q - l * nr, idx = l * nrs + n1;
      double al = 0.0, be[3] = {0.0, 0.0, 0.0};
      for (int lm = l * l; lm < (l + 1) * (l + 1); lm++) {
        const double cv = c[n1 * H + lm];
        al = fma(cv, Y[lm * kRowStride], al);
#pragma unroll
        for (int x = 0; x < 3; x++) be[x] = fma(cv, dY[(3 * lm + x) * kRowStride], be[x]);
      }
#pragma unroll
      for (int x = 0; x < 3; x++) {
        ab[x * nl + idx] = al * u[x];
        ab[(3 + x) * nl + idx] = be[x];
      }
    }
    __syncwarp();
    const KufColumn *tab = k.cols + (size_t)sj * k.kc;
    for (int q = 0; q < 3; q++) {
      const double *A = ab + q * nl, *B = ab + (3 + q) * nl;
      double td = 0.0;
      // both channels of the neighbor's species, then one (loops of their own: a branch
      // became predicated FP64 instructions for every column)
#pragma unroll 2
      for (int d = lane; d < k.k_same; d += 32) {
        const KufColumn w = tab[d];
        const int o = w.l * nrs, i1 = o + w.n1, i2 = o + sj * N + w.n2, n1 = w.n1 - sj * N;
        double v = fma(dg[w.n2 * kRowStride], A[i1], g[w.n2 * kRowStride] * B[i1]);
        v = fma(dg[n1 * kRowStride], A[i2], v);
        v = fma(g[n1 * kRowStride], B[i2], v);
        row[d] = v;
        td = fma(v, phat[w.d], td);
      }
#pragma unroll 4
      for (int d = k.k_same + lane; d < k.kc; d += 32) {
        const KufColumn w = tab[d];
        const int i1 = w.l * nrs + w.n1;
        const double v = fma(dg[w.n2 * kRowStride], A[i1], g[w.n2 * kRowStride] * B[i1]);
        row[d] = v;
        td = fma(v, phat[w.d], td);
      }
      __syncwarp();
      const int r = 3 * (t0 + pi) + q;
      const int e = ozaki_split_row(
          k.kc, k.k_pad, plane, k.planes + (size_t)r * k.k_pad, lane,
          [&](int d, unsigned long long (&b)[4]) {
            const ulonglong2 x = reinterpret_cast<const ulonglong2 *>(row + d)[0];
            const ulonglong2 y = reinterpret_cast<const ulonglong2 *>(row + d)[1];
            b[0] = x.x;
            b[1] = d + 1 < k.kc ? x.y : 0ull;
            b[2] = d + 2 < k.kc ? y.x : 0ull;
            b[3] = d + 3 < k.kc ? y.y : 0ull;
          });
      td = wsum64(td);
      if (lane == 0) {
        k.exps[r] = e;
        k.t[r] = td;
      }
      __syncwarp();
    }
  }
}

// a_ik = sig^2 power z^(power - 1) / |p_i| (zero for empty environments), and the sums
// of t over an atom's pairs: a warp per atom.
__global__ void __launch_bounds__(32 * kKufAtoms) k_kuf_coef(const KufGemmArgs k) {
  const int2 b = k.blocks[blockIdx.x];
  const KufGemmStruc &S = k.strucs[b.x];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = b.y + warp;
  if (i >= S.noa) return;
  const int si = S.s.species[i];
  if (si < k.s0 || si >= k.s1) return;
  const double nrm = S.s.norm64[i];
  const bool live = nrm >= 1e-8;
  const double pref = live ? k.sig2 * k.power / nrm : 0.0;
  const KufSpecies &SP = k.sp[si];
  const size_t zr = (size_t)(S.zbase[si] + S.s.row_of_atom[i]) * k.ldf;
  for (int kk = lane; kk < SP.n_sparse; kk += 32) {
    const double z = k.z[zr + kk];
    k.acoef[zr + kk] =
        live && SP.norms[kk] >= 1e-8 ? pref * kpow(z, k.power - 1.0) : 0.0;
  }
  if (!S.want_pairs) return;
  double T[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
  for (int p = S.s.offset[i] + lane; p < S.s.offset[i + 1]; p += 32) {
    const int q = k.place[S.pair0 + p];
    if (q < 0) continue;
    const double *t = k.t + 3 * (size_t)(q - k.place0);
    const dvec4 r = S.s.rel[p];
    T[0] += t[0];
    T[1] += t[1];
    T[2] += t[2];
    T[3] = fma(t[0], r.y, T[3]);
    T[4] = fma(t[0], r.z, T[4]);
    T[5] = fma(t[0], r.w, T[5]);
    T[6] = fma(t[1], r.z, T[6]);
    T[7] = fma(t[1], r.w, T[7]);
    T[8] = fma(t[2], r.w, T[8]);
  }
#pragma unroll
  for (int q = 0; q < 9; q++) T[q] = wsum64(T[q]);
  if (lane == 0)
#pragma unroll
    for (int q = 0; q < 9; q++) k.tsum[(size_t)(S.atom0 + i) * 9 + q] = T[q];
}

// Force columns of eight atoms (a warp each) for 32 sparse environments (a lane each):
//   F_a = a_ak (sum f - z_ak sum t) - sum_rev a_jk (f_rev - z_jk t_rev),
// own pairs only if the atom is of the environments' species; energies and virials
// a_ak (sum f (x) r - z_ak sum t (x) r) as partial sums of the block.
__global__ void __launch_bounds__(32 * kKufAtoms) k_kuf_gather(const KufGemmArgs k) {
  __shared__ double sm[kKufAtoms][7][33];
  const int2 b = k.blocks[blockIdx.x];
  const KufGemmStruc &S = k.strucs[b.x];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  int s = k.s0;
  while (s + 1 < k.s1 && (int)blockIdx.y >= k.tiles[s + 1]) s++;
  const KufSpecies &SP = k.sp[s];
  const int k0 = ((int)blockIdx.y - k.tiles[s]) * 32, kk = k0 + lane;
  const bool ok = kk < SP.n_sparse;
  const int ke = ok ? kk : 0;
  const int i = b.y + warp;
  const bool live_atom = i < S.noa;
  double F[3] = {0, 0, 0}, V[7] = {0, 0, 0, 0, 0, 0, 0};
  if (live_atom) {
    const int si = S.s.species[i];
    const bool own = si == s, vir = own && S.s.col_s >= 0;
    if (S.want_pairs) {
      double own_f[3] = {0, 0, 0};
      for (int p = S.s.offset[i]; p < S.s.offset[i + 1]; p++) {
        if (own) {
          const int q = k.place[S.pair0 + p];
          if (q >= 0) {
            const double *f = k.f + 3 * (size_t)(q - k.place0) * k.ldf + ke;
            const double f0 = f[0], f1 = f[k.ldf], f2 = f[2 * k.ldf];
            own_f[0] += f0;
            own_f[1] += f1;
            own_f[2] += f2;
            if (vir) {
              const dvec4 r = S.s.rel[p];
              V[1] = fma(f0, r.y, V[1]);
              V[2] = fma(f0, r.z, V[2]);
              V[3] = fma(f0, r.w, V[3]);
              V[4] = fma(f1, r.z, V[4]);
              V[5] = fma(f1, r.w, V[5]);
              V[6] = fma(f2, r.w, V[6]);
            }
          }
        }
        if (S.s.nbr_s[p] == s) {
          const int rv = S.rev[p];
          const int q = rv >= 0 ? k.place[S.pair0 + rv] : -1;
          if (q >= 0) {
            const size_t zr = (size_t)(S.zbase[s] + S.s.row_of_atom[S.s.nbr_j[p]]) * k.ldf + ke;
            const double ac = k.acoef[zr], z = k.z[zr];
            const double *f = k.f + 3 * (size_t)(q - k.place0) * k.ldf + ke;
            const double *t = k.t + 3 * (size_t)(q - k.place0);
#pragma unroll
            for (int c = 0; c < 3; c++)
              F[c] = fma(-ac, fma(-z, t[c], f[(size_t)c * k.ldf]), F[c]);
          }
        }
      }
      if (own) {
        const size_t zr = (size_t)(S.zbase[s] + S.s.row_of_atom[i]) * k.ldf + ke;
        const double ac = k.acoef[zr], z = k.z[zr];
        const double *T = k.tsum + (size_t)(S.atom0 + i) * 9;
#pragma unroll
        for (int c = 0; c < 3; c++) F[c] = fma(ac, fma(-z, T[c], own_f[c]), F[c]);
        if (vir)
#pragma unroll
          for (int c = 0; c < 6; c++) V[1 + c] = ac * fma(-z, T[3 + c], V[1 + c]);
      }
    }
    if (own && S.s.col_e >= 0 && S.s.norm64[i] >= 1e-8 && SP.norms[ke] >= 1e-8)
      V[0] = k.sig2 *
             kpow(k.z[(size_t)(S.zbase[s] + S.s.row_of_atom[i]) * k.ldf + ke], k.power);
  }
  // the block's forces, eight atoms of an environment side by side
  const bool forces = S.s.force_col || S.col_f0 >= 0;
  if (forces) {
#pragma unroll
    for (int c = 0; c < 3; c++) sm[warp][c][lane] = F[c];
    __syncthreads();
    const int at = threadIdx.x & (kKufAtoms - 1), row = threadIdx.x / kKufAtoms;
    const int ia = b.y + at;
    if (ia < S.noa && k0 + row < SP.n_sparse) {
      const long long col = S.s.force_col ? S.s.force_col[ia] : S.col_f0 + 3ll * ia;
      if (col >= 0) {
        double *dst = k.kuf + (size_t)(SP.row0 + k0 + row) * k.n_labels + col;
#pragma unroll
        for (int c = 0; c < 3; c++) dst[c] = sm[at][c][row];
      }
    }
    __syncthreads();
  }
  if (S.want_es) {
#pragma unroll
    for (int c = 0; c < 7; c++) sm[warp][c][lane] = V[c];
    __syncthreads();
    if (warp < 7 && ok) {
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < kKufAtoms; w++) v += sm[w][warp][lane];
      k.partial[((size_t)blockIdx.x * 7 + warp) * k.n_sparse_total + SP.row0 + kk] = v;
    }
  }
}

// Energy and stress columns: the blocks' partial sums of a structure, eight runs of
// blocks side by side and then in order.
__global__ void __launch_bounds__(256) k_kuf_es(const KufGemmArgs k, int row0, int rows) {
  __shared__ double sm[8][7][33];
  const KufGemmStruc &S = k.strucs[k.struc0 + blockIdx.y];
  if (!S.want_es) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = blockIdx.x * 32 + lane;
  double v[7] = {0, 0, 0, 0, 0, 0, 0};
  if (r < rows)
    for (int q = warp; q < S.n_blocks; q += 8)
#pragma unroll
      for (int c = 0; c < 7; c++)
        v[c] += k.partial[((size_t)(S.block0 + q) * 7 + c) * k.n_sparse_total + row0 + r];
#pragma unroll
  for (int c = 0; c < 7; c++) sm[warp][c][lane] = v[c];
  __syncthreads();
  if (warp < 7 && r < rows) {
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < 8; w++) t += sm[w][warp][lane];
    double *dst = k.kuf + (size_t)(row0 + r) * k.n_labels;
    if (warp == 0) {
      if (S.s.col_e >= 0) dst[S.s.col_e] = t;
    } else if (S.s.col_s >= 0) {
      dst[S.s.col_s + warp - 1] = -t * S.s.vol_inv;
    }
  }
}

// ---------------------------------------------------------------------------
int upload_kuf_tables(cudaStream_t st) {
  const HarmonicTables t = harmonic_tables();
  return cudaMemcpyToSymbolAsync(c_harm, &t, sizeof(t), 0, cudaMemcpyHostToDevice, st) ==
                 cudaSuccess
             ? 0
             : -1;
}

size_t kuf_rows_smem(const B2Args &a, int kc, int *warps) {
  // the most warps of a block that leave room for two blocks on an SM, else that fit
  for (size_t cap : {(size_t)113 * 1024, (size_t)227 * 1024})
    for (int w = 8; w >= 1; w >>= 1) {
      const size_t b =
          sizeof(double) * (rows_shared_doubles(a) + w * rows_warp_doubles(a, kc));
      if (b + kRowStatic > cap || (cap < 200 * 1024 && w < 4)) continue;
      if (warps) *warps = w;
      return b;
    }
  return 0;
}

int launch_kuf_classes(const KufGemmArgs &k, int max_pairs, cudaStream_t st) {
  if (max_pairs <= 0) return 0;
  k_kuf_classes<<<dim3((max_pairs + 255) / 256, k.n_strucs), 256, 0, st>>>(k);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_kuf_places(const KufGemmArgs &k, int n_classes, cudaStream_t st) {
  k_kuf_places<<<k.n_pairs / 256 + 1, 256, 0, st>>>(k, n_classes);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_kuf_compact(int rows, int kc, const double *const *src, const int *sj,
                       const KufColumn *cols, double *dst, cudaStream_t st) {
  if (rows <= 0) return 0;
  k_kuf_compact<<<rows, 128, 0, st>>>(kc, src, sj, cols, dst);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_kuf_rows(const KufGemmArgs &k, cudaStream_t st) {
  if (k.n_places <= 0) return 0;
  int warps = 0;
  const size_t smem = kuf_rows_smem(k.a, k.kc, &warps);
  if (smem == 0) return -1;
  // sixteen pairs where blocks of 32 would not even out over the SMs: the bases then cost
  // twice as much per pair (a tenth of the kernel's time), the last round less
  const int bp = k.n_places >= 4 * 152 * kRowPairs ? kRowPairs : kRowPairs / 2;
  auto run = [&](auto kern) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
      return -1;
    kern<<<(k.n_places + bp - 1) / bp, 32 * warps, smem, st>>>(k, bp);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
  };
  switch (k.a.lmax) {
    case 0: return run(k_kuf_rows<0>);
    case 1: return run(k_kuf_rows<1>);
    case 2: return run(k_kuf_rows<2>);
    case 3: return run(k_kuf_rows<3>);
    case 4: return run(k_kuf_rows<4>);
    default: return run(k_kuf_rows<-1>);
  }
}

int launch_kuf_coef(const KufGemmArgs &k, cudaStream_t st) {
  if (k.n_blocks <= 0) return 0;
  k_kuf_coef<<<k.n_blocks, 32 * kKufAtoms, 0, st>>>(k);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int launch_kuf_gather(const KufGemmArgs &k, cudaStream_t st) {
  const int tiles = k.tiles[k.s1];
  if (k.n_blocks <= 0 || tiles <= 0) return 0;
  k_kuf_gather<<<dim3(k.n_blocks, tiles), 32 * kKufAtoms, 0, st>>>(k);
  if (cudaGetLastError() != cudaSuccess) return -1;
  // the unit's rows of Kuf are consecutive (species by species)
  const int row0 = k.sp[k.s0].row0;
  const int rows = k.sp[k.s1 - 1].row0 + k.sp[k.s1 - 1].n_sparse - row0;
  k_kuf_es<<<dim3((rows + 31) / 32, k.struc1 - k.struc0), 256, 0, st>>>(k, row0, rows);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace fpp
