// The mixed-precision (FP32) B3 coupling and its adjoint in real arithmetic.
//
// On real coefficients r[n, lm] (what the B2 stages accumulate) the bispectrum of
// b3.cpp:134-240 is
//   B[(n1 <= n2 <= n3), (l1, l2, l3)] = sum_{x, y, z} G(x, y, z) r[n1, l1 x]
//                                       r[n2, l2 y] r[n3, l3 z]
// with G the Wigner 3j symbols carried over to real harmonics.  G is real for even
// l1 + l2 + l3 and imaginary for odd ones, whose B (a real part) is therefore 0: of
// the 34 triangles of lmax = 3 the 11 odd ones are zero columns, which the mixed
// operand leaves out (1288 columns instead of 1904 for six radial channels), and
// the other 23 have 353 terms instead of 449 complex ones.
//
// The work is shared over n1: for a pair (n2 <= n3) the sums
//   S[t, x] = sum_{y, z} G r[n2, l2 y] r[n3, l3 z]
// are formed once and meet every r[n1], n1 <= n2 (about 18k multiply-adds per atom
// for six channels; a triple at a time took 160k, its adjoint 455k).  A thread
// takes one pair of one atom, several atoms to a block, an l1's triangles in parts; every
// index and coefficient is a compile-time constant.
//
// Measured at 32,000 atoms, six channels, lmax 3 (1,048,576 atoms in brackets): forward
// 465 us (15.0 ms) in one complex kernel before, 62 + 95 us now (single bond, coupling);
// adjoint 1240 us (40 ms) before, 279 us now, bound by latency (loads, barriers, dependent
// multiply-adds; 43 % of the issue slots taken) at the 12 warps per SM that its registers
// and shared memory admit (28 KB of rows per three atoms);
// contraction 365 us (11.8 ms) before on 1904 columns, 214 us now on 1288.
// (FP64 and lmax 0 and 4 use the complex form of b3.cuh.)
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>

#include "b2_device.cuh"
#include "b2_kernels.h"
#include "b3_real.h"
#include "common.cuh"
#include "tc_prims.cuh"

namespace fpp {

namespace {
constexpr int kMinL = 1, kMaxLM = 3;
constexpr int kMaxTerms = 192;  // terms of one l1

constexpr int iabs(int v) { return v < 0 ? -v : v; }
constexpr bool tri_even(int LM, int l1, int l2, int l3) {
  return l3 >= iabs(l1 - l2) && l3 <= l1 + l2 && l3 <= LM && (l1 + l2 + l3) % 2 == 0;
}
// the even triangles of block LM with first index l1, in loop order l2, l3
constexpr int n_tri_l1(int LM, int l1) {
  int n = 0;
  for (int l2 = 0; l2 <= LM; l2++)
    for (int l3 = 0; l3 <= LM; l3++) n += tri_even(LM, l1, l2, l3) ? 1 : 0;
  return n;
}
constexpr int tri_before(int LM, int l1) {
  int n = 0;
  for (int l = 0; l < l1; l++) n += n_tri_l1(LM, l);
  return n;
}
constexpr int n_even(int LM) { return tri_before(LM, LM + 1); }
// Where G can be non-zero for even l1 + l2 + l3: an even number of sines (negative
// orders) and one |order| the sum of the other two.
constexpr bool may_couple(int x, int y, int z) {
  const int s = (x < 0) + (y < 0) + (z < 0), a = iabs(x), b = iabs(y), c = iabs(z);
  return s % 2 == 0 && (a + b == c || a + c == b || b + c == a);
}

// ---- G(x, y, z) at compile time (an immediate operand of its multiply-add) ----
constexpr double ct_sqrt(double v) {
  double s = v > 1.0 ? v : 1.0;
  for (int k = 0; k < 64; k++) s = 0.5 * (s + v / s);
  return v == 0.0 ? 0.0 : s;
}
constexpr double ct_fact(int n) {
  double f = 1.0;
  for (int k = 2; k <= n; k++) f *= k;
  return f;
}
// Wigner 3j symbol by Racah's formula (lmax <= 3: the reference's tables hold the
// exact symbols there)
constexpr double ct_3j(int l1, int l2, int l3, int m1, int m2, int m3) {
  if (m1 + m2 + m3 != 0) return 0.0;
  int kmin = 0, kmax = l1 + l2 - l3;
  if (l2 - l3 - m1 > kmin) kmin = l2 - l3 - m1;
  if (l1 - l3 + m2 > kmin) kmin = l1 - l3 + m2;
  if (l1 - m1 < kmax) kmax = l1 - m1;
  if (l2 + m2 < kmax) kmax = l2 + m2;
  double s = 0.0;
  for (int k = kmin; k <= kmax; k++)
    s += (k % 2 ? -1.0 : 1.0) /
         (ct_fact(k) * ct_fact(l3 - l2 + k + m1) * ct_fact(l3 - l1 + k - m2) *
          ct_fact(l1 + l2 - l3 - k) * ct_fact(l1 - k - m1) * ct_fact(l2 - k + m2));
  const double pre = ct_fact(l1 + l2 - l3) * ct_fact(l1 - l2 + l3) * ct_fact(-l1 + l2 + l3) /
                     ct_fact(l1 + l2 + l3 + 1) * ct_fact(l1 + m1) * ct_fact(l1 - m1) *
                     ct_fact(l2 + m2) * ct_fact(l2 - m2) * ct_fact(l3 + m3) * ct_fact(l3 - m3);
  return ((l1 - l2 - m3) % 2 != 0 ? -1.0 : 1.0) * ct_sqrt(pre) * s;
}
struct Cplx {
  double re, im;
};
constexpr Cplx cmul(Cplx a, Cplx b) {
  return Cplx{a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re};
}
// U(m, x) of c[l, m] = sum_x U(m, x) r[l, x] for |m| = |x| (b3.cuh's map of real to
// complex coefficients)
constexpr Cplx real_to_complex(int m, int x) {
  const double h = ct_sqrt(0.5);
  if (m == 0) return Cplx{1.0, 0.0};
  if (m > 0) {
    const double sg = m % 2 ? -h : h;
    return x > 0 ? Cplx{sg, 0.0} : Cplx{0.0, sg};
  }
  return x > 0 ? Cplx{h, 0.0} : Cplx{0.0, -h};
}
// G = Re sum_m W(m1, m2, m3) U(m1, x) U(m2, y) U(m3, z)
constexpr double coupling(int l1, int l2, int l3, int x, int y, int z) {
  double s = 0.0;
  for (int i = 0; i < (x ? 2 : 1); i++)
    for (int j = 0; j < (y ? 2 : 1); j++)
      for (int k = 0; k < (z ? 2 : 1); k++) {
        const int m1 = i ? -x : x, m2 = j ? -y : y, m3 = k ? -z : z;
        if (m1 + m2 + m3 != 0) continue;
        const Cplx u =
            cmul(cmul(real_to_complex(m1, x), real_to_complex(m2, y)), real_to_complex(m3, z));
        s += ct_3j(l1, l2, l3, m1, m2, m3) * u.re;
      }
  return s;
}

// The triangles of one l1 are taken in parts of at most kPartSums S values, so that
// S, its adjoint and the rows they meet stay in registers.  (A product belongs to the
// triangles of one (l2, l3), so no part repeats another's.)
constexpr int kPartSums = 21;
constexpr int part_size(int l1) { return kPartSums / (2 * l1 + 1); }
constexpr int n_parts(int LM, int l1) {
  return (n_tri_l1(LM, l1) + part_size(l1) - 1) / part_size(l1);
}

// The terms of one part, grouped by their product r[n2, y] r[n3, z].
struct Terms {
  int n = 0;
  short t[kMaxTerms] = {}, x[kMaxTerms] = {};  // triangle (within the part), x + l1
  short b[kMaxTerms] = {}, c[kMaxTerms] = {};  // harmonic indices of n2 and n3
  float g[kMaxTerms] = {};                     // G(x, y, z)
  bool first[kMaxTerms] = {}, last[kMaxTerms] = {};
};
constexpr Terms make_terms(int LM, int l1, int part) {
  Terms T;
  int tri = -1;  // index of (l2, l3) among the triangles of l1
  for (int l2 = 0; l2 <= LM; l2++)
    for (int l3 = 0; l3 <= LM; l3++) {
      if (!tri_even(LM, l1, l2, l3)) continue;
      tri++;
      if (tri / part_size(l1) != part) continue;
      for (int y = -l2; y <= l2; y++)
        for (int z = -l3; z <= l3; z++) {
          bool any = false;
          for (int x = -l1; x <= l1; x++) {
            if (!may_couple(x, y, z)) continue;
            T.t[T.n] = (short)(tri - part * part_size(l1));
            T.x[T.n] = (short)(x + l1);
            T.b[T.n] = (short)(l2 * l2 + l2 + y);
            T.c[T.n] = (short)(l3 * l3 + l3 + z);
            T.g[T.n] = (float)coupling(l1, l2, l3, x, y, z);
            T.first[T.n] = !any;
            any = true;
            T.n++;
          }
          if (any) T.last[T.n - 1] = true;
        }
    }
  return T;
}
template <int LM, int L1, int P> struct PartTerms {
  static constexpr Terms T = make_terms(LM, L1, P);
  static constexpr int PT = part_size(L1);
  static constexpr int NT = n_tri_l1(LM, L1) - P * PT < PT ? n_tri_l1(LM, L1) - P * PT : PT;
  static constexpr int T0 = tri_before(LM, L1) + P * PT;  // columns before its triangles
  static constexpr int NX = 2 * L1 + 1;
  static constexpr int NS = NT * NX;                      // S values
};
template <int L1> constexpr int part_size_v = part_size(L1);
template <int LM, int L1> constexpr int n_tri_v = n_tri_l1(LM, L1);
}  // namespace

std::vector<int> b3_real_columns(int lmax, int n_tri) {
  std::vector<int> tri;  // the even triangles' columns among all of a triple
  int t = 0;
  for (int l1 = 0; l1 <= lmax; l1++)
    for (int l2 = 0; l2 <= lmax; l2++)
      for (int l3 = 0; l3 <= lmax; l3++) {
        if (iabs(l1 - l2) > l3 || l3 > l1 + l2) continue;
        if ((l1 + l2 + l3) % 2 == 0) tri.push_back(t);
        t++;
      }
  std::vector<int> cols;
  for (int r = 0; r < n_tri; r++)
    for (int e : tri) cols.push_back(r * t + e);
  while (cols.size() % 4) cols.push_back(-1);
  return cols;
}

// ---------------------------------------------------------------------------
// One term, and all terms of an l1.
// ---------------------------------------------------------------------------
template <int LM, int L1, int P, size_t I>
__device__ __forceinline__ void term_forward(const float (&r2)[(LM + 1) * (LM + 1)],
                                             const float (&r3)[(LM + 1) * (LM + 1)],
                                             float (&S)[PartTerms<LM, L1, P>::NS], float &prod) {
  using Q = PartTerms<LM, L1, P>;
  constexpr int b = Q::T.b[I], c = Q::T.c[I], k = Q::T.t[I] * Q::NX + Q::T.x[I];
  if constexpr (Q::T.first[I]) prod = r2[b] * r3[c];
  constexpr float g = Q::T.g[I];
  S[k] = fmaf(g, prod, S[k]);
}
template <int LM, int L1, int P, size_t... I>
__device__ __forceinline__ void sums_forward(const float (&r2)[(LM + 1) * (LM + 1)],
                                             const float (&r3)[(LM + 1) * (LM + 1)],
                                             float (&S)[PartTerms<LM, L1, P>::NS],
                                             std::index_sequence<I...>) {
  float prod = 0.0f;
#pragma unroll
  for (int k = 0; k < PartTerms<LM, L1, P>::NS; k++) S[k] = 0.0f;
  (term_forward<LM, L1, P, I>(r2, r3, S, prod), ...);
}

template <int LM, int L1, int P, size_t I>
__device__ __forceinline__ void term_adjoint(const float (&r2)[(LM + 1) * (LM + 1)],
                                             const float (&r3)[(LM + 1) * (LM + 1)],
                                             const float (&dS)[PartTerms<LM, L1, P>::NS],
                                             float (&u2)[(LM + 1) * (LM + 1)],
                                             float (&u3)[(LM + 1) * (LM + 1)], float &d) {
  using Q = PartTerms<LM, L1, P>;
  constexpr int b = Q::T.b[I], c = Q::T.c[I], k = Q::T.t[I] * Q::NX + Q::T.x[I];
  constexpr float g = Q::T.g[I];
  if constexpr (Q::T.first[I])
    d = g * dS[k];
  else
    d = fmaf(g, dS[k], d);
  if constexpr (Q::T.last[I]) {
    u2[b] = fmaf(d, r3[c], u2[b]);
    u3[c] = fmaf(d, r2[b], u3[c]);
  }
}
template <int LM, int L1, int P, size_t... I>
__device__ __forceinline__ void sums_adjoint(const float (&r2)[(LM + 1) * (LM + 1)],
                                             const float (&r3)[(LM + 1) * (LM + 1)],
                                             const float (&dS)[PartTerms<LM, L1, P>::NS],
                                             float (&u2)[(LM + 1) * (LM + 1)],
                                             float (&u3)[(LM + 1) * (LM + 1)],
                                             std::index_sequence<I...>) {
  float d = 0.0f;
  (term_adjoint<LM, L1, P, I>(r2, r3, dS, u2, u3, d), ...);
}

// f(l1, part) over all parts of all l1 (compile-time constants)
template <int LM, int L1 = 0, int P = 0, typename F>
__device__ __forceinline__ void for_each_part(F &&f) {
  if constexpr (L1 <= LM) {
    f(std::integral_constant<int, L1>{}, std::integral_constant<int, P>{});
    if constexpr ((P + 1) * part_size_v<L1> < n_tri_v<LM, L1>)
      for_each_part<LM, L1, P + 1>(f);
    else
      for_each_part<LM, L1 + 1, 0>(f);
  }
}

// Rows r[n, 0..H) of one atom at stride HS, in 16-byte loads where H allows.
template <int H>
__device__ __forceinline__ void load_row(const float *__restrict__ src, float (&r)[H]) {
  if constexpr (H % 4 == 0) {
#pragma unroll
    for (int k = 0; k < H / 4; k++) {
      const float4 v = reinterpret_cast<const float4 *>(src)[k];
      r[4 * k] = v.x, r[4 * k + 1] = v.y, r[4 * k + 2] = v.z, r[4 * k + 3] = v.w;
    }
  } else {
#pragma unroll
    for (int k = 0; k < H; k++) r[k] = src[k];
  }
}

// pair q of the list (n2, n3 >= n2), n2 outer; and the triple (n1, n2, n3)'s index
// in the list n1 <= n2 <= n3, n1 outermost (b3.cpp:176-178)
__device__ __forceinline__ int2 pair_of(int q, int nr) {
  int n2 = 0;
  while (q >= nr - n2) {
    q -= nr - n2;
    n2++;
  }
  return make_int2(n2, n2 + q);
}
__device__ __forceinline__ int triple_index(int n1, int n2, int n3, int nr) {
  const int a = nr - n1;  // channels from n1 up
  const int before = (nr * (nr + 1) * (nr + 2) - a * (a + 1) * (a + 2)) / 6;
  const int i = n2 - n1;
  return before + i * a - i * (i - 1) / 2 + (n3 - n2);
}

// Sizes of block LM: c rows (padded in shared memory to 16-byte rows on different
// banks), columns per triple, floats of a pair's two u rows and of a
// triple's (odd: at 16 floats the triples of a warp met in two banks, and the adjoint of
// 32,000 atoms took 400 us).
template <int LM> struct RowPad {
  static constexpr int H = (LM + 1) * (LM + 1);
  static constexpr int HS = (H + 3) / 4 * 4 + 4;
  static constexpr int NE = n_even(LM);
  static constexpr int US = 2 * H + 1, TS = H | 1;
};

// Floats of the adjoint's w region (xn: the rows that may take its place).
static __host__ __device__ inline size_t w_floats(size_t wn, size_t xn, bool one_round) {
  return one_round && xn > wn ? (xn + 3) / 4 * 4 : wn;
}

// Index of the triple (n1, n2, n3): tab[n1 nr + n2] + n3.
__device__ __forceinline__ void triple_table(int nr, int *tab) {
  for (int k = threadIdx.x; k < nr * nr; k += blockDim.x) {
    const int n1 = k / nr, n2 = k - n1 * nr;
    tab[k] = n2 >= n1 ? triple_index(n1, n2, n2, nr) - n2 : 0;
  }
}

// A block's coefficient rows: [atom][n][HS], atoms at stride nr HS + 4 (a warp reads
// the same row of several atoms).
template <int LM> __host__ __device__ constexpr int atom_stride(int nr) {
  return nr * RowPad<LM>::HS + 4;
}
template <int LM>
__device__ __forceinline__ void stage_rows(const float *__restrict__ c_in, size_t a0, int na,
                                           int nr, float *c_s) {
  constexpr int H = RowPad<LM>::H, HS = RowPad<LM>::HS;
  for (int k = threadIdx.x; k < na * nr * H; k += blockDim.x) {
    const int row = k / H, lm = k - row * H;
    const int at = row / nr;
    c_s[at * atom_stride<LM>(nr) + (row - at * nr) * HS + lm] = c_in[a0 * nr * H + k];
  }
}

// Bytes of an fp16 operand row of nd entries as it is copied (whole 16-byte units;
// rows are padded further in global memory).
__host__ __device__ inline uint32_t operand_bytes(int nd) {
  return ((uint32_t)nd * 2u + 15u) & ~15u;
}

// Items of a block are (pair, atom), atoms fastest and pairs in list order: the
// lanes of a warp then have about the same n2, which is their count of n1 less one
// (a warp runs to its largest: 13 rounds per four warps at six channels, 24 with
// the pairs of an atom side by side).

// ---------------------------------------------------------------------------
// Forward: p of `apb` atoms per block, |p|, and the centred split operand rows.
// ---------------------------------------------------------------------------
template <int LM>
__global__ void __launch_bounds__(128, 5)
k_b3_couple(int noa, int apb, int nr, int nd, const int *__restrict__ species,
            const int *__restrict__ row_of_atom, const float *__restrict__ c_in,
            double *__restrict__ norm_out, __half *__restrict__ phat_hi,
            __half *__restrict__ phat_lo, int ldp, const float *__restrict__ pbar) {
  constexpr int H = RowPad<LM>::H, HS = RowPad<LM>::HS, NE = RowPad<LM>::NE;
  extern __shared__ __align__(16) float smem[];
  const int cs = atom_stride<LM>(nr);
  float *c_s = smem;                               // [apb][cs]
  float *p_s = smem + (size_t)apb * cs;            // [apb][nd]
  int *tri_s = reinterpret_cast<int *>(p_s + (size_t)apb * nd);  // [nr][nr]
  const int a0 = blockIdx.x * apb, na = min(apb, noa - a0);
  stage_rows<LM>(c_in, a0, na, nr, c_s);
  triple_table(nr, tri_s);
  const int used = nr * (nr + 1) * (nr + 2) / 6 * NE;  // columns past it pad rows to 16 bytes
  for (int k = threadIdx.x; k < na * (nd - used); k += blockDim.x) {
    const int at = k / (nd - used);
    p_s[(size_t)at * nd + used + (k - at * (nd - used))] = 0.0f;
  }
  __syncthreads();
  const int np = nr * (nr + 1) / 2;
  for (int it = threadIdx.x; it < na * np; it += blockDim.x) {
    const int q = it / na, at = it - q * na;
    const int2 n23 = pair_of(q, nr);
    const float *ca = c_s + at * cs;
    float *pa = p_s + (size_t)at * nd;
    float r2[H], r3[H];
    load_row<H>(ca + n23.x * HS, r2);
    load_row<H>(ca + n23.y * HS, r3);
    for_each_part<LM>([&](auto lc, auto pc) {
      constexpr int L1 = decltype(lc)::value, P = decltype(pc)::value;
      using Q = PartTerms<LM, L1, P>;
      float S[Q::NS];
      sums_forward<LM, L1, P>(r2, r3, S, std::make_index_sequence<Q::T.n>{});
      for (int n1 = 0; n1 <= n23.x; n1++) {
        float r1[Q::NX];
#pragma unroll
        for (int x = 0; x < Q::NX; x++) r1[x] = ca[n1 * HS + L1 * L1 + x];
        float *dst = pa + (tri_s[n1 * nr + n23.x] + n23.y) * NE + Q::T0;
#pragma unroll
        for (int t = 0; t < Q::NT; t++) {
          float v = r1[0] * S[t * Q::NX];
#pragma unroll
          for (int x = 1; x < Q::NX; x++) v = fmaf(r1[x], S[t * Q::NX + x], v);
          dst[t] = v;
        }
      }
    });
  }
  __syncthreads();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int at = warp; at < na; at += (int)(blockDim.x >> 5)) {
    const int atom = a0 + at, si = species[atom];
    const size_t row = row_of_atom[atom];
    const float *pa = p_s + (size_t)at * nd;
    float invf;
    const float2 nrm = norm_ff(sum_squares(pa, nd, lane), invf);
    if (lane == 0) reinterpret_cast<float2 *>(norm_out)[atom] = nrm;
    write_split_row(pa, nd, invf, pbar + (size_t)si * nd, phat_hi + row * ldp,
                    phat_lo + row * ldp, lane);
  }
}

// ---------------------------------------------------------------------------
// Adjoint: w = dE/dp and E from the contraction, then u = dE/dr.
//   u[n1, l1 x] += sum_t w S[t, x],   dS[t, x] = sum_n1 w r[n1, l1 x],   and dS back
// through the products to n2 and n3.  A triple's row for n1 and a pair's rows for
// n2 and n3 go to shared memory and are summed per (n, lm) in list order, so the
// result does not depend on timing.
// ---------------------------------------------------------------------------
template <int LM>
__global__ void __launch_bounds__(128, 3)
k_b3_adjoint(int noa, int apb, int nr, int nd, AdjArgs g, const int *__restrict__ species,
             const int *__restrict__ row_of_atom, const float *__restrict__ c_in,
             const double *__restrict__ norm_in, double *__restrict__ atom_e,
             float *__restrict__ u_out) {
  constexpr int H = RowPad<LM>::H, HS = RowPad<LM>::HS, NE = RowPad<LM>::NE;
  constexpr int US = RowPad<LM>::US, TS = RowPad<LM>::TS;
  extern __shared__ __align__(16) float smem[];
  const int np = nr * (nr + 1) / 2, nt = nr * (nr + 1) * (nr + 2) / 6;
  const int cs = atom_stride<LM>(nr);
  // the rows for n2 and n3 take the place of w where every pair has a thread
  const bool one_round = np <= (int)blockDim.x;
  const size_t wn = (size_t)apb * nd, xn = (size_t)blockDim.x * US;
  const uint32_t bar = smem_u32(smem), hb = operand_bytes(nd);
  float *w_s = smem + 4;                            // [apb][nd], first the V rows
  float *c_s = w_s + w_floats(wn, xn, one_round);   // [apb][cs]
  int *tri_s = reinterpret_cast<int *>(c_s + (size_t)apb * cs);            // [nr][nr]
  float *t_s = reinterpret_cast<float *>(tri_s + (nr * nr + 3) / 4 * 4);   // [apb][nt][TS]
  // the split operand rows, before the rows for n1 take their place
  unsigned char *h_s = reinterpret_cast<unsigned char *>(t_s);
  // [threads][US], and with several rounds their sums so far [apb][nr][H]
  float *x_s = one_round ? w_s : t_s + (size_t)apb * nt * TS;
  float *u_s = x_s + xn;
  const int a0 = blockIdx.x * apb, na = min(apb, noa - a0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // every atom's V and split operand rows (10 KB at six channels) come by bulk
  // asynchronous copies on one mbarrier, all in flight at once
  if (threadIdx.x == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(bar, (uint32_t)na * ((uint32_t)nd * 4u + 2u * hb));
    for (int at = 0; at < na; at++) {
      const size_t row = row_of_atom[a0 + at];
      bulk_load(smem_u32(w_s + (size_t)at * nd), g.V32 + row * g.ldv, (uint32_t)nd * 4u, bar);
      bulk_load(smem_u32(h_s + (size_t)(2 * at) * hb), g.phat_hi + row * g.ldp, hb, bar);
      bulk_load(smem_u32(h_s + (size_t)(2 * at + 1) * hb), g.phat_lo + row * g.ldp, hb, bar);
    }
  }
  stage_rows<LM>(c_in, a0, na, nr, c_s);
  triple_table(nr, tri_s);
  __syncthreads();
  if (!__syncthreads_and(mbar_wait(bar, 0))) {
    if (threadIdx.x == 0) set_status(g.status, FPP_ERR_TIMEOUT, 231, a0);
    mbar_wait(bar, 0);
    return;
  }
  for (int at = warp; at < na; at += (int)(blockDim.x >> 5)) {
    const int atom = a0 + at;
    float *wa = w_s + (size_t)at * nd;
    const double e = w_mixed2(
        g, species[atom], nd, reinterpret_cast<const float2 *>(norm_in)[atom],
        reinterpret_cast<const float4 *>(wa),
        reinterpret_cast<const uint2 *>(h_s + (size_t)(2 * at) * hb),
        reinterpret_cast<const uint2 *>(h_s + (size_t)(2 * at + 1) * hb),
        [&](int q, float4 v) { reinterpret_cast<float4 *>(wa)[q] = v; }, lane);
    if (lane == 0) atom_e[atom] = e;
  }
  __syncthreads();
  for (int it0 = 0; it0 < na * np; it0 += blockDim.x) {
    const int it = it0 + threadIdx.x;
    const bool live = it < na * np;
    float u2[H], u3[H];
#pragma unroll
    for (int k = 0; k < H; k++) u2[k] = u3[k] = 0.0f;
    if (live) {
      const int q = it / na, at = it - q * na;
      const int2 n23 = pair_of(q, nr);
      const float *ca = c_s + at * cs;
      const float *wa = w_s + (size_t)at * nd;
      float *ta = t_s + (size_t)at * nt * TS;
      const int *tab = tri_s + n23.x;
      for_each_part<LM>([&](auto lc, auto pc) {
        constexpr int L1 = decltype(lc)::value, P = decltype(pc)::value;
        using Q = PartTerms<LM, L1, P>;
        float dS[Q::NS];
#pragma unroll
        for (int k = 0; k < Q::NS; k++) dS[k] = 0.0f;
        {
          float S[Q::NS];
          {
            // (r2 and r3 are read again below: both do not fit beside S and dS)
            float r2[H], r3[H];
            load_row<H>(ca + n23.x * HS, r2);
            load_row<H>(ca + n23.y * HS, r3);
            sums_forward<LM, L1, P>(r2, r3, S, std::make_index_sequence<Q::T.n>{});
          }
          for (int n1 = 0; n1 <= n23.x; n1++) {
            const int tr = tab[n1 * nr] + n23.y;
            float r1[Q::NX], w[Q::NT], u1[Q::NX];
#pragma unroll
            for (int x = 0; x < Q::NX; x++) r1[x] = ca[n1 * HS + L1 * L1 + x];
#pragma unroll
            for (int t = 0; t < Q::NT; t++) w[t] = wa[tr * NE + Q::T0 + t];
#pragma unroll
            for (int x = 0; x < Q::NX; x++) u1[x] = 0.0f;
#pragma unroll
            for (int t = 0; t < Q::NT; t++)
#pragma unroll
              for (int x = 0; x < Q::NX; x++) {
                dS[t * Q::NX + x] = fmaf(w[t], r1[x], dS[t * Q::NX + x]);
                u1[x] = fmaf(w[t], S[t * Q::NX + x], u1[x]);
              }
#pragma unroll
            for (int x = 0; x < Q::NX; x++) {
              float *dst = ta + tr * TS + L1 * L1 + x;
              *dst = P == 0 ? u1[x] : *dst + u1[x];
            }
          }
        }
        float r2[H], r3[H];
        load_row<H>(ca + n23.x * HS, r2);
        load_row<H>(ca + n23.y * HS, r3);
        sums_adjoint<LM, L1, P>(r2, r3, dS, u2, u3, std::make_index_sequence<Q::T.n>{});
      });
    }
    if (one_round) __syncthreads();  // every w has been read
    if (live) {
#pragma unroll
      for (int k = 0; k < H; k++) {
        x_s[threadIdx.x * US + k] = u2[k];
        x_s[threadIdx.x * US + H + k] = u3[k];
      }
    }
    __syncthreads();
    // the rows of this round's pairs for n2 and n3 (items it0 .. it0 + blockDim.x),
    // and after the last round the triples' rows for n1
    const bool last = it0 + (int)blockDim.x >= na * np;
    for (int o = threadIdx.x; o < na * nr * H; o += blockDim.x) {
      const int oa = o / (nr * H), rem = o - oa * nr * H;
      const int n = rem / H, lm = rem - n * H;
      float s = it0 == 0 ? 0.0f : u_s[o];
      for (int m = 0; m <= n; m++) {  // pairs (m, n): n3 = n
        const int i = (m * nr - m * (m - 1) / 2 + (n - m)) * na + oa - it0;
        if (i >= 0 && i < (int)blockDim.x) s += x_s[i * US + H + lm];
      }
      for (int m = n; m < nr; m++) {  // pairs (n, m): n2 = n
        const int i = (n * nr - n * (n - 1) / 2 + (m - n)) * na + oa - it0;
        if (i >= 0 && i < (int)blockDim.x) s += x_s[i * US + lm];
      }
      if (!last) {
        u_s[o] = s;
        continue;
      }
      // (the triples with n1 = n are consecutive)
      const int m = nr - n, count = m * (m + 1) / 2;
      const float *t = t_s + ((size_t)oa * nt + (nt - m * (m + 1) * (m + 2) / 6)) * TS + lm;
      for (int i = 0; i < count; i++) s += t[i * TS];
      u_out[(size_t)a0 * nr * H + o] = s;
    }
    if (!last) __syncthreads();
  }
}

// Threads per block, and atoms per block, whose pairs fill them (64 threads pack the
// SM's shared memory better, but mix the pairs' counts of n1 more: 508 against 400
// us for the adjoint of 32,000 atoms).
struct B3Block {
  int threads, atoms;
};
static B3Block block_of(int nr) { return B3Block{128, std::max(1, 128 / (nr * (nr + 1) / 2))}; }

template <int LM> static size_t couple_smem(int nr, int nd) {
  return sizeof(float) * ((size_t)block_of(nr).atoms * (atom_stride<LM>(nr) + (size_t)nd) +
                          (size_t)nr * nr);
}
template <int LM> static size_t adjoint_smem(int nr, int nd) {
  constexpr int H = RowPad<LM>::H, US = RowPad<LM>::US, TS = RowPad<LM>::TS;
  const B3Block b = block_of(nr);
  const size_t nt = (size_t)nr * (nr + 1) * (nr + 2) / 6, apb = b.atoms;
  const bool one_round = nr * (nr + 1) / 2 <= b.threads;
  const size_t wn = apb * nd, xn = (size_t)b.threads * US;
  // the split operand rows, then in their place the rows for n1 (and for n2 and n3)
  const size_t late = std::max(
      2 * apb * operand_bytes(nd),
      sizeof(float) * (apb * nt * TS + (one_round ? 0 : xn + apb * nr * H)));
  return 16 +
         sizeof(float) * (w_floats(wn, xn, one_round) + apb * atom_stride<LM>(nr) +
                          (size_t)(nr * nr + 3) / 4 * 4) +
         late;
}

template <typename F> static int with_lm(int lmax, F &&f) {
  switch (lmax) {
    case 1: return f(std::integral_constant<int, 1>{});
    case 2: return f(std::integral_constant<int, 2>{});
    case 3: return f(std::integral_constant<int, 3>{});
    default: return -1;
  }
}

bool b3_real_fits(int lmax, int nr) {
  if (lmax < kMinL || lmax > kMaxLM) return false;
  const int nd = (nr * (nr + 1) * (nr + 2) / 6 * n_even(lmax) + 3) / 4 * 4;
  size_t s = ~(size_t)0;
  with_lm(lmax, [&](auto lc) {
    constexpr int LM = decltype(lc)::value;
    s = std::max(couple_smem<LM>(nr, nd), adjoint_smem<LM>(nr, nd));
    return 0;
  });
  return s <= 227 * 1024;
}

int launch_b3_couple(const B2Args &a, int nd, const int *species, const int *row_of_atom,
                     const float *c_in, double *norm_out, __half *phat_hi, __half *phat_lo,
                     int ldp, const float *pbar, cudaStream_t stream) {
  if (a.noa == 0) return 0;
  const int nr = a.n_species * a.N;
  const B3Block b = block_of(nr);
  return with_lm(a.lmax, [&](auto lc) {
    constexpr int LM = decltype(lc)::value;
    const size_t smem = couple_smem<LM>(nr, nd);
    if (cudaFuncSetAttribute(k_b3_couple<LM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess)
      return -1;
    k_b3_couple<LM><<<ceil_div(a.noa, b.atoms), b.threads, smem, stream>>>(
        a.noa, b.atoms, nr, nd, species, row_of_atom, c_in, norm_out, phat_hi, phat_lo, ldp, pbar);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
  });
}

int launch_b3_adjoint(const B2Args &a, int nd, const AdjArgs &g, const int *species,
                      const int *row_of_atom, const float *c_in, const double *norm_in,
                      double *atom_e, float *u_out, cudaStream_t stream) {
  if (a.noa == 0) return 0;
  const int nr = a.n_species * a.N;
  const B3Block b = block_of(nr);
  return with_lm(a.lmax, [&](auto lc) {
    constexpr int LM = decltype(lc)::value;
    const size_t smem = adjoint_smem<LM>(nr, nd);
    if (cudaFuncSetAttribute(k_b3_adjoint<LM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess)
      return -1;
    k_b3_adjoint<LM><<<ceil_div(a.noa, b.atoms), b.threads, smem, stream>>>(
        a.noa, b.atoms, nr, nd, g, species, row_of_atom, c_in, norm_in, atom_e, u_out);
    return cudaGetLastError() == cudaSuccess ? 0 : -1;
  });
}

}  // namespace fpp
