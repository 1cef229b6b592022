// B3 bispectrum: coupling tables and the per-atom device stages.
//
// src/flare_pp/descriptors/b3.cpp:134-240 computes, per atom,
//   B3[(n1 <= n2 <= n3), (l1, l2, l3)] =
//       Re sum_{m1+m2+m3=0} W(l1 l2 l3; m1 m2 m3) c[n1,l1m1] c[n2,l2m2] c[n3,l3m3]
// on complex single-bond coefficients c (complex harmonics with the
// Condon-Shortley phase, src/flare_pp/y_grad.cpp:24), with the triangles
// (l1, l2, l3) in loop order l1, l2, l3 and |l1-l2| <= l3 <= l1+l2.
//
// The complex coefficients are a fixed linear map of the real ones that the
// B2 stages already accumulate: with R = c[l, m], S = c[l, -m] (real, m > 0),
//   c[l, +m] = (-1)^m (R + i S) / sqrt 2,  c[l, -m] = (R - i S) / sqrt 2.
// So the forward reuses the real accumulation, and the adjoint maps the
// holomorphic derivative u = dE/dc back to dE/dc_real, after which the B2
// pair-force kernel applies unchanged.
//
// W is the Wigner 3j symbol from Racah's formula.  The reference's table for
// lmax = 4 (descriptors/wigner3j.cpp:590-1986) holds 0 at the 57 symbols whose
// exact value is a non-integer rational (+-1/3, +-1/6): its generated source
// writes them as C++ integer divisions.  The tables here reproduce that.
//
// Included by exactly one translation unit (the constant bank is static).
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <type_traits>
#include <vector>

#include "common.cuh"

namespace fpp {

constexpr int kB3MaxL = 4;
constexpr int kB3MaxTerms = 2112;  // sum over lmax 0..4 of the m-terms (2052)
constexpr int kB3MaxLs = 130;      // sum over lmax 0..4 of (n_ls + 1)

struct B3Tables {
  int ls_off[kB3MaxL + 2];    // start of each lmax's triangle offsets in beg[]
  int beg[kB3MaxLs];          // per triangle: first term (absolute index)
  unsigned idx[kB3MaxTerms];  // i1 | i2 << 8 | i3 << 16 (harmonic index l*l+l+m)
  double w[kB3MaxTerms];
  float wf[kB3MaxTerms];      // w rounded to FP32 (the FP32 kernels convert nothing)
};

static __constant__ B3Tables c_b3;
// The coupling coefficient of term e in the kernel's precision.
template <typename T> __device__ __forceinline__ T b3_w(int e);
template <> __device__ __forceinline__ float b3_w<float>(int e) { return c_b3.wf[e]; }
template <> __device__ __forceinline__ double b3_w<double>(int e) { return c_b3.w[e]; }

inline double b3_factorial(int n) {
  double f = 1.0;
  for (int k = 2; k <= n; k++) f *= k;
  return f;
}

// Wigner 3j symbol by Racah's formula (all factorials <= 13! are exact).
inline double b3_wigner3j(int l1, int l2, int l3, int m1, int m2, int m3) {
  if (m1 + m2 + m3 != 0 || l3 < std::abs(l1 - l2) || l3 > l1 + l2) return 0.0;
  if (std::abs(m1) > l1 || std::abs(m2) > l2 || std::abs(m3) > l3) return 0.0;
  const double tri = b3_factorial(l1 + l2 - l3) * b3_factorial(l1 - l2 + l3) *
                     b3_factorial(-l1 + l2 + l3) / b3_factorial(l1 + l2 + l3 + 1);
  const double pre = tri * b3_factorial(l1 + m1) * b3_factorial(l1 - m1) *
                     b3_factorial(l2 + m2) * b3_factorial(l2 - m2) *
                     b3_factorial(l3 + m3) * b3_factorial(l3 - m3);
  int kmin = 0;
  if (l2 - l3 - m1 > kmin) kmin = l2 - l3 - m1;
  if (l1 - l3 + m2 > kmin) kmin = l1 - l3 + m2;
  int kmax = l1 + l2 - l3;
  if (l1 - m1 < kmax) kmax = l1 - m1;
  if (l2 + m2 < kmax) kmax = l2 + m2;
  double s = 0.0;
  for (int k = kmin; k <= kmax; k++) {
    const double d = b3_factorial(k) * b3_factorial(l3 - l2 + k + m1) *
                     b3_factorial(l3 - l1 + k - m2) * b3_factorial(l1 + l2 - l3 - k) *
                     b3_factorial(l1 - k - m1) * b3_factorial(l2 - k + m2);
    s += ((k & 1) ? -1.0 : 1.0) / d;
  }
  const double sign = ((l1 - l2 - m3) % 2 != 0) ? -1.0 : 1.0;
  return sign * std::sqrt(pre) * s;
}

// The coefficient compute_B3 applies for this lmax (see the header comment).
inline double b3_reference_coeff(int l1, int l2, int l3, int m1, int m2, int m3,
                                 int lmax) {
  const double w = b3_wigner3j(l1, l2, l3, m1, m2, m3);
  if (lmax == 4 && w != 0.0 && std::fabs(w) < 1.0) {
    const double inv2 = 1.0 / (w * w);
    const double k = std::round(std::sqrt(inv2));
    if (k > 1.0 && std::fabs(inv2 - k * k) < 1e-9 * inv2) return 0.0;
  }
  return w;
}

inline int b3_n_ls(int lmax) {
  int n = 0;
  for (int l1 = 0; l1 <= lmax; l1++)
    for (int l2 = 0; l2 <= lmax; l2++)
      for (int l3 = 0; l3 <= lmax; l3++)
        if (std::abs(l1 - l2) <= l3 && l3 <= l1 + l2) n++;
  return n;
}

inline int upload_b3_tables(cudaStream_t stream) {
  static B3Tables t;  // 25 KB: not on the stack
  int nt = 0, nb = 0;
  for (int lmax = 0; lmax <= kB3MaxL; lmax++) {
    t.ls_off[lmax] = nb;
    for (int l1 = 0; l1 <= lmax; l1++)
      for (int l2 = 0; l2 <= lmax; l2++)
        for (int l3 = 0; l3 <= lmax; l3++) {
          if (std::abs(l1 - l2) > l3 || l3 > l1 + l2) continue;
          t.beg[nb++] = nt;
          for (int m1 = -l1; m1 <= l1; m1++)
            for (int m2 = -l2; m2 <= l2; m2++) {
              const int m3 = -m1 - m2;
              if (std::abs(m3) > l3) continue;
              // every (m1, m2) with |m3| <= l3 in loop order, zeros included,
              // so that the term offsets within a triangle are fixed
              const double w = b3_reference_coeff(l1, l2, l3, m1, m2, m3, lmax);
              if (nt >= kB3MaxTerms) return -1;
              t.idx[nt] = (unsigned)(l1 * l1 + l1 + m1) |
                          ((unsigned)(l2 * l2 + l2 + m2) << 8) |
                          ((unsigned)(l3 * l3 + l3 + m3) << 16);
              t.w[nt] = w;
              t.wf[nt] = (float)w;
              nt++;
            }
        }
    t.beg[nb++] = nt;  // end of the last triangle of this lmax
  }
  t.ls_off[kB3MaxL + 1] = nb;
  cudaError_t e =
      cudaMemcpyToSymbolAsync(c_b3, &t, sizeof(t), 0, cudaMemcpyHostToDevice, stream);
  return e == cudaSuccess ? 0 : -1;
}

// Real single-bond block c (nr x H, row stride ldc, default H) -> complex (zr, zi) with
// row stride H + 1 (padded so that lanes on different radial rows hit
// different banks).  Lane-strided; the caller synchronizes the warp.
template <typename T>
__device__ __forceinline__ void b3_to_complex(const T *__restrict__ c, int nr, int H,
                                              T *__restrict__ zr, T *__restrict__ zi,
                                              int lane, int ldc = -1) {
  const int HC = ldc < 0 ? H : ldc;  // row stride of c
  const T is2 = T(0.70710678118654752440);
  for (int k = lane; k < nr * H; k += 32) {
    const int n = k / H, lm = k - n * H;
    int l = 0;
    while ((l + 1) * (l + 1) <= lm) l++;
    const int m = lm - l * l - l;
    const int am = m < 0 ? -m : m;
    const T R = c[n * HC + l * l + l + am];
    const T S = c[n * HC + l * l + l - am];
    T re, im;
    if (m == 0) {
      re = R;
      im = T(0);
    } else if (m > 0) {
      const T sg = (am & 1) ? T(-1) : T(1);
      re = sg * R * is2;
      im = sg * S * is2;
    } else {
      re = R * is2;
      im = -S * is2;
    }
    zr[n * (H + 1) + lm] = re;
    zi[n * (H + 1) + lm] = im;
  }
}

// (re, im) pairs for 8-byte (FP32) / 16-byte (FP64) shared-memory accesses.
template <typename T> struct V2T;
template <> struct V2T<float> { using type = float2; };
template <> struct V2T<double> { using type = double2; };
template <typename T> using V2 = typename V2T<T>::type;

// b3_to_complex with the complex block interleaved: z[n * (H + 1) + lm] = (re, im).
template <typename T>
__device__ __forceinline__ void b3_to_complex2(const T *__restrict__ c, int nr, int H,
                                               V2<T> *__restrict__ z, int lane, int ldc = -1) {
  const int HC = ldc < 0 ? H : ldc;
  const T is2 = T(0.70710678118654752440);
  for (int k = lane; k < nr * H; k += 32) {
    const int n = k / H, lm = k - n * H;
    int l = 0;
    while ((l + 1) * (l + 1) <= lm) l++;
    const int m = lm - l * l - l;
    const int am = m < 0 ? -m : m;
    const T R = c[n * HC + l * l + l + am];
    const T S = c[n * HC + l * l + l - am];
    V2<T> v;
    if (m == 0) {
      v.x = R;
      v.y = T(0);
    } else if (m > 0) {
      const T sg = (am & 1) ? T(-1) : T(1);
      v.x = sg * R * is2;
      v.y = sg * S * is2;
    } else {
      v.x = R * is2;
      v.y = -S * is2;
    }
    z[n * (H + 1) + lm] = v;
  }
}

// p[r * n_ls + t] for every radial triple r (table tri: n1 | n2<<8 | n3<<16)
// and triangle t, from the interleaved complex block; lanes take triples, all
// lanes walk the same term list (the coefficients and harmonic indices are
// uniform loads from constant memory).
template <typename T>
__device__ __forceinline__ void b3_contract(int lmax, int n_ls, int n_tri, int H,
                                             const int *__restrict__ tri,
                                             const V2<T> *__restrict__ z, T *__restrict__ p,
                                             int lane) {
  const int H1 = H + 1;
  const int *beg = c_b3.beg + c_b3.ls_off[lmax];
  for (int t = 0; t < n_ls; t++) {
    const int e0 = beg[t], e1 = beg[t + 1];
    for (int r = lane; r < n_tri; r += 32) {
      const int tr = tri[r];
      const V2<T> *z1 = z + (tr & 0xff) * H1, *z2 = z + ((tr >> 8) & 0xff) * H1;
      const V2<T> *z3 = z + (tr >> 16) * H1;
      T acc = T(0);
      for (int e = e0; e < e1; e++) {
        const unsigned ix = c_b3.idx[e];
        const V2<T> a = z1[ix & 0xff], b = z2[(ix >> 8) & 0xff], c = z3[ix >> 16];
        const T xr = a.x * b.x - a.y * b.y, xi = a.x * b.y + a.y * b.x;
        acc += b3_w<T>(e) * (xr * c.x - xi * c.y);
      }
      p[r * n_ls + t] = acc;
    }
  }
}

// Adjoint of b3_contract: for dE/dp = w, the holomorphic derivative
// u = dE/dc summed into u2[n * H + lm] = (re, im).  Lanes take radial triples
// in rounds of 32; within a round lane r only updates the rows n1(r), n2(r),
// n3(r) of its own triple, so it accumulates into three private rows in
// shared memory, priv[(pos * H + lm) * 32 + lane] (conflict-free banks, no
// atomics).  After each round the private rows are summed into u2 by output
// entry, over lanes in a fixed rotated order.  The caller zeroes u2 and
// synchronizes the warp before and after.
// u2[n, lm] += the private rows of one round, over lanes j in a fixed rotated
// order (lanes read different banks) and positions with n_pos(j) == n.  Each
// lane reads its own triple once; the others come by shuffle, in loops whose
// trip counts are the same for every lane.
template <typename T>
__device__ __forceinline__ void b3_reduce_private(int r0, int n_tri, int H, int nr,
                                                  const int *__restrict__ tri,
                                                  const V2<T> *__restrict__ priv,
                                                  V2<T> *__restrict__ u2, int lane) {
  const int own = r0 + lane < n_tri ? tri[r0 + lane] : -1;
  const int total = nr * H;
  for (int k0 = 0; k0 < total; k0 += 32) {
    const int k = k0 + lane;
    const bool act = k < total;
    const int n = act ? k / H : -1;
    const int lm = act ? k - n * H : 0;
    V2<T> acc{T(0), T(0)};
    for (int j0 = 0; j0 < 32; j0++) {
      const int j = (j0 + lane) & 31;
      const int tj = __shfl_sync(0xffffffffu, own, j);
      if (tj < 0) continue;  // no triple in this round's slot j
      const V2<T> *col = priv + (size_t)lm * 32 + j;
      if ((tj & 0xff) == n) {
        const V2<T> v = col[0];
        acc.x += v.x;
        acc.y += v.y;
      }
      if (((tj >> 8) & 0xff) == n) {
        const V2<T> v = col[H * 32];
        acc.x += v.x;
        acc.y += v.y;
      }
      if ((tj >> 16) == n) {
        const V2<T> v = col[(2 * H) * 32];
        acc.x += v.x;
        acc.y += v.y;
      }
    }
    if (act) {
      u2[k].x += acc.x;
      u2[k].y += acc.y;
    }
  }
}

template <typename T>
__device__ __forceinline__ void b3_contract_adjoint(int lmax, int n_ls, int n_tri, int H,
                                                    int nr, const int *__restrict__ tri,
                                                    const V2<T> *__restrict__ z,
                                                    const T *__restrict__ w,
                                                    V2<T> *__restrict__ priv,
                                                    V2<T> *__restrict__ u2, int lane) {
  const int H1 = H + 1;
  const int *beg = c_b3.beg + c_b3.ls_off[lmax];
  for (int r0 = 0; r0 < n_tri; r0 += 32) {
    const int r = r0 + lane;
    const bool live = r < n_tri;
    const int tr = live ? tri[r] : 0;
    for (int k = 0; k < 3 * H; k++) priv[k * 32 + lane] = V2<T>{T(0), T(0)};
    if (live) {
      const int n1 = tr & 0xff, n2 = (tr >> 8) & 0xff, n3 = tr >> 16;
      const V2<T> *z1 = z + n1 * H1, *z2 = z + n2 * H1, *z3 = z + n3 * H1;
      V2<T> *p1 = priv + lane;
      V2<T> *p2 = priv + (size_t)H * 32 + lane;
      V2<T> *p3 = priv + (size_t)(2 * H) * 32 + lane;
      for (int t = 0; t < n_ls; t++) {
        const int e0 = beg[t], e1 = beg[t + 1];
        const T wq = w[r * n_ls + t];
        for (int q = e0; q < e1; q++) {
          const unsigned ix = c_b3.idx[q];
          const int i1 = ix & 0xff, i2 = (ix >> 8) & 0xff, i3 = ix >> 16;
          const T f = wq * b3_w<T>(q);
          const V2<T> a = z1[i1], b = z2[i2], c = z3[i3];
          V2<T> s1 = p1[i1 * 32], s2 = p2[i2 * 32], s3 = p3[i3 * 32];
          s1.x += f * (b.x * c.x - b.y * c.y);
          s1.y += f * (b.x * c.y + b.y * c.x);
          s2.x += f * (a.x * c.x - a.y * c.y);
          s2.y += f * (a.x * c.y + a.y * c.x);
          s3.x += f * (a.x * b.x - a.y * b.y);
          s3.y += f * (a.x * b.y + a.y * b.x);
          p1[i1 * 32] = s1;
          p2[i2 * 32] = s2;
          p3[i3 * 32] = s3;
        }
      }
    }
    __syncwarp();
    b3_reduce_private<T>(r0, n_tri, H, nr, tri, priv, u2, lane);
    __syncwarp();
  }
}

}  // namespace fpp
