// Device helpers shared by the descriptor kernels (b2_kernels.cu, b3_real.cu):
// compensated and float-float sums, the norm and the centred split operand row
// of the mixed form, and its w = dE/dp.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "b2_kernels.h"
#include "common.cuh"
#include "geom.cuh"

namespace fpp {

// Running sum; compensated (Neumaier) when T is float.
template <typename T> struct Acc {
  T s = T(0), c = T(0);
  __device__ __forceinline__ void add(T x) {
    if (sizeof(T) == 4) {
      T t = s + x;
      if (fabs_t(s) >= fabs_t(x))
        c += (s - t) + x;
      else
        c += (x - t) + s;
      s = t;
    } else {
      s += x;
    }
  }
};

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Error-free sum a + b = s + e (Knuth's two-sum), FP32.
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// Warp sum of the float-float values (hi, lo), kept as float-float: FP32
// arithmetic only (FP64 instructions are scarce on this GPU).
__device__ __forceinline__ void ff_warp_sum(float &hi, float &lo) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float h2 = __shfl_xor_sync(0xffffffffu, hi, o);
    const float l2 = __shfl_xor_sync(0xffffffffu, lo, o);
    float s, e;
    two_sum(hi, h2, s, e);
    e += lo + l2;
    hi = s + e;
    lo = e - (hi - s);
  }
}

// |p| as a float-float pair and 1 / |p| from the lanes' sums of p^2: sqrt and
// 1/sqrt by one correction step of the FP32 values (relative error ~1 ulp of FP32),
// no FP64 arithmetic.
__device__ __forceinline__ float2 norm_ff(const Acc<float> &acc, float &invf) {
  float hi = acc.s, lo = acc.c;
  ff_warp_sum(hi, lo);
  const float r0 = sqrtf(hi);
  const float rc = r0 > 0.0f ? (fmaf(-r0, r0, hi) + lo) / (2.0f * r0) : 0.0f;
  const float y0 = r0 > 0.0f ? 1.0f / r0 : 0.0f;
  invf = fmaf(-y0 * y0, rc, y0);
  return make_float2(r0, rc);
}

// This lane's part of sum p^2 over a row in shared memory (nd a multiple of four, 16-byte
// aligned), every square compensated.
__device__ __forceinline__ Acc<float> sum_squares(const float *p, int nd, int lane) {
  Acc<float> acc;
  for (int q = lane; q < (nd >> 2); q += 32) {
    const float4 v = reinterpret_cast<const float4 *>(p)[q];
    acc.add(v.x * v.x);
    acc.add(v.y * v.y);
    acc.add(v.z * v.z);
    acc.add(v.w * v.w);
  }
  return acc;
}

// The centred split operand row of one atom, delta = p / |p| - pbar scaled by 2^13
// as fp16 value and residual (scaled by 2^11), from p in shared memory; nd a
// multiple of four, rows 8-byte aligned: four entries per lane, 16-byte reads,
// 8-byte writes.
__device__ __forceinline__ void write_split_row(const float *p, int nd, float invf,
                                                const float *__restrict__ pbar, __half *hi,
                                                __half *lo, int lane) {
  const float4 *P4 = reinterpret_cast<const float4 *>(p);
  const float4 *B4 = reinterpret_cast<const float4 *>(pbar);
  uint2 *H4 = reinterpret_cast<uint2 *>(hi), *L4 = reinterpret_cast<uint2 *>(lo);
  for (int q = lane; q < (nd >> 2); q += 32) {
    const float4 v = P4[q], b = B4[q];
    const float2 x01 = make_float2((v.x * invf - b.x) * 8192.0f, (v.y * invf - b.y) * 8192.0f);
    const float2 x23 = make_float2((v.z * invf - b.z) * 8192.0f, (v.w * invf - b.w) * 8192.0f);
    // paired conversions (round to nearest)
    const __half2 h01 = __float22half2_rn(x01), h23 = __float22half2_rn(x23);
    const float2 g01 = __half22float2(h01), g23 = __half22float2(h23);
    const __half2 r01 =
        __float22half2_rn(make_float2((x01.x - g01.x) * 2048.0f, (x01.y - g01.y) * 2048.0f));
    const __half2 r23 =
        __float22half2_rn(make_float2((x23.x - g23.x) * 2048.0f, (x23.y - g23.y) * 2048.0f));
    H4[q] = make_uint2(*reinterpret_cast<const unsigned *>(&h01),
                       *reinterpret_cast<const unsigned *>(&h23));
    L4[q] = make_uint2(*reinterpret_cast<const unsigned *>(&r01),
                       *reinterpret_cast<const unsigned *>(&r23));
  }
}

// The mixed power-2 w = dE/dp and energy of one atom from its rows of V and of
// the split operand (global or shared memory): four consecutive entries per
// lane, 16-byte (8-byte for the fp16 planes) loads, |p| and E as float-float.
// store(q, w of entries 4q .. 4q + 3) runs on the lane that read them, so it may
// overwrite V4 in place.
template <typename Store>
__device__ __forceinline__ double w_mixed2(const AdjArgs &g, int si, int nd, float2 nrm32,
                                           const float4 *V4, const uint2 *H4,
                                           const uint2 *L4, Store store, int lane) {
  double e;
  const bool empty = nrm32.x * nrm32.x < g.empty_thresh_f;
  const int nq = nd >> 2;
  const float4 *G4 = reinterpret_cast<const float4 *>(g.gvec + (size_t)si * nd);
  const float4 *B4 = reinterpret_cast<const float4 *>(g.pbar + (size_t)si * nd);
  auto deltas = [&](uint2 h, uint2 l, float (&dl)[4]) {
    const float2 h01 = __half22float2(*reinterpret_cast<const __half2 *>(&h.x));
    const float2 h23 = __half22float2(*reinterpret_cast<const __half2 *>(&h.y));
    const float2 l01 = __half22float2(*reinterpret_cast<const __half2 *>(&l.x));
    const float2 l23 = __half22float2(*reinterpret_cast<const __half2 *>(&l.y));
    dl[0] = (h01.x + l01.x * (1.0f / 2048.0f)) * (1.0f / 8192.0f);
    dl[1] = (h01.y + l01.y * (1.0f / 2048.0f)) * (1.0f / 8192.0f);
    dl[2] = (h23.x + l23.x * (1.0f / 2048.0f)) * (1.0f / 8192.0f);
    dl[3] = (h23.y + l23.y * (1.0f / 2048.0f)) * (1.0f / 8192.0f);
  };
  // loads of kU iterations are issued before any of them is used (one atom's
  // rows are a few KB: the loop is latency-bound without this)
  constexpr int kU = 4;
  Acc<float> acc;
  for (int q0 = lane; q0 < nq; q0 += 32 * kU) {
    uint2 h[kU], l[kU];
    float4 v[kU], gg[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int q = q0 + 32 * u;
      if (q < nq) {
        h[u] = H4[q];
        l[u] = L4[q];
        v[u] = V4[q];
        gg[u] = G4[q];
      }
    }
#pragma unroll
    for (int u = 0; u < kU; u++) {
      if (q0 + 32 * u < nq) {
        float dl[4];
        deltas(h[u], l[u], dl);
        acc.add(fmaf(2.0f, gg[u].x, v[u].x) * dl[0]);
        acc.add(fmaf(2.0f, gg[u].y, v[u].y) * dl[1]);
        acc.add(fmaf(2.0f, gg[u].z, v[u].z) * dl[2]);
        acc.add(fmaf(2.0f, gg[u].w, v[u].w) * dl[3]);
      }
    }
  }
  float hi = acc.s, lo = acc.c;
  ff_warp_sum(hi, lo);
  const ff et = ff_add(ff_norm(hi, lo), ff{g.c0_hi[si], g.c0_lo[si]});
  const float ef = empty ? 0.0f : et.hi + et.lo;
  const float inv = empty ? 0.0f : 1.0f / nrm32.x;
  e = empty ? 0.0 : double(et.hi) + double(et.lo);
  for (int q0 = lane; q0 < nq; q0 += 32 * kU) {
    uint2 h[kU], l[kU];
    float4 v[kU], gg[kU], pb[kU];
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int q = q0 + 32 * u;
      if (q < nq) {
        h[u] = H4[q];
        l[u] = L4[q];
        v[u] = V4[q];
        gg[u] = G4[q];
        pb[u] = B4[q];
      }
    }
#pragma unroll
    for (int u = 0; u < kU; u++) {
      const int q = q0 + 32 * u;
      if (q < nq) {
        float dl[4];
        deltas(h[u], l[u], dl);
        store(q, make_float4(2.0f * ((gg[u].x + v[u].x) - ef * (pb[u].x + dl[0])) * inv,
                             2.0f * ((gg[u].y + v[u].y) - ef * (pb[u].y + dl[1])) * inv,
                             2.0f * ((gg[u].z + v[u].z) - ef * (pb[u].z + dl[2])) * inv,
                             2.0f * ((gg[u].w + v[u].w) - ef * (pb[u].w + dl[3])) * inv));
      }
    }
  }
  return e;
}

}  // namespace fpp
