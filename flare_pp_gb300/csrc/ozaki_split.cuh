// One row of the FP64-accurate GEMM's operands cut into digit planes (gemm_ozaki.cu).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "gemm_ozaki.h"

namespace fpp {

// A warp writes the kOzakiDigits digits of the row whose entries load4(k, bits) gives
// (k a multiple of four below k_pad; entries from K on are zeros) at dst + s * plane,
// and returns the row's exponent.  All in integer arithmetic (FP64 issues 2 per clock
// and SM, a split moves an entry per clock): the row maximum by comparing the bit
// patterns of |x|, the digits as the bit fields of the significand shifted to the row's
// scale (rounded to nearest) plus 64 in every place, each pair of digits turned to fp16 by
// one packed subtract.
template <typename Load4>
__device__ __forceinline__ int ozaki_split_row(int K, int k_pad, size_t plane, __half *dst,
                                               int lane, Load4 load4) {
  constexpr unsigned long long kAbs = 0x7fffffffffffffffull;
  unsigned long long mx = 0ull;
  for (int k = 4 * lane; k < K; k += 128) {
    unsigned long long b[4];
    load4(k, b);
#pragma unroll
    for (int i = 0; i < 4; i++) mx = max(mx, b[i] & kAbs);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  // max |x| < 2^e: the biased exponent of the largest entry (a subnormal row
  // keeps the scale of the smallest normal number); Inf and NaN mark the row
  const bool bad = mx >= 0x7ff0000000000000ull;
  const int bex = max((int)(mx >> 52), 1);
  for (int q = lane; q < (k_pad >> 2); q += 32) {
    const int k = 4 * q;
    unsigned long long b[4] = {0ull, 0ull, 0ull, 0ull};
    if (k < K) load4(k, b);
    // signed 55-bit fixed point of x 2^-(e + 1), LSB 2^-56, plus half a digit in every
    // place: the balanced digits are then the plain 7-bit fields less 64
    constexpr unsigned long long kHalf = 0x0081020408102040ull;
    unsigned long long f[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
      const unsigned long long a = b[i] & kAbs;
      const int ex = (int)(a >> 52);
      unsigned long long m = a & 0xfffffffffffffull;
      if (ex > 0) m |= 0x10000000000000ull;
      m <<= 2;                                    // the largest entry's place
      const int sh = bex - max(ex, 1);            // >= 0
      if (sh > 0) m = sh < 56 ? (m + (1ull << (sh - 1))) >> sh : 0ull;
      if (bad) m = 0ull;
      f[i] = (b[i] >> 63) ? kHalf - m : kHalf + m;
    }
#pragma unroll
    for (int s = 0; s < kOzakiDigits; s++) {
      unsigned d[4];
#pragma unroll
      for (int i = 0; i < 4; i++)
        d[i] = (unsigned)(f[i] >> (kOzakiBits * (kOzakiDigits - 1 - s)));
      // 0x6400 | n is the fp16 number 1024 + n, n < 1024 (the top field may be 128)
      const unsigned mask = s == 0 ? 0x00ff00ffu : 0x007f007fu;
      const unsigned p01 = (__byte_perm(d[0], d[1], 0x5410) & mask) | 0x64006400u;
      const unsigned p23 = (__byte_perm(d[2], d[3], 0x5410) & mask) | 0x64006400u;
      const __half2 off = __float2half2_rn(1024.0f + 64.0f);
      const __half2 h01 = __hsub2(*reinterpret_cast<const __half2 *>(&p01), off);
      const __half2 h23 = __hsub2(*reinterpret_cast<const __half2 *>(&p23), off);
      reinterpret_cast<uint2 *>(dst + s * plane)[q] =
          make_uint2(*reinterpret_cast<const unsigned *>(&h01),
                     *reinterpret_cast<const unsigned *>(&h23));
    }
  }
  return bad ? kOzakiNanRow : (mx == 0ull ? 0 : bex - 1022);
}

}  // namespace fpp
