// Prints what the mixed form's summation helpers (b2_device.cuh) give for rows of `quads`
// quads of entries whose largest cancel or outweigh the rest.  One warp.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "b2_device.cuh"

using namespace fpp;

// E of a row whose products (2 g + V) delta are 1, 2^-25, 2^-25, -1 in every quad
__global__ void k_energy(AdjArgs g, int nd, const float4 *V, const uint2 *hi, const uint2 *lo,
                         double *out) {
  const int lane = threadIdx.x;
  const double e = w_mixed2(g, 0, nd, make_float2(1.0f, 0.0f), V, hi, lo, [](int, float4) {},
                            lane);
  if (lane == 0) out[0] = e;
}

// |p| of a row that holds 2^-13, 2^-13, 2^-13, 1 in every quad
__global__ void k_norm(int nd, const float *p, double *out) {
  const int lane = threadIdx.x;
  float inv;
  const float2 n = norm_ff(sum_squares(p, nd, lane), inv);
  if (lane == 0) out[1] = (double)n.x + (double)n.y;
}

template <typename T> static T *upload(const std::vector<T> &v) {
  void *p = nullptr;
  if (cudaMalloc(&p, sizeof(T) * v.size()) != cudaSuccess ||
      cudaMemcpy(p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice) != cudaSuccess)
    std::exit(2);
  return static_cast<T *>(p);
}

int main(int argc, char **argv) {
  const int quads = std::atoi(argv[1]), nd = 4 * quads;
  if (quads < 1 || quads > 100000) return 2;
  const float small = 2.98023223876953125e-8f;  // 2^-25
  std::vector<float> v(nd), zero(nd, 0.0f);
  std::vector<__half> hi(nd, __float2half(8192.0f)), lo(nd, __float2half(0.0f));  // delta 1
  for (int q = 0; q < quads; q++) {
    v[4 * q] = 1.0f;
    v[4 * q + 1] = v[4 * q + 2] = small;
    v[4 * q + 3] = -1.0f;
  }
  double *out = upload(std::vector<double>(2, -1.0));
  AdjArgs g;
  std::memset(&g, 0, sizeof(g));
  g.gvec = g.pbar = upload(zero);
  k_energy<<<1, 32>>>(g, nd, reinterpret_cast<const float4 *>(upload(v)),
                      reinterpret_cast<const uint2 *>(upload(hi)),
                      reinterpret_cast<const uint2 *>(upload(lo)), out);
  std::vector<float> p(nd, 1.220703125e-4f);  // 2^-13
  for (int q = 0; q < quads; q++) p[4 * q + 3] = 1.0f;
  k_norm<<<1, 32>>>(nd, upload(p), out);
  double h[2];
  if (cudaMemcpy(h, out, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
  std::printf("energy %.17g\nnorm %.17g\n", h[0], h[1]);
  return 0;
}
