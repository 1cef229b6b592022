// C ABI: mapped-beta prediction of a batch of uneven structures in one pass.
//
// The structures' atoms and neighbor lists are packed into one structure
// (atoms concatenated, each pair list shifted by its structure's atom and pair
// offsets, the FP64 pair table authoritative as for lists given from
// outside), so the forward pass, the contraction and the adjoint each run as
// one launch over every atom of the batch.  A segmented reduction then sums
// each structure's atom energies and pair virials (pair_f (x) r over its own
// pair range), and each stress is its virial over its own volume.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "capi_state.h"
#include "internal.h"

namespace fpp {

// One structure's neighbor data and its place in the packed structure.
struct BatchSrc {
  const int *nbr_i, *nbr_j, *nbr_s, *rev, *offset, *species;
  const dvec4 *rel;
  const float4 *rel32;
  int noa, atom_off;
  long long np, pair_off;
};

// blockIdx.y = structure; its pairs (shifted by its atom and pair offsets)
// and atoms are copied into the packed arrays.  FP64 geometry (32 of a pair's 64 bytes):
// of every pair, or (band) of those whose FP32 distance does not decide the cutoff, the
// only ones whose FP64 geometry the mixed form's kernels read (keep_pair32): 2.9 million
// pairs in 47 us instead of 55.
__global__ void k_batch_pack(const B2Args a, const int band, const BatchSrc *__restrict__ src, int *__restrict__ o_i,
                             int *__restrict__ o_j, int *__restrict__ o_s,
                             int *__restrict__ o_rev, dvec4 *__restrict__ o_rel,
                             float4 *__restrict__ o_rel32, int *__restrict__ o_offset,
                             int *__restrict__ o_species, const int n_atoms,
                             const int n_pairs) {
  const BatchSrc b = src[blockIdx.y];
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) o_offset[n_atoms] = n_pairs;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < b.np; p += stride) {
    const long long q = b.pair_off + p;
    const int i = b.nbr_i[p], sj = b.nbr_s[p];
    const float4 r = b.rel32[p];
    o_i[q] = i + b.atom_off;
    o_j[q] = b.nbr_j[p] + b.atom_off;
    o_s[q] = sj;
    o_rev[q] = b.rev[p] >= 0 ? (int)(b.rev[p] + b.pair_off) : -1;
    o_rel32[q] = r;
    bool exact = true;
    if (band) {
      const int si = b.species[i], k = si * a.n_species + sj;
      // (a species that the model lacks is refused before a kernel reads the pair)
      exact = si < a.n_species && sj < a.n_species && !(r.w < a.cut_lo[k] || r.w > a.cut_hi[k]);
    }
    if (exact) o_rel[q] = b.rel[p];
  }
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < b.noa; i += stride) {
    o_offset[b.atom_off + i] = b.offset[i] + (int)b.pair_off;
    o_species[b.atom_off + i] = b.species[i];
  }
}

// Operand rows of the packed atoms (species by species, in packed order): base[s] of the
// block's structure is the row of its first atom of species s.  (Two host loops over
// 69,380 atoms and a synchronization before, 160 us in which the GPU waited.)
__global__ void __launch_bounds__(256)
k_batch_rows(const BatchSrc *__restrict__ src, int ns, const int *__restrict__ base,
             int *__restrict__ row_of_atom) {
  __shared__ int warp_cnt[8][kMaxSpecies], next[kMaxSpecies];
  const BatchSrc b = src[blockIdx.x];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  if (t < ns) next[t] = base[(size_t)blockIdx.x * ns + t];
  for (int c0 = 0; c0 < b.noa; c0 += 256) {
    const int i = c0 + t, sp = i < b.noa ? b.species[i] : -1;
    int rank = 0;
    for (int s = 0; s < ns; s++) {
      const unsigned m = __ballot_sync(0xffffffffu, sp == s);
      if (sp == s) rank = __popc(m & ((1u << lane) - 1u));
      if (lane == 0) warp_cnt[warp][s] = __popc(m);
    }
    __syncthreads();
    if (sp >= 0) {
      int r = next[sp] + rank;
      for (int w = 0; w < warp; w++) r += warp_cnt[w][sp];
      row_of_atom[b.atom_off + i] = r;
    }
    __syncthreads();
    if (t < ns)
      for (int w = 0; w < 8; w++) next[t] += warp_cnt[w][t];
    __syncthreads();
  }
}

// A finite float as a double by its bit pattern (a conversion is an FP64-pipe
// instruction, of which an SM issues two per clock); zeros, subnormals, Inf and NaN by
// the conversion, out of line (inline, it was issued for every float).
static __device__ __noinline__ double convert(float f) { return (double)f; }
__device__ __forceinline__ double widen(float f) {
  const unsigned u = __float_as_uint(f), e = (u >> 23) & 255u;
  if (__builtin_expect(e - 1u >= 254u, 0)) return convert(f);
  return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + 0x38000000u)),
                          (int)(u << 29));
}
__device__ __forceinline__ double widen(double f) { return f; }

// Sums of f_a r_b over a run of kSumPairs pairs of one structure (a block each), fixed
// order.  Runs of one length because structures differ sixteenfold: with a block per
// structure the SMs that held two large ones took 146 us for 256 structures of 69,380
// atoms (2.9 million pairs; the nine FP64 multiply-adds of a pair take 43), 54 so.
constexpr int kSumPairs = 4096;
template <typename T, typename R>
__global__ void __launch_bounds__(256)
k_batch_sums(const int2 *__restrict__ runs, const long long *__restrict__ pair_off,
             const T *__restrict__ pair_f, const R *__restrict__ rel,
             double *__restrict__ partial) {
  __shared__ double sm[9][256];
  const int2 run = runs[blockIdx.x];  // structure, first pair in it
  const int t = threadIdx.x;
  const long long p0 = pair_off[run.x] + run.y;
  const long long p1 = min(p0 + kSumPairs, pair_off[run.x + 1]);
  double v[9];
#pragma unroll
  for (int k = 0; k < 9; k++) v[k] = 0.0;
#pragma unroll 4
  for (long long p = p0 + t; p < p1; p += 256) {
    double f[3], r[3];
    if constexpr (sizeof(R) == sizeof(dvec4)) {
      const dvec4 d = reinterpret_cast<const dvec4 *>(rel)[p];  // (r, x, y, z)
      const dvec4 g = reinterpret_cast<const dvec4 *>(pair_f)[p];
      f[0] = g.x, f[1] = g.y, f[2] = g.z;
      r[0] = d.y, r[1] = d.z, r[2] = d.w;
    } else {
      const float4 d = reinterpret_cast<const float4 *>(rel)[p];  // (x, y, z, r)
      const float4 g = reinterpret_cast<const float4 *>(pair_f)[p];
      f[0] = widen(g.x), f[1] = widen(g.y), f[2] = widen(g.z);
      r[0] = widen(d.x), r[1] = widen(d.y), r[2] = widen(d.z);
    }
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
      for (int b = 0; b < 3; b++) v[3 * a + b] = fma(f[a], r[b], v[3 * a + b]);
  }
#pragma unroll
  for (int k = 0; k < 9; k++) sm[k][t] = v[k];
  __syncthreads();
  // a warp per sum (FP64 adds of whole warps: 13 per sum, 45 by nine sums in each warp)
  for (int k = t >> 5; k < 9; k += 8) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < 8; w++) s += sm[k][32 * w + (t & 31)];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((t & 31) == 0) partial[(size_t)blockIdx.x * 9 + k] = s;
  }
}

// Per structure (a block each): out[10 s] = sum of its atom energies, out[10 s + 1 + k]
// = sum of its runs' partial sums.
__global__ void __launch_bounds__(128)
k_batch_finish(const int *__restrict__ atom_off, const int *__restrict__ run_off,
               const double *__restrict__ atom_e, const double *__restrict__ partial,
               double *__restrict__ out) {
  __shared__ double sm[4];
  const int s = blockIdx.x, t = threadIdx.x;
  double e = 0.0;
  for (int i = atom_off[s] + t; i < atom_off[s + 1]; i += 128) e += atom_e[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if ((t & 31) == 0) sm[t >> 5] = e;
  __syncthreads();
  if (t < 9) {
    double v = 0.0;
    for (int q = run_off[s]; q < run_off[s + 1]; q++) v += partial[(size_t)q * 9 + t];
    out[10 * s + 1 + t] = v;
  } else if (t == 32) {
    out[10 * s] = (sm[0] + sm[1]) + (sm[2] + sm[3]);
  }
}

}  // namespace fpp

using namespace fpp;

extern "C" int fpp_predict_mapped_batched(fpp_model *m, fpp_structure *const *structures,
                                          int32_t n_structures, int precision,
                                          double *energies, double *forces, double *stresses,
                                          void *stream) {
  if (!m || (n_structures > 0 && !structures)) return fail(FPP_ERR_INVALID, "null argument");
  if (n_structures < 0) return fail(FPP_ERR_INVALID, "negative structure count");
  if (n_structures == 0) return FPP_OK;
  cudaStream_t st = (cudaStream_t)stream;
  std::vector<int> aoff(n_structures + 1, 0);
  std::vector<long long> poff(n_structures + 1, 0);
  for (int k = 0; k < n_structures; k++) {
    fpp_structure *s = structures[k];
    if (!s) return fail(FPP_ERR_INVALID, "null structure");
    FPP_TRY(ensure_rel64(s->st, st));  // the FP64 pair table of each list
    aoff[k + 1] = aoff[k] + s->st.noa;
    poff[k + 1] = poff[k] + s->st.n_pairs;
  }
  const int N = aoff[n_structures];
  const long long P = poff[n_structures];
  if (P >= (1ll << 31)) return fail(FPP_ERR_CAPACITY, "more than 2^31 pairs in the batch");
  if (!m->batch) m->batch = new fpp_structure();
  fpp_structure *b = m->batch;
  StructureState &B = b->st;
  B.noa = N;
  B.n_pairs = P;
  // operand rows as for one structure of all atoms (ensure_layout), their places on the
  // device from each structure's first row of a species
  const int ns = m->n_species;
  b->layout_species = -1;  // species differ from batch to batch
  b->n_rows.assign(ns, 0);
  b->row_off.assign(ns, 0);
  std::vector<int> base((size_t)n_structures * ns);
  for (int k = 0; k < n_structures; k++) {
    const std::vector<int> &c = structures[k]->st.species_count;
    if ((int)c.size() > ns)
      return fail(FPP_ERR_INVALID, "structure species exceeds the descriptor's n_species");
    for (int t = 0; t < ns; t++) {
      base[(size_t)k * ns + t] = b->n_rows[t];
      b->n_rows[t] += t < (int)c.size() ? c[t] : 0;
    }
  }
  b->total_rows = 0;
  for (int t = 0; t < ns; t++) {
    b->row_off[t] = b->total_rows;
    b->total_rows += (std::max(b->n_rows[t], 1) + 127) / 128 * 128;
  }
  for (size_t q = 0; q < base.size(); q++) base[q] += b->row_off[q % ns];
  B.ci.volume = 1.0;
  B.rel64_valid = true;    // the packed FP64 table is authoritative (cells differ)
  const size_t np = (size_t)std::max<long long>(P, 1);
  FPP_TRY(B.species.reserve(sizeof(int) * std::max(N, 1)));
  FPP_TRY(B.nbr_offset.reserve(sizeof(int) * (N + 1)));
  FPP_TRY(B.nbr_i.reserve(sizeof(int) * np));
  FPP_TRY(B.nbr_j.reserve(sizeof(int) * np));
  FPP_TRY(B.nbr_s.reserve(sizeof(int) * np));
  FPP_TRY(B.nbr_rev.reserve(sizeof(int) * np));
  FPP_TRY(B.nbr_rel.reserve(sizeof(dvec4) * np));
  FPP_TRY(B.nbr_rel32.reserve(sizeof(float4) * np));
  if (B.status.bytes < sizeof(DeviceStatus)) {
    FPP_TRY(B.status.reserve(sizeof(DeviceStatus)));
    FPP_CUDA(cudaMemsetAsync(B.status.ptr, 0, sizeof(DeviceStatus), st));
  }
  std::vector<BatchSrc> src(n_structures);
  long long max_work = 1;
  for (int k = 0; k < n_structures; k++) {
    StructureState &S = structures[k]->st;
    BatchSrc &q = src[k];
    q.nbr_i = S.nbr_i.as<int>();
    q.nbr_j = S.nbr_j.as<int>();
    q.nbr_s = S.nbr_s.as<int>();
    q.rev = S.nbr_rev.as<int>();
    q.offset = S.nbr_offset.as<int>();
    q.species = S.species.as<int>();
    q.rel = S.nbr_rel.as<dvec4>();
    q.rel32 = S.nbr_rel32.as<float4>();
    q.noa = S.noa;
    q.atom_off = aoff[k];
    q.np = S.n_pairs;
    q.pair_off = poff[k];
    max_work = std::max(max_work, std::max<long long>(S.n_pairs, S.noa));
  }
  const size_t b_src = sizeof(BatchSrc) * n_structures;
  std::vector<char> up0(b_src + sizeof(int) * base.size());
  std::memcpy(up0.data(), src.data(), b_src);
  std::memcpy(up0.data() + b_src, base.data(), sizeof(int) * base.size());
  FPP_TRY(m->batch_src.reserve(up0.size()));
  FPP_CUDA(cudaMemcpyAsync(m->batch_src.ptr, up0.data(), up0.size(), cudaMemcpyHostToDevice,
                           st));
  FPP_TRY(b->row_of_atom.reserve(sizeof(int) * std::max(N, 1)));
  k_batch_rows<<<n_structures, 256, 0, st>>>(
      m->batch_src.as<BatchSrc>(), ns,
      reinterpret_cast<const int *>(m->batch_src.as<char>() + b_src), b->row_of_atom.as<int>());
  FPP_CUDA(cudaGetLastError());
  b->layout_species = ns;
  // FP64 geometry of every pair where an FP64 kernel runs: the FP64 form, and the first
  // mixed evaluation of a species (which centres it)
  bool band = precision != FPP_PREC_FP64 && (int)m->centred.size() == m->n_species;
  for (char c : m->centred) band = band && c;
  const int tb = 256;
  const int bx = (int)std::min<long long>((max_work + tb - 1) / tb, 1024);
  for (int c0 = 0; c0 < n_structures; c0 += 65535) {  // grid y holds 65535 structures
    const int cy = std::min(65535, n_structures - c0);
    k_batch_pack<<<dim3(bx, cy), tb, 0, st>>>(
        m->args, band, m->batch_src.as<BatchSrc>() + c0, B.nbr_i.as<int>(), B.nbr_j.as<int>(),
        B.nbr_s.as<int>(), B.nbr_rev.as<int>(), B.nbr_rel.as<dvec4>(),
        B.nbr_rel32.as<float4>(), B.nbr_offset.as<int>(), B.species.as<int>(), N, (int)P);
    FPP_CUDA(cudaGetLastError());
  }
  FPP_TRY(mapped_core(m, b, precision, st, 0));
  // per-structure energies and virials
  // one upload: pair offsets, runs of pairs, atom and run offsets
  std::vector<int2> runs;
  std::vector<int> roff(n_structures + 1, 0);
  for (int k = 0; k < n_structures; k++) {
    for (long long p = 0; p < poff[k + 1] - poff[k]; p += kSumPairs)
      runs.push_back(make_int2(k, (int)p));
    roff[k + 1] = (int)runs.size();
  }
  const size_t b_poff = sizeof(long long) * poff.size(), b_runs = sizeof(int2) * runs.size();
  const size_t b_off = sizeof(int) * aoff.size();
  std::vector<char> up(b_poff + b_runs + 2 * b_off);
  std::memcpy(up.data(), poff.data(), b_poff);
  if (b_runs) std::memcpy(up.data() + b_poff, runs.data(), b_runs);
  std::memcpy(up.data() + b_poff + b_runs, aoff.data(), b_off);
  std::memcpy(up.data() + b_poff + b_runs + b_off, roff.data(), b_off);
  DevBuf &d_off = m->batch_off, &d_out = m->batch_sums;
  FPP_TRY(d_off.reserve(up.size()));
  FPP_TRY(d_out.reserve(sizeof(double) * (10 * (size_t)n_structures + 9 * runs.size())));
  FPP_CUDA(cudaMemcpyAsync(d_off.ptr, up.data(), up.size(), cudaMemcpyHostToDevice, st));
  const long long *d_poff = d_off.as<long long>();
  const int2 *d_runs = reinterpret_cast<const int2 *>(d_off.as<char>() + b_poff);
  const int *d_aoff = reinterpret_cast<const int *>(d_off.as<char>() + b_poff + b_runs);
  const int *d_roff = reinterpret_cast<const int *>(d_off.as<char>() + b_poff + b_runs + b_off);
  double *partial = d_out.as<double>() + 10 * (size_t)n_structures;
  if (!runs.empty()) {
    if (precision == FPP_PREC_FP64)
      k_batch_sums<double, dvec4><<<(unsigned)runs.size(), 256, 0, st>>>(
          d_runs, d_poff, B.pair_f.as<double>(), B.nbr_rel.as<dvec4>(), partial);
    else
      k_batch_sums<float, float4><<<(unsigned)runs.size(), 256, 0, st>>>(
          d_runs, d_poff, B.pair_f.as<float>(), B.nbr_rel32.as<float4>(), partial);
    FPP_CUDA(cudaGetLastError());
  }
  k_batch_finish<<<n_structures, 128, 0, st>>>(d_aoff, d_roff, B.atom_e.as<double>(), partial,
                                               d_out.as<double>());
  FPP_CUDA(cudaGetLastError());
  std::vector<double> sums(10 * (size_t)n_structures);
  DeviceStatus hs;
  FPP_CUDA(cudaMemcpyAsync(sums.data(), d_out.ptr, sizeof(double) * sums.size(),
                           cudaMemcpyDeviceToHost, st));
  FPP_CUDA(cudaMemcpyAsync(&hs, B.status.ptr, sizeof(hs), cudaMemcpyDeviceToHost, st));
  if (forces && N)
    FPP_CUDA(cudaMemcpyAsync(forces, B.forces.ptr, sizeof(double) * 3 * N,
                             cudaMemcpyDeviceToHost, st));
  FPP_CUDA(cudaStreamSynchronize(st));
  if (hs.code != 0) {
    FPP_CUDA(cudaMemsetAsync(B.status.ptr, 0, sizeof(DeviceStatus), st));
    return fail(hs.code, "batched prediction: device status " + std::to_string(hs.code) +
                             " at " + std::to_string(hs.where));
  }
  for (int k = 0; k < n_structures; k++) {
    const double *r = sums.data() + 10 * (size_t)k;
    if (energies) energies[k] = r[0];
    if (stresses) {
      // -(1/V) sum f_a r_b, order xx xy xz yy yz zz
      const double vi = 1.0 / structures[k]->st.ci.volume;
      const int ab[6] = {0, 1, 2, 4, 5, 8};
      for (int c = 0; c < 6; c++) stresses[6 * k + c] = -r[1 + ab[c]] * vi;
    }
  }
  return FPP_OK;
}
