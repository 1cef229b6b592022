// FP64-accurate C = A B^T on the fp16 tensor cores (tcgen05), by exact
// integer slices (the splitting scheme of Ozaki, Ogita, Oishi and Rump,
// "Error-free transformations of matrix multiplication by using fast routines
// of matrix multiplication and its applications", Numer. Algorithms 59, 2012).
//
// Each row of A (and of B) is scaled by a power of two 2^(e + 1) so that its
// entries lie in (-1/2, 1/2), then cut into kOzakiDigits balanced digits of
// kOzakiBits bits:  a = 2^(e + 1) sum_s d_s 2^(-7 (s + 1)),  |d_s| <= 64, which
// fp16 holds exactly.  For one pair of digit planes (s, t) the products
// d_s d_t are integers of at most 2^12 and a K-sum of them stays an integer;
// the pairs of one level L = s + t (at most 8) summed over a chunk of columns (512
// for 8 pairs, more for fewer) stay within 8 * 512 * 2^12 = 2^24, so the FP32 TMEM
// accumulator holds them EXACTLY whatever order or truncation the tensor cores
// use.  Groups of four levels L0..L1 are then added exactly in 64-bit integers,
//   G = sum_{L0 <= L <= L1} 2^(7 (L1 - L)) S_L,   weight 2^(-14 - 7 L1),
// and the groups, lowest first, by one FP64 multiply-add each.  The operands keep
// 55 bits relative to their row's largest entry, rounded to nearest.  With levels
// 0..7 (36 pairs) the dropped pairs are the largest error, about 2^-55 sqrt(K) of
// the row maxima's product (the digits being balanced they have no common sign);
// with level 8 too (43 pairs) they are below the operands' rounding.
//
// Eleven truncated 5-bit digits held the same bits with 66 pairs instead of 36
// (their level sums could run over 1536 columns, which FP64 epilogue sums need:
// FP64 issues 2 per clock and SM; the integer ones do not).
//
// What bounds it: an N = 128 MMA of one SM takes 64 cycles and reads 8 KB, all of the
// SM's 128 bytes per cycle, and TMA writes there too.  So
//  - a CTA pair (cluster of two, cta_group::2) takes a 256-row tile: each SM reads its own
//    128 rows of A and half of the columns' rows of B, and half of B is loaded;
//  - a K block's digit tiles are loaded once per group of levels and used in all its
//    pairs: the pairs of levels L0..L1 run by ascending A digit s, whose partners
//    t = L0-s .. L1-s are a window sliding down the B digits; A tiles live one step,
//    B tiles four or five (24 tile loads feed 36 pairs; one A and one B tile per
//    pair before).
// Then come the single threads that feed the tensor cores.  The issuer's loops are
// unrolled per group (376 cycles per pair with the slots worked out at run time, where
// the pair's MMAs take 256), its tcgen05 instructions stand under elect.sync, and it
// waits for a step's operands behind the first MMAs of the step before (the tensor
// cores' queue is short: a wait between steps left them idle).  A and B have a producer
// each (one thread took as long to issue 24 loads as the pairs take).
// Measured at 4096 x 2048 x 1500 (36 pairs, one launch), TFLOP/s FP64-equivalent: 13.8
// with the 5-bit digits; 17.7 with these and run-time slots; 26.6 unrolled; 28.9 with
// elect.sync; 34.2 with integer group sums in place of FP64 conversions and 32-byte
// accesses to C; 34.5 with two producers, 37.0 with the waits moved, 41.1 in CTA pairs
// (pairs alone, before the producers and the waits, gave nothing).  1000 x 1050 x 1050:
// 154 us before the last three, 117 so.  The MMAs alone would take 52; 256 tiles over 76
// pairs fill 84 % of four rounds.
//
// Kernel layout (one persistent CTA per SM, 608 threads; in pairs):
//   warps 0, 18    TMA producers (one lane): 128B-swizzled digit tiles, 128 x 64 of A and
//                  bn / 2 x 64 of B, into two rings (A: 8 slots, B: 12); the pair's
//                  loads are counted on the even CTA's barriers
//   warp 1         MMA issuer (the even CTA's, one elected lane): per unit (tile, group
//                  of levels, K chunk) the pairs of its four levels into four
//                  accumulators of bn columns; a level is handed to both epilogues as
//                  soon as its last pair of the chunk is issued
//   warps 2-17     epilogue: four warps per TMEM lane quarter, each owning 32
//                  columns of its 32 rows: tcgen05.ld, then the level's integer
//                  into 64-bit sums held in registers over all chunks.  The
//                  lowest group comes first; its sum waits in C.
// Every wait is bounded; a wait that runs out records FPP_ERR_TIMEOUT in the
// status word and the CTA skips to its exit.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>
#include <mutex>

#include "common.cuh"
#include "gemm_ozaki.h"
#include "ozaki_split.cuh"
#include "tc_prims.cuh"

namespace fpp {

namespace {
constexpr int OBM = 128, OBN = 128, OBK = kTmaBoxK;  // OBN: most columns of a tile
constexpr int OTILE = OBM * OBK * 2;    // bytes of one CTA's A digit tile
constexpr int OBTILE = OTILE / 2;       // most bytes of its half of a B digit tile
constexpr int ONA = 8, ONB = 12;        // ring slots
constexpr int OLEV = 4;                 // levels per half (TMEM accumulators)
constexpr int OTMEM_COLS = OLEV * OBN;
constexpr int OEPI = 16;                // epilogue warps
constexpr int OCOLS = 4 * OBN / OEPI;   // columns of an epilogue warp
constexpr int OPROD_B = 2 + OEPI;       // the second producer warp
constexpr int OTHREADS = 32 * (3 + OEPI);
constexpr int OSMEM_BYTES =
    ONA * OTILE + ONB * OBTILE + 1024 /*align*/ + 512 /*barriers*/;
static_assert(OTMEM_COLS == 512, "four levels of a group fill TMEM");
static_assert(ONB > OLEV + 1, "the live B digits of a step and a slot to fill");
}  // namespace

struct OzakiGroup {
  int M, N, Mp, Np, a_row0, b_row0, kblocks, tiles_n, tile0;
  int b_lower;               // B lower triangular: tile n0 needs K < n0 + bn only
  const int *ea, *eb;        // row exponents of A and of B
  double *C;
  long long ldc;
};

struct OzakiParams {
  // digit planes: rows s * Mp + m (s * Np + n), inner k_pad
  CUtensorMap a[kOzakiMaxGroups], b[kOzakiMaxGroups];
  OzakiGroup g[kOzakiMaxGroups];
  int n_groups, n_tiles;
  int bn;                    // columns of a tile (a multiple of 32, 64 .. OBN)
  int n_levels;              // levels 0 .. n_levels - 1 (8 or 9)
  DeviceStatus *status;
};

// Group sums are at most K 2^34.1 (levels 1-4): below 2^51 up to this K.
constexpr int kLongK = 1 << 16;

// A 64-bit integer below 2^51 in magnitude as FP64, by its bit pattern.
__device__ __forceinline__ double exact_double(long long v) {
  return __longlong_as_double(0x4338000000000000ll + v) - 6755399441055744.0;
}

// hi 2^28 + lo rounded once, for |hi| < 2^50 and |lo| < 2^62: two FP64
// instructions (a 64-bit integer conversion alone takes three).
__device__ __forceinline__ double combine(long long hi, long long lo) {
  constexpr int kB = kOzakiBits * OLEV;
  static_assert(kB == 28, "the constants below");
  hi += lo >> kB;                                  // lo = 2^28 (lo >> 28) + rem, rem >= 0
  const long long rem = lo & ((1ll << kB) - 1);
  const double h = exact_double(hi - (1ll << 24));
  const double r = __longlong_as_double(0x4330000000000000ll | rem);
  return fma(h, 268435456.0, r);
}

// The same where the group sums may leave that range (K above kLongK).
static __device__ __noinline__ double combine_long(long long hi, long long lo) {
  return fma(__ll2double_rn(hi), 268435456.0, __ll2double_rn(lo));
}

// Four consecutive entries of a row of C, of which the first nc are there:
// one 32-byte access where rows are 32-byte aligned (vec).
__device__ __forceinline__ void store4(double *dst, const double (&o)[4], int nc, bool vec) {
  if (vec && nc == 4) {
    asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(dst), "d"(o[0]), "d"(o[1]),
                 "d"(o[2]), "d"(o[3])
                 : "memory");
    return;
  }
#pragma unroll
  for (int k = 0; k < 4; k++)
    if (k < nc) dst[k] = o[k];
}
__device__ __forceinline__ void load4(const double *src, double (&o)[4], int nc, bool vec) {
  if (vec && nc == 4) {
    asm volatile("ld.global.v4.f64 {%0, %1, %2, %3}, [%4];"
                 : "=d"(o[0]), "=d"(o[1]), "=d"(o[2]), "=d"(o[3])
                 : "l"(src)
                 : "memory");
    return;
  }
#pragma unroll
  for (int k = 0; k < 4; k++) o[k] = k < nc ? src[k] : 0.0;
}

// The levels L0..L1 of one pass over a tile and their pairs (s, t) by steps s:
// the partners of A digit s are B digits hi(s) .. lo(s), loaded from top down.
struct LevelGroup {
  int L0, L1;
  // groups of four from the highest level down; the last takes what remains
  __host__ __device__ constexpr LevelGroup(int n_levels, int gr)
      : L0(n_levels - OLEV * (gr + 1) > 0 ? n_levels - OLEV * (gr + 1) : 0),
        L1(n_levels - 1 - OLEV * gr) {}
  static constexpr int D = kOzakiDigits;
  __host__ __device__ constexpr int top() const { return L1 < D ? L1 : D - 1; }
  __host__ __device__ constexpr int steps() const { return top() + 1; }
  __host__ __device__ constexpr int hi(int s) const { return L1 - s < D ? L1 - s : D - 1; }
  __host__ __device__ constexpr int lo(int s) const { return L0 > s ? L0 - s : 0; }
  // K blocks whose level sums stay exact: pairs of one level * K * 64^2 <= 2^24
  __host__ __device__ constexpr int chunk() const { return 4096 / (OBK * (top() + 1)); }
  // first and last step with a pair of level L
  __host__ __device__ static constexpr int first_step(int L) { return L < D ? 0 : L - (D - 1); }
  __host__ __device__ static constexpr int last_step(int L) { return L < D ? L : D - 1; }
};

template <int NL, int GR> struct GroupConst {
  __host__ __device__ static constexpr LevelGroup value() { return LevelGroup(NL, GR); }
};

// A position in a ring of N slots: slot and phase parity without divisions
// (one thread walks the rings, its instruction latency is the kernel's rate).
template <int N> struct RingPos {
  int slot = 0;
  uint32_t parity = 0;
  __device__ __forceinline__ RingPos ahead(int k) const {  // k < N
    RingPos r = *this;
    r.slot += k;
    if (r.slot >= N) {
      r.slot -= N;
      r.parity ^= 1u;
    }
    return r;
  }
  __device__ __forceinline__ void advance(int k) { *this = ahead(k); }
};
// TMEM column of the accumulator of a group's level L0 + l: descending, as the
// B digits of a step (largest first) meet the levels.
__device__ __forceinline__ int acc_col(int l, int bn) { return (OLEV - 1 - l) * bn; }
__device__ __forceinline__ int level_groups(int n_levels) { return (n_levels + OLEV - 1) / OLEV; }

// v 2^k for a finite v, exactly where the result is a normal number (the
// exponent field is moved by an integer add; FP64 instructions are scarce).
__device__ __forceinline__ double scale_pow2(double v, int k) {
  const long long b = __double_as_longlong(v);
  const int ex = (int)((b >> 52) & 0x7ff);
  if (ex != 0 && ex + k > 0 && ex + k < 0x7ff)
    return __longlong_as_double(b + ((long long)k << 52));
  // zero, or a result at the ends of the range: |k| < 3 * 1000
  auto p2 = [](int n) { return __longlong_as_double((long long)(1023 + n) << 52); };
  const int k1 = k / 3, k2 = (k - k1) / 2;
  return v * p2(k1) * p2(k2) * p2(k - k1 - k2);
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(OTHREADS, 1)
k_ozaki_gemm(const __grid_constant__ OzakiParams p) {
  const int bn = p.bn;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  unsigned char *gbase = smem_raw + (base - raw);
  constexpr int kBarOff = ONA * OTILE + ONB * OBTILE;
  constexpr int kBars = 2 * (ONA + ONB) + 2 * OLEV;
  const uint32_t bars = base + kBarOff;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(gbase + kBarOff + 8 * kBars);
  volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
  auto a_slot = [&](int s) { return base + (uint32_t)s * OTILE; };
  const uint32_t b_bytes = (uint32_t)bn * OBK;  // half a B digit tile (bn / 2 rows)
  auto b_slot = [&](int s) { return base + (uint32_t)ONA * OTILE + (uint32_t)s * b_bytes; };
  auto a_full = [&](int s) { return bars + 8u * s; };
  auto a_empty = [&](int s) { return bars + 8u * (ONA + s); };
  auto b_full = [&](int s) { return bars + 8u * (2 * ONA + s); };
  auto b_empty = [&](int s) { return bars + 8u * (2 * ONA + ONB + s); };
  auto accf_bar = [&](int l) { return bars + 8u * (2 * (ONA + ONB) + l); };
  auto acce_bar = [&](int l) { return bars + 8u * (2 * (ONA + ONB) + OLEV + l); };

  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
  const int lane = threadIdx.x & 31;
  // CTA pairs walk the tiles; the even CTA issues the pair's MMAs
  const uint32_t rank = blockIdx.x & 1u;
  const int cid = (int)blockIdx.x >> 1, ncta = (int)gridDim.x >> 1;
  const int ngr = level_groups(p.n_levels);

  if (threadIdx.x == 0) {
    for (int s = 0; s < ONA; s++) {
      mbar_init(a_full(s), 1);
      mbar_init(a_empty(s), 1);
    }
    for (int s = 0; s < ONB; s++) {
      mbar_init(b_full(s), 1);
      mbar_init(b_empty(s), 1);
    }
    for (int l = 0; l < OLEV; l++) {
      mbar_init(accf_bar(l), 1);
      mbar_init(acce_bar(l), 2 * OEPI);  // both CTAs' epilogues (the even CTA's is used)
    }
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 2) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(OTMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster_sync();  // both CTAs' barriers are there
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  // tile t -> its product, row and column origin, K blocks (all of K, or with
  // a lower-triangular B, whose row n is zero beyond column n, only the blocks
  // below n0 + bn)
  auto locate = [&](int t, int &gi, int &mrow, int &n0, int &kbt) {
    gi = 0;
    while (gi + 1 < p.n_groups && t >= p.g[gi + 1].tile0) gi++;
    const OzakiGroup &g = p.g[gi];
    const int lt = t - g.tile0;
    mrow = (lt / g.tiles_n) * (2 * OBM) + (int)rank * OBM;  // this CTA's rows
    n0 = (lt % g.tiles_n) * bn;
    kbt = g.kblocks;
    if (g.b_lower) kbt = min(kbt, (n0 + bn + OBK - 1) / OBK);
  };

  if (warp == 0 || warp == OPROD_B) {
    // ---------------- TMA producers: A digits, B digits ----------------
    if (lane == 0) {
      bool stop = false;
      auto wait_slot = [&](uint32_t bar, uint32_t parity, int t) {
        if (!mbar_wait(bar, parity)) {
          set_status(p.status, FPP_ERR_TIMEOUT, 211, t);
          *abort_flag = 1;
        }
        if (*abort_flag) stop = true;
        return !stop;
      };
      auto walk = [&](auto pos, auto &&load) {  // load(next position, digit) of each K block
        for (int t = cid; t < p.n_tiles && !stop; t += ncta) {
          int gi, mrow, n0, kbt;
          locate(t, gi, mrow, n0, kbt);
          for (int gr = 0; gr < ngr && !stop; gr++) {
            const LevelGroup G(p.n_levels, gr);
            for (int kb = 0; kb < kbt && !stop; kb++)
              for (int s = 0; s < G.steps() && !stop; s++) load(pos, t, gi, mrow, n0, kb, s, G);
          }
        }
        return pos;
      };
      if (warp == 0) {
        RingPos<ONA> ia = walk(RingPos<ONA>{}, [&](RingPos<ONA> &i, int t, int gi, int mrow, int,
                                                   int kb, int s, const LevelGroup &) {
          if (!wait_slot(a_empty(i.slot), i.parity ^ 1u, t)) return;
          if (rank == 0) mbar_expect_tx(a_full(i.slot), 2 * OTILE);  // both CTAs' loads
          tma_pair_load_2d(a_slot(i.slot), &p.a[gi], in_cta(a_full(i.slot), 0), kb * OBK,
                           s * p.g[gi].Mp + p.g[gi].a_row0 + mrow);
          i.advance(1);
        });
        // drain: every slot this CTA filled has been read before it exits
        for (int d = 0; d < ONA && !*abort_flag; d++, ia.advance(1))
          if (!mbar_wait(a_empty(ia.slot), ia.parity ^ 1u)) {
            set_status(p.status, FPP_ERR_TIMEOUT, 215, d);
            *abort_flag = 1;
          }
      } else {
        // a group's steps use B digits top .. 0, largest first: digit top - s at turn s
        RingPos<ONB> ib = walk(RingPos<ONB>{}, [&](RingPos<ONB> &i, int t, int gi, int, int n0,
                                                   int kb, int s, const LevelGroup &G) {
          if (!wait_slot(b_empty(i.slot), i.parity ^ 1u, t)) return;
          if (rank == 0) mbar_expect_tx(b_full(i.slot), 2 * b_bytes);
          tma_pair_load_2d(b_slot(i.slot), &p.b[gi], in_cta(b_full(i.slot), 0), kb * OBK,
                           (G.top() - s) * p.g[gi].Np + p.g[gi].b_row0 + n0 +
                               (int)rank * (bn / 2));
          i.advance(1);
        });
        for (int d = 0; d < ONB && !*abort_flag; d++, ib.advance(1))
          if (!mbar_wait(b_empty(ib.slot), ib.parity ^ 1u)) {
            set_status(p.status, FPP_ERR_TIMEOUT, 216, d);
            *abort_flag = 1;
          }
      }
    }
  } else if (warp == 1 && rank == 0) {
    // ---------------- MMA issuer (the even CTA's) ----------------
    // ib: slot of the K block's first B digit; unit: uses of accumulator 0, of
    // the others (a group of one level leaves them out).  Everything but the
    // waits is unrolled per group of levels: with the slots and levels worked
    // out at run time this thread took 376 cycles per pair, the pair's four
    // MMAs 256.
    RingPos<ONA> ia;
    RingPos<ONB> ib;
    int unit = 0, unit_rest = 0;
    bool stop = false;
    const uint64_t da0 = smem_desc(base), db0 = smem_desc(base + ONA * OTILE);
    const uint32_t b_step = b_bytes >> 4;
    auto wait_or_abort = [&](uint32_t bar, uint32_t parity, int site, int t) {
      if (!mbar_wait(bar, parity)) {
        if (lane == 0) set_status(p.status, FPP_ERR_TIMEOUT, site, t);
        *abort_flag = 1;
      }
    };
    auto k_block = [&](auto lc, bool chunk_first, bool chunk_last, int t) {
      constexpr LevelGroup G = decltype(lc)::value();
      // the A digit and the B digits first used at step s
      auto wait_step = [&](int s, RingPos<ONA> qa) {
        wait_or_abort(a_full(qa.slot), qa.parity, 213, t);
#pragma unroll
        for (int d = s == 0 ? G.top() : G.lo(s - 1) - 1; d >= G.lo(s); d--) {
          const RingPos<ONB> q = ib.ahead(G.top() - d);
          wait_or_abort(b_full(q.slot), q.parity, 213, t);
        }
      };
      wait_step(0, ia);
      if (__any_sync(0xffffffffu, *abort_flag)) return false;
#pragma unroll
      for (int s = 0; s < G.steps(); s++) {
        const bool fresh = chunk_first && s <= G.first_step(G.L1);
        if (fresh) {
          // the accumulators of the levels that start at this step
#pragma unroll
          for (int L = G.L0; L <= G.L1; L++)
            if (s == G.first_step(L))
              wait_or_abort(acce_bar(L - G.L0),
                            (uint32_t)((L == G.L0 ? unit : unit_rest) & 1) ^ 1u, 212, t);
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t pa = da0 + (uint64_t)(ia.slot * (OTILE >> 4));
#pragma unroll
        for (int j = 0; j < OLEV; j++) {
          const int d = G.hi(s) - j;
          if (d < G.lo(s)) continue;
          const uint64_t pb = db0 + (uint64_t)(ib.ahead(G.top() - d).slot * b_step);
          const uint32_t acc = tmem + (uint32_t)acc_col(s + d - G.L0, bn);
          const uint32_t add = s == G.first_step(s + d) && chunk_first ? 0u : 1u;
          if (elect_one()) {
#pragma unroll
            for (int ks = 0; ks < OBK / 16; ks++)
              mma_pair_f16(acc, pa + ks * 2, pb + ks * 2, bn, ks == 0 ? add : 1u);
          }
          // the next step's operands, while these MMAs run: a wait costs more than
          // the few MMAs that queue behind each other take
          if (j == 0 && s + 1 < G.steps()) wait_step(s + 1, ia.ahead(1));
        }
        // free the slots once these MMAs read them: the A digit, and the B
        // digits without a later partner
        if (elect_one()) {
          mma_pair_commit(a_empty(ia.slot));
#pragma unroll
          for (int d = G.top(); d >= 0; d--) {
            const int last = G.L1 - d < G.steps() ? G.L1 - d : G.steps() - 1;
            if (s == last) mma_pair_commit(b_empty(ib.ahead(G.top() - d).slot));
          }
          if (chunk_last) {
#pragma unroll
            for (int L = G.L0; L <= G.L1; L++)
              if (s == G.last_step(L)) mma_pair_commit(accf_bar(L - G.L0));
          }
        }
        __syncwarp();
        ia.advance(1);
      }
      ib.advance(G.steps());
      if (chunk_last) {
        unit++;
        if (G.L1 > G.L0) unit_rest++;
      }
      return true;
    };
    for (int t = cid; t < p.n_tiles && !stop; t += ncta) {
      int gi, mrow, n0, kbt;
      locate(t, gi, mrow, n0, kbt);
      for (int gr = 0; gr < ngr && !stop; gr++)
        for (int kb = 0; kb < kbt && !stop; kb++) {
          const int chunk = LevelGroup(p.n_levels, gr).chunk();
          const bool first = kb % chunk == 0;
          const bool last = kb + 1 == kbt || (kb + 1) % chunk == 0;
          bool ok;
          if (p.n_levels == 8)
            ok = gr == 0 ? k_block(GroupConst<8, 0>{}, first, last, t)
                         : k_block(GroupConst<8, 1>{}, first, last, t);
          else
            ok = gr == 0   ? k_block(GroupConst<9, 0>{}, first, last, t)
                 : gr == 1 ? k_block(GroupConst<9, 1>{}, first, last, t)
                           : k_block(GroupConst<9, 2>{}, first, last, t);
          stop = !ok;
        }
    }
    if (__any_sync(0xffffffffu, *abort_flag)) {  // release the epilogue
      if (elect_one())
        for (int l = 0; l < OLEV; l++) mma_pair_commit(accf_bar(l));
    }
  } else if (warp != 1) {
    // ---------------- epilogue ----------------
    const int q = warp & 3;                 // TMEM lane quarter this warp may access
    const int colh = (warp - 2) / 4;        // which OCOLS columns of the tile
    const uint32_t lane_base = (uint32_t)(q * 32) << 16;
    int unit = 0, unit_rest = 0;
    bool stop = false;
    for (int t = cid; t < p.n_tiles && !stop; t += ncta) {
      int gi, mrow, n0, kbt;
      locate(t, gi, mrow, n0, kbt);
      const OzakiGroup &g = p.g[gi];
      const int n_end = min(g.N, n0 + bn);  // this tile's columns
      n0 += colh * OCOLS;
      const int r = mrow + q * 32 + lane;
      double *crow = g.C + (size_t)r * g.ldc + n0;
      const bool long_k = kbt * OBK > kLongK;
      const bool vec = (g.ldc & 3) == 0 && (reinterpret_cast<uintptr_t>(g.C) & 31u) == 0;
      for (int gr = 0; gr < ngr && !stop; gr++) {
        const LevelGroup G(p.n_levels, gr);
        const int nch = (kbt + G.chunk() - 1) / G.chunk();
        long long acc[OCOLS];
#pragma unroll
        for (int i = 0; i < OCOLS; i++) acc[i] = 0;
        for (int c = 0; c < nch && !stop; c++, unit++, unit_rest += G.L1 > G.L0) {
          for (int l = 0; l < OLEV; l++) {
            if (l > G.L1 - G.L0) break;  // a group of one level
            bool have = mbar_wait(accf_bar(l), (uint32_t)((l == 0 ? unit : unit_rest) & 1));
            have = __all_sync(0xffffffffu, have) != 0;
            if (!have) {
              if (lane == 0) set_status(p.status, FPP_ERR_TIMEOUT, 214, t);
              *abort_flag = 1;
            }
            if (__shfl_sync(0xffffffffu, *abort_flag, 0)) {
              stop = true;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t tm = tmem + (uint32_t)(acc_col(l, bn) + colh * OCOLS) + lane_base;
            const int w = 1 << (kOzakiBits * (G.L1 - G.L0 - l));  // weight of the level
#pragma unroll
            for (int i0 = 0; i0 < OCOLS; i0 += 16) {
              float v[16];
              tmem_ld16(tm + i0, v);
#pragma unroll
              for (int i = 0; i < 16; i++)
                acc[i0 + i] += (long long)__float2int_rn(v[i]) * w;
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(in_cta(acce_bar(l), 0));
          }
        }
        if (stop) break;
        if (r < g.M) {
          // The sum of the groups so far returns to the thread that stored it:
          // the lowest group as a 64-bit integer, then FP64, in units of the lowest
          // group's weight.
          const bool last = gr + 1 == ngr;
          const int er = last ? g.ea[r] : 0;
          const int shift = 2 - kOzakiBits * (2 + p.n_levels - 1);
#pragma unroll
          for (int i = 0; i < OCOLS; i += 4) {
            asm volatile("" ::: "memory");  // one block of loads in flight per four columns
            const int nc = min(n_end - (n0 + i), 4);
            if (nc <= 0) break;
            double *dst = crow + i;
            if (gr == 0) {
              const long long o[4] = {acc[i], acc[i + 1], acc[i + 2], acc[i + 3]};
              store4(dst, reinterpret_cast<const double(&)[4]>(o), nc, vec);
              continue;
            }
            double before[4], o[4];
            load4(dst, before, nc, vec);
#pragma unroll
            for (int k = 0; k < 4; k++) {
              // after combine in units of the lowest group's weight
              double v;
              if (gr == 1)
                v = long_k ? combine_long(acc[i + k], __double_as_longlong(before[k]))
                           : combine(acc[i + k], __double_as_longlong(before[k]));
              else
                v = fma(long_k ? __ll2double_rn(acc[i + k]) : exact_double(acc[i + k]),
                        72057594037927936.0, before[k]);
              if (last) {
                const int ec = k < nc ? g.eb[n0 + i + k] : 0;
                v = (er == kOzakiNanRow || ec == kOzakiNanRow)
                        ? __longlong_as_double(0x7ff8000000000000ll)
                        : scale_pow2(v, er + ec + shift);
              }
              o[k] = v;
            }
            store4(dst, o, nc, vec);
          }
        }
        __syncwarp();
      }
    }
  }
  if (*abort_flag) settle_in_flight();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  cluster_sync();  // the peer no longer reads, writes or signals this CTA's memory
  if (warp == 2) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(OTMEM_COLS)
                 : "memory");
  }
}

// The bits of v 2^k (exactly where that is a normal number; zeros, Inf and NaN as they are).
__device__ __forceinline__ unsigned long long shift_bits(unsigned long long b, int k) {
  const int ex = (int)((b >> 52) & 0x7ff);
  if (ex != 0 && ex != 0x7ff && ex + k > 0 && ex + k < 0x7ff)
    return b + ((unsigned long long)(long long)k << 52);
  if (ex == 0x7ff || (b << 1) == 0ull) return b;
  return (unsigned long long)__double_as_longlong(
      scale_pow2(__longlong_as_double((long long)b), k));
}

// Digit planes of the rows of X (rows x K, leading dimension ldx; or the rows that
// `ptr` points to), their columns scaled by cols: a warp per row, four entries per lane;
// rows >= rows and columns >= K of the padded planes are zeros.
__global__ void __launch_bounds__(256)
k_ozaki_split(int rows, int K, long long ldx, const double *__restrict__ X,
              const double *const *__restrict__ ptr, int rows_pad, int k_pad,
              __half *__restrict__ planes, int *__restrict__ exps, const OzakiColumns cols) {
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (r >= rows_pad) return;
  const size_t plane = (size_t)rows_pad * k_pad;
  __half *dst = planes + (size_t)r * k_pad;
  if (r >= rows) {
    for (int s = 0; s < kOzakiDigits; s++)
      for (int q = lane; q < (k_pad >> 2); q += 32)
        reinterpret_cast<uint2 *>(dst + s * plane)[q] = make_uint2(0u, 0u);
    return;
  }
  const double *x = ptr ? ptr[r] : X + (size_t)r * ldx;
  const bool al = (reinterpret_cast<uintptr_t>(x) & 15u) == 0;
  const int *sh = nullptr;
  for (int g = 0; g < cols.n; g++)
    if (r >= cols.row0[g]) sh = cols.shift[g];
  const int e = ozaki_split_row(
      K, k_pad, plane, dst, lane, [&](int k, unsigned long long (&b)[4]) {
        if (al && k + 4 <= K) {
          const ulonglong2 u = reinterpret_cast<const ulonglong2 *>(x + k)[0];
          const ulonglong2 v = reinterpret_cast<const ulonglong2 *>(x + k)[1];
          b[0] = u.x, b[1] = u.y, b[2] = v.x, b[3] = v.y;
        } else {
#pragma unroll
          for (int i = 0; i < 4; i++)
            b[i] = k + i < K ? (unsigned long long)__double_as_longlong(x[k + i]) : 0ull;
        }
        if (sh) {
          const int4 c = *reinterpret_cast<const int4 *>(sh + k);
          b[0] = shift_bits(b[0], cols.sign * c.x);
          b[1] = shift_bits(b[1], cols.sign * c.y);
          b[2] = shift_bits(b[2], cols.sign * c.z);
          b[3] = shift_bits(b[3], cols.sign * c.w);
        }
      });
  if (lane == 0) exps[r] = e;
}

// One damped step of the equilibration of a symmetric matrix: e_out[i] = (e_i + r_i) / 2
// with 2^r_i the largest |a_ij| 2^-e_j of row i (at its fixed point the largest
// |a_ij| 2^(-e_i - e_j) of every row is about 1); e_in null: zeros.  A warp per row;
// entries n .. n4 - 1 of e_out are set to zero.
constexpr int kMaxShift = 400;
__global__ void __launch_bounds__(128)
k_equilibrate(int n, int n4, int lda, const double *__restrict__ a,
              const int *__restrict__ e_in, int *__restrict__ e_out) {
  const int i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (i >= n) {
    if (i < n4 && lane == 0) e_out[i] = 0;
    return;
  }
  constexpr int kNone = -(1 << 20);
  int r = kNone;
  const double *row = a + (size_t)i * lda;
  for (int j0 = lane; j0 < n; j0 += 32 * 16) {  // sixteen loads in flight
    long long b[16];
    int e[16];
#pragma unroll
    for (int u = 0; u < 16; u++) {
      const int j = j0 + 32 * u;
      b[u] = j < n ? __double_as_longlong(row[j]) : 0ll;
      e[u] = e_in && j < n ? e_in[j] : 0;
    }
#pragma unroll
    for (int u = 0; u < 16; u++) {
      const int ex = (int)((b[u] >> 52) & 0x7ff);
      if (ex != 0) r = max(r, ex - 1023 - e[u]);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) r = max(r, __shfl_xor_sync(0xffffffffu, r, o));
  // a column of zeros: out of the way of its rows' largest entry
  if (lane == 0)
    e_out[i] = r == kNone
                   ? -kMaxShift
                   : max(-kMaxShift, min(kMaxShift, ((e_in ? e_in[i] : 0) + r) >> 1));
}

int launch_equilibrate(int n, const double *a, int lda, int *shift, int *tmp,
                       cudaStream_t stream) {
  if (n <= 0) return 0;
  const int n4 = (n + 3) / 4 * 4;
  // six steps: a factor that spans 2^80 is then within 2^(80 / 64) of its fixed point
  for (int it = 0; it < 6; it++)
    k_equilibrate<<<ceil_div(n4, 4), 128, 0, stream>>>(
        n, n4, lda, a, it == 0 ? nullptr : (it & 1 ? tmp : shift), it & 1 ? shift : tmp);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

static int ozaki_launch_shape(int dev, int *pairs) {
  constexpr int kMaxDev = 64;
  static std::mutex mu;
  static int cached[kMaxDev] = {0};
  if (dev < 0 || dev >= kMaxDev) return -1;
  std::lock_guard<std::mutex> lock(mu);
  if (cached[dev] == 0) {
    if (cudaFuncSetAttribute(k_ozaki_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             OSMEM_BYTES) != cudaSuccess)
      return -1;
    // resident CTA pairs (an SM without a partner in its cluster group stays idle)
    cudaLaunchConfig_t cfg;
    std::memset(&cfg, 0, sizeof(cfg));
    cfg.gridDim = dim3(2, 1, 1);
    cfg.blockDim = dim3(OTHREADS, 1, 1);
    cfg.dynamicSmemBytes = OSMEM_BYTES;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 2;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, k_ozaki_gemm, &cfg) != cudaSuccess || n < 1) return -1;
    cached[dev] = n;
  }
  *pairs = cached[dev];
  return 0;
}

OzakiShape ozaki_shape(int rows, int K) {
  OzakiShape s;
  s.rows_pad = (rows + OBM - 1) / OBM * OBM;
  s.k_pad = (K + OBK - 1) / OBK * OBK;
  s.plane_bytes = (size_t)s.rows_pad * s.k_pad * sizeof(__half) * kOzakiDigits;
  return s;
}

int launch_ozaki_split(int rows, int K, const double *X, long long ldx, __half *planes,
                       int *exps, cudaStream_t stream, const double *const *row_ptr,
                       const OzakiColumns *cols) {
  if (rows <= 0) return 0;
  const OzakiShape sh = ozaki_shape(rows, K);
  const int threads = 256;
  const long long warps = sh.rows_pad;
  const int blocks = (int)((warps * 32 + threads - 1) / threads);
  k_ozaki_split<<<blocks, threads, 0, stream>>>(rows, K, ldx, X, row_ptr, sh.rows_pad,
                                                 sh.k_pad, planes, exps,
                                                 cols ? *cols : OzakiColumns{});
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

// Columns of a tile for all products of a launch (the rings' slots are sized by
// them): the cheapest count of rounds of tiles over the CTA pairs, a tile costing about
// bn + 300 (its A digits are read and its sums drained whatever bn is).  Narrower tiles
// pay where they add no round: 16384 x 150 x 544 with two tiles of 96 columns instead
// of 128 takes 160 us instead of 176, 1000 x 1050 x 1050 with 68 tiles of 64 instead of
// 36 of 128 takes 117 instead of 141.  Over 224 shapes (M 128 to 16384, N 50 to 1500, K 144 to
// 1500; whole calls) the choice is within 5 % of the fastest width at all but four, 13 % at
// worst.
static int tile_columns(const OzakiProblem *probs, int n, int pairs) {
  int best = OBN;
  long long cost = 0;
  for (int bn : {OBN, 96, 64}) {
    long long tiles = 0;
    for (int k = 0; k < n; k++)
      if (probs[k].M > 0 && probs[k].N > 0)
        tiles += (long long)ceil_div(probs[k].M, 2 * OBM) * ceil_div(probs[k].N, bn);
    const long long c = (tiles + pairs - 1) / pairs * (bn + 300);
    if (bn == OBN || c < cost) {
      best = bn;
      cost = c;
    }
  }
  return best;
}

int launch_ozaki_gemm(const OzakiProblem *probs, int n_probs, DeviceStatus *status,
                      cudaStream_t stream, int n_levels) {
  if (n_probs > kOzakiMaxGroups || (n_levels != 8 && n_levels != 9)) return -2;
  int dev = 0, pairs = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || ozaki_launch_shape(dev, &pairs) != 0) return -1;
  OzakiParams p;
  std::memset(&p, 0, sizeof(p));
  p.bn = tile_columns(probs, n_probs, pairs);
  int tiles = 0;
  for (int k = 0; k < n_probs; k++) {
    const OzakiProblem &q = probs[k];
    if (q.M <= 0 || q.N <= 0) continue;
    if (q.a.K <= 0 || q.a.K != q.b.K || q.a_row0 < 0 || q.a_row0 + q.M > q.a.rows ||
        q.b_row0 < 0 || q.b_row0 + q.N > q.b.rows || q.ldc < q.N)
      return -2;
    const OzakiShape sa = ozaki_shape(q.a.rows, q.a.K), sb = ozaki_shape(q.b.rows, q.b.K);
    if (((uintptr_t)q.a.planes | (uintptr_t)q.b.planes) % 16 != 0) return -2;
    const int i = p.n_groups++;
    // one map over all digit planes of an operand: rows s * rows_pad + row
    if (make_map(&p.a[i], q.a.planes, sa.k_pad, sa.rows_pad * kOzakiDigits, sa.k_pad, OBM) ||
        make_map(&p.b[i], q.b.planes, sb.k_pad, sb.rows_pad * kOzakiDigits, sb.k_pad, p.bn / 2))
      return -3;
    OzakiGroup &g = p.g[i];
    g.M = q.M;
    g.N = q.N;
    g.Mp = sa.rows_pad;
    g.Np = sb.rows_pad;
    g.a_row0 = q.a_row0;
    g.b_row0 = q.b_row0;
    g.kblocks = sa.k_pad / OBK;
    g.tiles_n = ceil_div(q.N, p.bn);
    g.tile0 = tiles;
    g.b_lower = q.b_lower ? 1 : 0;
    g.ea = q.a.exps + q.a_row0;
    g.eb = q.b.exps + q.b_row0;
    g.C = q.C;
    g.ldc = q.ldc;
    tiles += ceil_div(q.M, 2 * OBM) * g.tiles_n;
  }
  if (tiles == 0) return 0;
  p.n_tiles = tiles;
  p.n_levels = n_levels;
  p.status = status;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof(cfg));
  cfg.blockDim = dim3(OTHREADS, 1, 1);
  cfg.dynamicSmemBytes = OSMEM_BYTES;
  cfg.stream = stream;
  cfg.gridDim = dim3(2 * (tiles < pairs ? tiles : pairs), 1, 1);
  if (cudaLaunchKernelEx(&cfg, k_ozaki_gemm, p) != cudaSuccess) return -1;
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

}  // namespace fpp
