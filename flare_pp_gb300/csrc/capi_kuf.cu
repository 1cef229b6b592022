// Host side of the kernel columns by one GEMM (kuf_gemm.cu).
#include <cub/cub.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <string>
#include <vector>

#include "capi_kuf.h"

namespace fpp {

static int round_up(int n, int m) { return (n + m - 1) / m * m; }

// Descriptors that a pair with a neighbor of one species changes.
static int kuf_columns(const B2Args &a) {
  const int N = a.N, others = (a.n_species - 1) * N;
  return (others * N + N * (N + 1) / 2) * (a.lmax + 1);
}

bool kuf_gemm_fits(const fpp_model *m) {
  return m->args.kind == kB2 && kuf_rows_smem(m->args, kuf_columns(m->args), nullptr) > 0;
}

static size_t row_bytes(const fpp_model *m, int ldf) {
  const int k_pad = round_up(kuf_columns(m->args), 64);
  return (size_t)k_pad * 2 * kOzakiDigits + sizeof(double) * (ldf + 1) + sizeof(int);
}

static int sparse_ld(const fpp_model *m) {
  int ldf = 4;
  for (auto &x : m->sp) ldf = std::max(ldf, round_up(x.n_sparse, 4));
  return ldf;
}

size_t kuf_gemm_bytes(const fpp_model *m, long long n_pairs) {
  return (size_t)(3 * n_pairs) * row_bytes(m, sparse_ld(m));
}

// Column tables per neighbor species, and dhat in each class's columns as digit
// planes: rows of class (si, sj) from cls_row[si * n_species + sj].
static int class_operands(fpp_model *m, std::vector<int> &cls_row, cudaStream_t st) {
  const int ns = m->n_species, N = m->args.N, L1 = m->args.lmax + 1, kc = kuf_columns(m->args);
  cls_row.assign(ns * ns + 1, 0);
  for (int c = 0; c < ns * ns; c++) cls_row[c + 1] = cls_row[c] + m->sp[c / ns].n_sparse;
  const int rows = cls_row[ns * ns];
  if (m->kuf_tab.bytes == 0) {
    std::vector<KufColumn> tab;
    tab.reserve((size_t)ns * kc);
    // columns with both channels of the neighbor's species first (they take twice the
    // arithmetic)
    for (int sj = 0; sj < ns; sj++)
      for (int pass = 0; pass < 2; pass++)
        for (size_t q = 0; q < m->pair_tab_host.size(); q++) {
          const int n1 = m->pair_tab_host[q] & 0xffff, n2 = m->pair_tab_host[q] >> 16;
          const bool in1 = n1 / N == sj, in2 = n2 / N == sj;
          if (pass == 0 ? !(in1 && in2) : in1 == in2) continue;
          for (int l = 0; l < L1; l++) {
            KufColumn w;
            w.n1 = (unsigned short)(in2 ? n1 : n2);
            w.n2 = (unsigned char)((in2 ? n2 : n1) % N);
            w.l = (unsigned char)l;
            w.d = (int)q * L1 + l;
            tab.push_back(w);
          }
        }
    if ((int)tab.size() != ns * kc) return fail(FPP_ERR_INVALID, "descriptor column table");
    DevBuf up;
    FPP_TRY(up.reserve(sizeof(KufColumn) * tab.size()));
    FPP_CUDA(cudaMemcpyAsync(up.ptr, tab.data(), sizeof(KufColumn) * tab.size(),
                             cudaMemcpyHostToDevice, st));
    FPP_CUDA(cudaStreamSynchronize(st));
    std::swap(m->kuf_tab.ptr, up.ptr);
    std::swap(m->kuf_tab.bytes, up.bytes);
  }
  if (m->oz_kuf.ready && m->oz_kuf.rows == rows && m->oz_kuf.K == kc) return FPP_OK;
  std::vector<const double *> src;
  std::vector<int> sj;
  for (int c = 0; c < ns * ns; c++)
    for (int k = 0; k < m->sp[c / ns].n_sparse; k++) {
      src.push_back(m->sp[c / ns].d_dhat.as<double>() + (size_t)k * m->n_d);
      sj.push_back(c % ns);
    }
  DevBuf dsrc, dsj, compact;
  FPP_TRY(dsrc.reserve(sizeof(double *) * rows));
  FPP_TRY(dsj.reserve(sizeof(int) * rows));
  FPP_TRY(compact.reserve(sizeof(double) * (size_t)rows * kc));
  FPP_CUDA(cudaMemcpyAsync(dsrc.ptr, src.data(), sizeof(double *) * rows,
                           cudaMemcpyHostToDevice, st));
  FPP_CUDA(cudaMemcpyAsync(dsj.ptr, sj.data(), sizeof(int) * rows, cudaMemcpyHostToDevice, st));
  if (launch_kuf_compact(rows, kc, dsrc.as<const double *>(), dsj.as<int>(),
                         m->kuf_tab.as<KufColumn>(), compact.as<double>(), st) != 0)
    return fail(FPP_ERR_CUDA, "sparse descriptor gather launch failed");
  return ozaki_const(m->oz_kuf, rows, kc, compact.as<double>(), kc, st);
}

// One slice of the batch (its pairs fit in an int).
static int slice(fpp_model *m, KufWork &w, const KufItem *items, int n, double *dK,
                 long long n_labels, cudaStream_t st) {
  const int ns = m->n_species, nd = m->n_d, ldp = round_up(nd, 64), kc = kuf_columns(m->args);
  const int nst = m->n_sparse_total, ldf = sparse_ld(m);
  const size_t rb = row_bytes(m, ldf);
  std::vector<int> cls_row;
  FPP_TRY(class_operands(m, cls_row, st));
  for (int s = 0; s < ns; s++)
    if (m->sp[s].n_sparse > 0)
      FPP_TRY(ozaki_const(m->sp[s].oz_dhat, m->sp[s].n_sparse, nd,
                          m->sp[s].d_dhat.as<double>(), nd, st));
  // structures in chunks of about kuf_chunk_bytes of rows; the digit planes and products
  // of a chunk are written and read once
  struct Chunk {
    int s0, s1;                      // structures
    int blocks0, rows0;              // first atom block, first z row pointer
    int n_blocks, n_atoms;
    std::vector<int> z0;             // first z row of each species (n_species + 1)
    size_t bytes;
  };
  std::vector<Chunk> chunks;
  std::vector<KufGemmStruc> hs(n);
  std::vector<int2> blocks;
  std::vector<const double *> zptr;
  int pairs = 0, max_pairs = 0;
  for (int k = 0; k < n;) {
    Chunk c;
    c.s0 = k;
    c.blocks0 = (int)blocks.size();
    c.rows0 = (int)zptr.size();
    c.n_atoms = 0;
    c.bytes = 0;
    for (; k < n; k++) {
      fpp_structure *s = items[k].s;
      StructureState &S = s->st;
      const bool want_pairs = items[k].q.force_col || items[k].col_f0 >= 0 ||
                              items[k].q.col_s >= 0;
      const size_t b = want_pairs ? 3 * (size_t)S.n_pairs * rb : 0;
      if (k > c.s0 && c.bytes + b > m->kuf_chunk_bytes) break;
      c.bytes += b;
      KufGemmStruc &g = hs[k];
      std::memset(&g, 0, sizeof(g));
      g.s = items[k].q;
      g.s.c64 = S.c64.as<double>();
      g.s.phat64 = S.phat64.as<double>();
      g.s.norm64 = S.norm64.as<double>();
      g.s.row_of_atom = s->row_of_atom.as<int>();
      g.s.species = S.species.as<int>();
      g.s.offset = S.nbr_offset.as<int>();
      g.s.nbr_j = S.nbr_j.as<int>();
      g.s.nbr_s = S.nbr_s.as<int>();
      g.s.rel = S.nbr_rel.as<dvec4>();
      g.s.vol_inv = 1.0 / S.ci.volume;
      g.nbr_i = S.nbr_i.as<int>();
      g.rev = S.nbr_rev.as<int>();
      g.noa = S.noa;
      g.n_pairs = (int)S.n_pairs;
      g.pair0 = pairs;
      g.chunk = (int)chunks.size();
      g.atom0 = c.n_atoms;
      g.block0 = (int)blocks.size() - c.blocks0;
      g.n_blocks = ceil_div(S.noa, kKufAtoms);
      g.want_pairs = want_pairs;
      g.want_es = g.s.col_e >= 0 || g.s.col_s >= 0;
      g.col_f0 = items[k].col_f0;
      for (int b0 = 0; b0 < S.noa; b0 += kKufAtoms) blocks.push_back(make_int2(k, b0));
      c.n_atoms += S.noa;
      pairs += g.n_pairs;
      max_pairs = std::max(max_pairs, g.n_pairs);
    }
    c.s1 = k;
    c.n_blocks = (int)blocks.size() - c.blocks0;
    // z rows of the chunk, species by species
    c.z0.assign(ns + 1, 0);
    for (int s = 0; s < ns; s++) {
      c.z0[s] = (int)zptr.size() - c.rows0;
      for (int q = c.s0; q < c.s1; q++) {
        const fpp_structure *x = items[q].s;
        hs[q].zbase[s] = (int)zptr.size() - c.rows0 - x->row_off[s];
        for (int r = 0; r < x->n_rows[s]; r++)
          zptr.push_back(hs[q].s.phat64 + (size_t)(x->row_off[s] + r) * ldp);
      }
    }
    c.z0[ns] = (int)zptr.size() - c.rows0;
    chunks.push_back(c);
  }
  const int n_chunks = (int)chunks.size(), n_classes = n_chunks * ns * ns;
  // one upload: the structures, the atom blocks, the z row pointers
  const size_t at_blocks = sizeof(KufGemmStruc) * hs.size();
  const size_t at_zptr = at_blocks + sizeof(int2) * blocks.size();
  std::vector<char> up(at_zptr + sizeof(double *) * zptr.size());
  std::memcpy(up.data(), hs.data(), at_blocks);
  std::memcpy(up.data() + at_blocks, blocks.data(), at_zptr - at_blocks);
  std::memcpy(up.data() + at_zptr, zptr.data(), up.size() - at_zptr);
  FPP_TRY(w.tables.reserve(up.size()));
  FPP_CUDA(cudaMemcpyAsync(w.tables.ptr, up.data(), up.size(), cudaMemcpyHostToDevice, st));
  KufGemmArgs ka;
  std::memset(&ka, 0, sizeof(ka));
  ka.a = m->args;
  ka.strucs = w.tables.as<KufGemmStruc>();
  ka.n_strucs = n;
  ka.n_chunks = n_chunks;
  for (int s = 0; s < ns; s++) {
    ka.sp[s].dhat = m->sp[s].d_dhat.as<double>();
    ka.sp[s].norms = m->sp[s].d_norms.as<double>();
    ka.sp[s].n_sparse = m->sp[s].n_sparse;
    ka.sp[s].row0 = m->sp[s].sparse_offset;
  }
  ka.sig2 = m->sigma * m->sigma;
  ka.power = m->power;
  ka.ldp = ldp;
  ka.kuf = dK;
  ka.n_labels = n_labels;
  ka.n_pairs = pairs;
  ka.n_sparse_total = nst;
  ka.cols = m->kuf_tab.as<KufColumn>();
  ka.kc = kc;
  ka.k_same = m->args.N * (m->args.N + 1) / 2 * (m->args.lmax + 1);
  ka.k_pad = round_up(kc, 64);
  ka.ldf = ldf;
  // pairs by class: keys and values in and out, places, class starts, sort scratch
  int bits = 1;
  while ((1ll << bits) <= n_classes) bits++;
  const size_t np4 = sizeof(int) * (size_t)round_up(std::max(pairs, 1), 4);
  size_t sort_bytes = 0;
  FPP_CUDA(cub::DeviceRadixSort::SortPairs(
      nullptr, sort_bytes, (const unsigned *)nullptr, (unsigned *)nullptr, (const int *)nullptr,
      (int *)nullptr, pairs, 0, bits, st));
  FPP_TRY(w.pairs.reserve(5 * np4 + sizeof(int) * (size_t)round_up(n_classes + 1, 4) +
                          sort_bytes + 256));
  char *wp = w.pairs.as<char>();
  ka.keys_in = reinterpret_cast<unsigned *>(wp);
  ka.keys = reinterpret_cast<unsigned *>(wp + np4);
  ka.vals_in = reinterpret_cast<int *>(wp + 2 * np4);
  ka.vals = reinterpret_cast<int *>(wp + 3 * np4);
  ka.place = reinterpret_cast<int *>(wp + 4 * np4);
  ka.start = reinterpret_cast<int *>(wp + 5 * np4);
  const size_t at_sort = (5 * np4 + sizeof(int) * (size_t)round_up(n_classes + 1, 4) + 255) &
                         ~(size_t)255;
  std::vector<int> start(n_classes + 1, 0);
  if (pairs > 0) {
    if (launch_kuf_classes(ka, max_pairs, st) != 0)
      return fail(FPP_ERR_CUDA, "pair class launch failed");
    FPP_CUDA(cub::DeviceRadixSort::SortPairs(wp + at_sort, sort_bytes, ka.keys_in, ka.keys,
                                             ka.vals_in, ka.vals, pairs, 0, bits, st));
    if (launch_kuf_places(ka, n_classes, st) != 0)
      return fail(FPP_ERR_CUDA, "pair class launch failed");
    FPP_CUDA(cudaMemcpyAsync(start.data(), ka.start, sizeof(int) * start.size(),
                             cudaMemcpyDeviceToHost, st));
  }
  FPP_CUDA(cudaStreamSynchronize(st));
  // units: a chunk, or one species of it where its rows exceed the budget (a single
  // large structure)
  struct Unit {
    int chunk, s0, s1;
  };
  std::vector<Unit> units;
  size_t max_rows = 0, max_z = 0, max_atoms = 0, max_blocks = 0;
  auto places = [&](int c, int s0, int s1) {
    return start[(size_t)(c * ns + s1) * ns] - start[(size_t)(c * ns + s0) * ns];
  };
  for (int c = 0; c < n_chunks; c++) {
    if ((size_t)places(c, 0, ns) * 3 * rb <= 2 * m->kuf_chunk_bytes) {
      units.push_back({c, 0, ns});
      max_rows = std::max(max_rows, (size_t)places(c, 0, ns) * 3);
    } else {
      for (int s = 0; s < ns; s++) {
        units.push_back({c, s, s + 1});
        max_rows = std::max(max_rows, (size_t)places(c, s, s + 1) * 3);
      }
    }
    max_z = std::max(max_z, (size_t)chunks[c].z0[ns]);
    max_atoms = std::max(max_atoms, (size_t)chunks[c].n_atoms);
    max_blocks = std::max(max_blocks, (size_t)chunks[c].n_blocks);
  }
  if (max_rows * 2 > (size_t)INT32_MAX / kOzakiDigits)
    return fail(FPP_ERR_CAPACITY, "too many descriptor pairs in one structure");
  const OzakiShape zs = ozaki_shape((int)max_z, nd);
  const OzakiShape rs = ozaki_shape((int)std::max<size_t>(max_rows, 1), kc);
  FPP_TRY(w.z_planes.reserve(zs.plane_bytes + sizeof(int) * std::max<size_t>(max_z, 1)));
  FPP_TRY(w.z.reserve(sizeof(double) * (2 * max_z * ldf + 9 * max_atoms)));
  FPP_TRY(w.planes.reserve(rs.plane_bytes + sizeof(int) * std::max<size_t>(max_rows, 1)));
  FPP_TRY(w.f.reserve(sizeof(double) * std::max<size_t>(max_rows, 1) * (ldf + 1)));
  FPP_TRY(w.partial.reserve(sizeof(double) * 7 * max_blocks * std::max(nst, 1)));
  DeviceStatus *status;
  FPP_TRY(ozaki_status(m->oz, st, &status));
  ka.z = w.z.as<double>();
  ka.acoef = ka.z + max_z * ldf;
  ka.tsum = ka.acoef + max_z * ldf;
  ka.f = w.f.as<double>();
  ka.t = ka.f + max_rows * ldf;
  ka.partial = w.partial.as<double>();
  ka.planes = w.planes.as<__half>();
  ka.exps = reinterpret_cast<int *>(w.planes.as<char>() + rs.plane_bytes);
  int *zexps = reinterpret_cast<int *>(w.z_planes.as<char>() + zs.plane_bytes);
  const int2 *dblocks = reinterpret_cast<const int2 *>(w.tables.as<char>() + at_blocks);
  const double *const *dzptr =
      reinterpret_cast<const double *const *>(w.tables.as<char>() + at_zptr);
  int split = -1;  // the chunk whose descriptors z_planes holds
  for (const Unit &u : units) {
    const Chunk &c = chunks[u.chunk];
    ka.s0 = u.s0;
    ka.s1 = u.s1;
    ka.place0 = start[(size_t)(u.chunk * ns + u.s0) * ns];
    ka.n_places = places(u.chunk, u.s0, u.s1);
    ka.rows_pad = ozaki_shape(std::max(3 * ka.n_places, 1), kc).rows_pad;
    ka.blocks = dblocks + c.blocks0;
    ka.n_blocks = c.n_blocks;
    ka.struc0 = c.s0;
    ka.struc1 = c.s1;
    std::memset(ka.tiles, 0, sizeof(ka.tiles));
    for (int s = u.s0; s < u.s1; s++)
      ka.tiles[s + 1] = ka.tiles[s] + ceil_div(m->sp[s].n_sparse, 32);
    if (ka.tiles[u.s1] == 0) continue;
    // z rows: one split of the chunk's descriptors, before the first of its units that
    // runs (species without sparse environments have none)
    const int nz = c.z0[ns];
    if (split != u.chunk) {
      if (nz > 0 && launch_ozaki_split(nz, nd, nullptr, 0, w.z_planes.as<__half>(), zexps, st,
                                       dzptr + c.rows0) != 0)
        return fail(FPP_ERR_CUDA, "digit-plane split launch failed");
      split = u.chunk;
    }
    if (launch_kuf_rows(ka, st) != 0)
      return fail(FPP_ERR_CUDA, "derivative rows launch failed");
    const OzakiMat zm{w.z_planes.as<__half>(), zexps, nz, nd};
    const OzakiMat fm{ka.planes, ka.exps, 3 * ka.n_places, kc};
    std::vector<OzakiProblem> prob;
    for (int s = u.s0; s < u.s1; s++) {
      const int S = m->sp[s].n_sparse, M = c.z0[s + 1] - c.z0[s];
      if (S == 0 || M == 0) continue;
      prob.push_back(OzakiProblem{zm, ozaki_mat(m->sp[s].oz_dhat), c.z0[s], M, S,
                                  ka.z + (size_t)c.z0[s] * ldf, ldf, false, 0});
      for (int sj = 0; sj < ns; sj++) {
        const size_t cls = (size_t)(u.chunk * ns + s) * ns + sj;
        const int r0 = 3 * (start[cls] - ka.place0), rows = 3 * (start[cls + 1] - start[cls]);
        if (rows > 0)
          prob.push_back(OzakiProblem{fm, ozaki_mat(m->oz_kuf), r0, rows, S,
                                      ka.f + (size_t)r0 * ldf, ldf, false,
                                      cls_row[s * ns + sj]});
      }
    }
    for (size_t q = 0; q < prob.size(); q += kOzakiMaxGroups)
      FPP_TRY(ozaki_run(prob.data() + q, (int)std::min<size_t>(kOzakiMaxGroups, prob.size() - q),
                        status, st));
    if (launch_kuf_coef(ka, st) != 0 || launch_kuf_gather(ka, st) != 0)
      return fail(FPP_ERR_CUDA, "kernel column assembly launch failed");
  }
  return FPP_OK;
}

int kuf_gemm(fpp_model *m, KufWork &w, const std::vector<KufItem> &items, double *dK,
             long long n_labels, cudaStream_t st) {
  // slices whose pairs (and structures, a grid dimension) are counted in an int
  for (size_t k = 0; k < items.size();) {
    size_t e = k;
    long long pairs = 0;
    while (e < items.size() && (e == k || (pairs + items[e].s->st.n_pairs <= m->kuf_slice_pairs &&
                                           e - k < 32768)))
      pairs += items[e++].s->st.n_pairs;
    FPP_TRY(slice(m, w, items.data() + k, (int)(e - k), dK, n_labels, st));
    k = e;
  }
  return FPP_OK;
}

}  // namespace fpp
