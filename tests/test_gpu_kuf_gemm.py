"""Kuf by one GEMM over the pairs' derivative rows, at the edges of its tiles and
tables: one to three species, one to sixteen channels, lmax 0 and past the unrolled
degrees, sparse counts around a 32-wide tile, structures of a few atoms, atoms
without neighbors, structures with some of the labels, and the count of sparse
environments at which the adjoint form takes over.

Tolerance: an entry is a sum over at most 100 pairs of products of K <= 2000
terms, each operand within 2^-55 of its row's largest entry: 2^-55 * 2000 * 100 =
6e-12 of the largest product a * dp * dhat, which is itself of the order of the
largest kernel entry; 1e-10 of that."""
import numpy as np
import pytest

import flare_pp_gb300 as fg
from flare_pp_gb300 import synth
from oracle.b2 import B2 as OB2
from oracle.b2 import ClusterDescriptor as OCD
from oracle.geometry import Structure as OStructure
from oracle.kernel import NormalizedDotProduct as ONDP

pytestmark = pytest.mark.gpu

RC = 4.5


def frames(ns, seed):
    """Cells of 4, 16 and 24 atoms, and a dimer with an atom out of its reach."""
    rng = np.random.default_rng(seed)
    out = [synth.rattled(synth.FCC_BASIS, 4.05, reps, 0.1, rng, n_species=ns)
           for reps in ((1, 1, 1), (2, 2, 1), (1, 2, 3))]
    out.append((np.eye(3) * 30.0, np.array([0, ns - 1, 0], np.int32),
                np.array([[1.0, 1.0, 1.0], [2.9, 2.2, 1.4], [16.0, 15.0, 14.0]])))
    return out


# labels of the frames: energy, forces of these atoms (None: all, (): none), stress
LABELS = [(1, None, 1), (0, (0, 3, 4, 11), 0), (1, (), 1), (1, None, 1)]


def gp_of(ns, N, lmax, power, n_sparse, cutoff="quadratic"):
    b = fg.B2("chebyshev", cutoff, [0, RC], [], [ns, N, lmax])
    gp = fg.SparseGP([fg.NormalizedDotProduct(1.7, power)], 0.001, 0.05, 0.006)
    cells = frames(ns, 12)
    for (cell, sp, pos), (e, f, s) in zip(cells, LABELS):
        st = fg.Structure(cell, sp, pos, RC, [b])
        n = len(sp)
        st.energy = np.zeros(1 if e else 0)
        st.forces = np.zeros(0 if f == () else 3 * n)
        st.stresses = np.zeros(6 if s else 0)
        gp.add_training_structure(st, (-1,) if not f else f)
    left = n_sparse
    for k, (_, sp, _) in enumerate(cells[:3]):
        m = min(left, len(sp))
        if m:
            gp.add_specific_environments(gp.training_structures[k], list(range(m)))
        left -= m
    assert left == 0
    return gp, cells


@pytest.mark.parametrize("ns,N,lmax,power,n_sparse,cutoff", [
    (1, 8, 3, 2, 33, "quadratic"),   # one sparse environment past a tile
    (1, 3, 2, 1, 32, "cosine"),
    (2, 5, 3, 2, 44, "quadratic"),
    (2, 16, 0, 2, 40, "quadratic"),  # the most channels, one degree
    (3, 4, 1, 3, 44, "quadratic"),
    (1, 1, 4, 2, 31, "cosine"),      # one channel
    (2, 2, 5, 2, 44, "quadratic"),   # past the unrolled degrees
])
def test_kuf_matches_oracle(gpu_lib, ns, N, lmax, power, n_sparse, cutoff):
    gp, cells = gp_of(ns, N, lmax, power, n_sparse, cutoff)
    sd = gp.sparse_descriptors[0]
    got = gp._kuf_batched(sd, gp.kernels[0])
    osd = OCD()
    osd.initialize_cluster(sd.n_types, sd.n_descriptors)
    osd.descriptors = [np.array(d) for d in sd.descriptors]
    osd.descriptor_norms = [np.array(n) for n in sd.descriptor_norms]
    osd.n_clusters_by_type = list(sd.n_clusters_by_type)
    osd.cumulative_type_count = list(sd.cumulative_type_count)
    osd.n_clusters = sd.n_clusters
    ob = OB2("chebyshev", cutoff, [0, RC], [], [ns, N, lmax])
    want = []
    for (cell, sp, pos), (e, f, s) in zip(cells, LABELS):
        os_ = OStructure(cell, sp, pos, RC, [ob])
        K = ONDP(1.7, power).envs_struc(osd, os_.descriptors[0])
        n = len(sp)
        cols = [0] if e else []
        for a in (range(n) if f is None else f):
            cols += [1 + 3 * a, 2 + 3 * a, 3 + 3 * a]
        if s:
            cols += list(range(1 + 3 * n, 7 + 3 * n))
        want.append(K[:, cols])
    want = np.hstack(want)
    np.testing.assert_allclose(got, want, rtol=0, atol=1e-10 * np.abs(want).max())
    # its sums run in a fixed order
    assert (gp._kuf_batched(sd, gp.kernels[0]) == got).all()


def test_kuf_few_sparse(gpu_lib):
    """Nine environments of a species go by the adjoint form, ten by the GEMM."""
    few, _ = gp_of(1, 6, 3, 2, 9)
    more, _ = gp_of(1, 6, 3, 2, 10)
    a = few._kuf_batched(few.sparse_descriptors[0], few.kernels[0])
    b = more._kuf_batched(more.sparse_descriptors[0], more.kernels[0])
    np.testing.assert_allclose(b[:9], a, rtol=0, atol=1e-10 * np.abs(a).max())
