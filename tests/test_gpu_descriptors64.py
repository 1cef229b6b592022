"""FP64 descriptors and stored derivatives at the edges of their kernels: a species'
sums dealt to the lanes in one and two passes, lmax past the unrolled degrees, one
channel, pairs outside their species' cutoff (the window is filled from those inside),
environments of more than one window, and atoms without a neighbor of a species; and
the per-structure sums of a batch around the length of a run of pairs.

Tolerances: sums of at most 150 products in FP64 with chunked compensated sums,
products of at most 17 of them: 1e-12 of the largest entry.  The batch's sums against
the single evaluations: 20,000 terms in another order, 20,000 * 2^-53 = 2e-12 relative
to the sum of magnitudes, 1e-10 of the largest virial (mixed: of FP32 pair forces that
are the same in both, summed in float-float by one and in FP64 by the other, 1e-7)."""
import numpy as np
import pytest

import flare_pp_gb300 as fg
from flare_pp_gb300 import synth
from oracle.b2 import B2 as OB2
from oracle.geometry import Structure as OStructure

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,N,lmax,rc,cutoff", [
    (1, 8, 3, 5.0, "quadratic"),
    (2, 16, 4, 5.4, "cosine"),      # 400 sums of a species: two passes of the lanes
    (2, 7, 3, 6.2, "quadratic"),    # 90 neighbors: three windows
    (3, 3, 2, 5.0, "quadratic"),
    (2, 4, 5, 4.6, "quadratic"),    # past the unrolled degrees
    (1, 1, 0, 4.2, "cosine"),
])
def test_descriptors_and_derivatives(gpu_lib, ns, N, lmax, rc, cutoff):
    rng = np.random.default_rng(31)
    cell, sp, pos = synth.rattled(synth.FCC_BASIS, 4.05, (2, 2, 2), 0.1, rng, n_species=ns)
    if ns == 3:
        sp = np.where(sp == 2, 0, sp)  # a species that no atom has
    # species pairs with shorter cutoffs than the list's, not symmetric
    cut = rc - 0.9 * rng.uniform(size=(ns, ns)) * (ns > 1)
    cut[0, 0] = rc
    ob = OB2("chebyshev", cutoff, [0, rc], [], [ns, N, lmax], cut)
    gb = fg.B2("chebyshev", cutoff, [0, rc], [], [ns, N, lmax], cut)
    want = OStructure(cell, sp, pos, rc, [ob]).descriptors[0]
    got = fg.Structure(cell, sp, pos, rc, [gb]).descriptors[0]
    for s in range(ns):
        assert list(got.neighbor_counts[s]) == list(want.neighbor_counts[s])
        for name in ("descriptors", "descriptor_norms", "descriptor_force_dervs",
                     "descriptor_force_dots"):
            g, w = np.asarray(getattr(got, name)[s]), np.asarray(getattr(want, name)[s])
            assert g.shape == w.shape
            if w.size:
                np.testing.assert_allclose(g, w, rtol=0, atol=1e-12 * np.abs(w).max())


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_batch_sums(gpu_lib, precision):
    rng = np.random.default_rng(8)
    b = fg.B2("chebyshev", "quadratic", [0, 5.0], [], [2, 4, 2])
    b.store_dervs = False
    cells = [synth.rattled(synth.FCC_BASIS, 4.05, reps, 0.1, rng, n_species=2)
             for reps in ((1, 1, 1), (3, 3, 3), (2, 3, 4), (4, 4, 4), (1, 2, 2))]
    # 96 atoms of 42 neighbors fill a run of 4096 pairs up to its last 64; the largest
    # takes three; two atoms out of reach have none
    cells.append((np.eye(3) * 30.0, np.array([0, 1], np.int32),
                  np.array([[1.0, 1.0, 1.0], [16.0, 15.0, 14.0]])))
    strucs = [fg.Structure(c, s, p, 5.0, [b] if k == 0 else []) for k, (c, s, p)
              in enumerate(cells)]
    cd = fg.ClusterDescriptor(strucs[0].descriptors[0])
    cd.descriptor_calculator = b
    gp = fg.SparseGP([fg.NormalizedDotProduct(2.0, 2)], 0.01, 0.05, 0.006)
    gp.set_model(b, cd, rng.uniform(-1, 2, size=cd.n_clusters))
    single = [gp.predict_mapped(s, precision) for s in strucs]
    for _ in range(2):  # the second evaluation packs FP64 geometry near the cutoffs only
        e, f, s = gp.predict_mapped_batched(strucs, precision)
        scale = max(np.abs(x[2]).max() for x in single)
        tol = 1e-10 if precision == "fp64" else 1e-7
        for k, (e1, f1, s1) in enumerate(single):
            assert abs(e[k] - e1) <= 1e-10 * max(1.0, abs(e1))
            np.testing.assert_allclose(f[k], f1, rtol=0, atol=1e-9 * np.abs(single[3][1]).max())
            np.testing.assert_allclose(s[k], s1, rtol=0, atol=tol * scale)
