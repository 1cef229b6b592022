"""FP64 descriptors and stored derivatives at the edges of their kernels: a species'
sums dealt to the lanes in one and two passes, lmax past the unrolled degrees, one
channel, pairs outside their species' cutoff (the window is filled from those inside),
environments of more than one window, and atoms without a neighbor of a species.

Tolerance: sums of at most 150 products in FP64 with chunked compensated sums,
products of at most 17 of them: 1e-12 of the largest entry."""
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
