"""The real-arithmetic mixed B3 form (lmax 1..3) against the FP64 form, at the
edges of its blocks: one radial channel, blocks filled in part, atoms whose pairs
take two rounds of a block's threads, two species, empty environments, and the same
evaluated twice (its sums run in a fixed order).

Tolerances are the mixed form's gates on |E| ~ 1 eV per atom, 1e-6 eV per atom and
1e-4 eV/A: FP32 descriptors (2^-24 relative per operation) and the split-fp16
contraction."""
import numpy as np
import pytest

import flare_pp_gb300 as fg
from flare_pp_gb300 import synth

pytestmark = pytest.mark.gpu


def model(ns, N, lmax, rc, seed):
    b = fg.B3("chebyshev", "quadratic", [0, rc], [], [ns, N, lmax])
    b.store_dervs = False
    cell, sp, pos = synth.rattled(synth.FCC_BASIS, 4.05, (2, 2, 2), 0.1,
                                  np.random.default_rng(seed), n_species=ns)
    s = fg.Structure(cell, sp, pos, rc, [b])
    cd = fg.ClusterDescriptor(s.descriptors[0])
    cd.descriptor_calculator = b
    rng = np.random.default_rng(seed + 1)
    alpha = rng.uniform(-1, 2, size=cd.n_clusters) / cd.n_clusters
    gp = fg.SparseGP([fg.NormalizedDotProduct(2.0, 2)], 0.01, 0.05, 0.006)
    gp.set_model(b, cd, alpha)
    return gp


@pytest.mark.parametrize("ns,N,lmax,reps,rc", [
    (1, 6, 3, (3, 3, 3), 5.0),      # 108 atoms, six to a block
    (1, 6, 3, (1, 1, 1), 4.2),      # 4 atoms: one block, filled in part
    (1, 5, 3, (2, 2, 3), 5.0),      # 35 triples: columns padded to a multiple of four
    (1, 1, 3, (2, 2, 2), 5.0),      # one channel: 128 atoms to a block
    (2, 3, 3, (2, 2, 2), 4.5),
    (3, 2, 2, (2, 3, 2), 4.5),
    (1, 4, 1, (2, 2, 2), 4.5),
    (1, 16, 1, (2, 2, 2), 4.5),     # 136 pairs: two rounds of 128 threads
])
def test_mixed_matches_fp64(gpu_lib, ns, N, lmax, reps, rc):
    gp = model(ns, N, lmax, rc, 71)
    cell, sp, pos = synth.rattled(synth.FCC_BASIS, 4.05, reps, 0.08, np.random.default_rng(5),
                                  n_species=ns)
    st = fg.Structure(cell, sp, pos, rc)
    n = len(sp)
    e64, f64, s64 = gp.predict_mapped(st, "fp64")
    e, f, s, ae = gp.predict_mapped(st, "mixed", atom_energies=True)
    assert abs(e - e64) / n < 1e-6
    assert np.abs(f - f64).max() < 1e-4
    assert np.abs(s - s64).max() < 1e-6
    assert abs(ae.sum() - e) < 1e-9 * max(1.0, abs(e))
    e2, f2, s2 = gp.predict_mapped(st, "mixed")
    assert e2 == e and (f2 == f).all() and (s2 == s).all()


def test_empty_environments(gpu_lib):
    """Atoms without neighbors have no energy and no force in either form."""
    gp = model(1, 6, 3, 4.0, 73)
    cell = np.diag([30.0, 30.0, 30.0])
    pos = np.array([[1.0, 1, 1], [15, 15, 15], [15, 15, 17.2], [25, 3, 9]])
    st = fg.Structure(cell, [0] * 4, pos, 4.0)
    e64, f64, _ = gp.predict_mapped(st, "fp64")
    e, f, s, ae = gp.predict_mapped(st, "mixed", atom_energies=True)
    assert ae[0] == 0 and ae[3] == 0 and (f[[0, 3]] == 0).all()
    assert abs(e - e64) / 4 < 1e-6 and np.abs(f - f64).max() < 1e-4
