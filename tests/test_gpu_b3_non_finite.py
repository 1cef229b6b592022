"""Mixed B3 with an Inf or NaN coefficient (a potential file may hold any number) among those
of the triangles that the real form leaves out, or among the others: no finite
results, as in FP64."""
import numpy as np
import pytest

import flare_pp_gb300 as fg
from flare_pp_gb300 import synth

pytestmark = pytest.mark.gpu


def triangles(lmax):
    return [(a, b, c) for a in range(lmax + 1) for b in range(lmax + 1)
            for c in range(abs(a - b), min(lmax, a + b) + 1)]


@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("where", ["odd", "even"])
def test_non_finite_coefficient(gpu_lib, where, value):
    b = fg.B3("chebyshev", "quadratic", [0, 4.5], [], [1, 2, 2])
    b.store_dervs = False
    cell, sp, pos = synth.rattled(synth.FCC_BASIS, 4.05, (2, 2, 2), 0.1,
                                  np.random.default_rng(6))
    s = fg.Structure(cell, sp, pos, 4.5, [b])
    cd = fg.ClusterDescriptor(s.descriptors[0])
    cd.descriptor_calculator = b
    gp = fg.SparseGP([fg.NormalizedDotProduct(2.0, 2)], 0.01, 0.05, 0.006)
    gp.set_model(b, cd, np.ones(cd.n_clusters))
    gp.predict_mapped(s, "mixed")
    tri = triangles(2)
    nd = b.n_descriptors
    assert nd == 4 * len(tri)  # four radial triples of two channels
    d = next(k for k, t in enumerate(tri) if sum(t) % 2 == (where == "odd"))
    beta = np.random.default_rng(7).normal(size=nd * (nd + 1) // 2)
    gp._model.set_beta(2, beta)
    assert np.isfinite(gp.predict_mapped(s, "mixed")[1]).all()
    beta[d * nd - d * (d - 1) // 2] = value  # beta_dd of the packed upper triangle
    gp._model.set_beta(2, beta)
    for precision in ("fp64", "mixed"):
        e, f, st = gp.predict_mapped(s, precision)
        assert not (np.isfinite(e) or np.isfinite(f).any() or np.isfinite(st).any()), precision
