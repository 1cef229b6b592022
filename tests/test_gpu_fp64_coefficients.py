"""FP64 mapped energies with coefficients that are large where descriptors are small (as a
fit to scaled descriptors gives them): beta_ij = b_ij / (s_i s_j), s the mean of each
normalised descriptor of a lattice whose small displacements make some of them 10^-9 of
the others.

The energies are compared with extended-precision sums over the call's own descriptors.
With x_i = |phat_i| / s_i and |b| <= 5, the digit planes of operands scaled to these x
err by at most 2^-54 of the row's largest entry each, in K products, and the powers of two
and the equilibration of b are within a factor of 16 of s: at most
16 * 5 * K 2^-53 max x sum x.  (Digits relative to the largest |phat_i| and |beta_ij| err by
up to 10^9 times as much.)  phat itself is p / |p|: 2^-52 of each product."""
import numpy as np
import pytest

import flare_pp_gb300 as fg
from flare_pp_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ns,kind", [(1, "dense"), (1, "diagonal"), (2, "dense"), (2, "mixed")])
def test_energy_of_scaled_coefficients(gpu_lib, ns, kind):
    rng = np.random.default_rng(31)
    b = fg.B2("chebyshev", "quadratic", [0, 5.0], [], [ns, 8 // ns, 3])
    b.store_dervs = False
    cell, sp, pos = synth.rattled(synth.FCC_BASIS, 4.05, (2, 2, 2), 1e-4, rng)
    sp = (np.arange(len(pos)) % ns).astype(np.int32)
    s = fg.Structure(cell, sp, pos, 5.0, [b])
    cd = fg.ClusterDescriptor(s.descriptors[0])
    cd.descriptor_calculator = b
    gp = fg.SparseGP([fg.NormalizedDotProduct(2.0, 2)], 0.01, 0.05, 0.006)
    gp.set_model(b, cd, np.ones(cd.n_clusters))
    gp.predict_mapped(s, "fp64")  # maps: the coefficients are replaced below
    nd = b.n_descriptors
    want, scale, packed = np.longdouble(0), 0.0, []
    for t in range(ns):
        p = np.asarray(s.descriptors[0].descriptors[t])
        phat = p / np.sqrt((p.astype(np.longdouble) ** 2).sum(1))[:, None]
        mean = np.abs(phat).mean(0)
        assert mean.min() > 0 and mean.max() / mean.min() > 1e6
        inv = (1.0 / mean).astype(np.float64)
        B = np.clip(rng.normal(size=(nd, nd)), -5, 5)
        if kind == "diagonal" or (kind == "mixed" and t == 0):
            B = np.diag(np.diag(B))
        B = np.triu(B) * np.outer(inv, inv)
        packed.append((np.triu(B, 1) * 2 + np.diag(np.diag(B)))[np.triu_indices(nd)])
        B = B + np.triu(B, 1).T
        want += (phat @ B.astype(np.longdouble) * phat).sum()
        x = (np.abs(phat) * inv).astype(np.float64)
        scale += (x.max(1) * x.sum(1)).sum()
    gp._model.set_beta(2, np.concatenate(packed))
    e = gp.predict_mapped(s, "fp64")[0]
    assert abs(float(e - want)) <= 16 * 5 * nd * 2.0 ** -53 * scale
