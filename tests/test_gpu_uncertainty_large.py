"""predict_energy_uncertainty of more atoms of one species than 65,535 chunks of 64: a
perfect BCC lattice, every atom as in the cell of 128.

Tolerances: coordinates of up to 384 A round to 2^-45, 1e-14 of a distance, which a radial
function of two channels and its square take to about 1e-12 of a descriptor; 4.2 million
energies summed in FP64 err by at most (64 + 65,536) 2^-53 = 7e-12 of the sum.  1e-10 of the
energy, twice that of its square, and 1e-10 of sigma^2 per atom."""
import numpy as np
import pytest

import flare_pp_gb300 as fg
from flare_pp_gb300 import synth

pytestmark = pytest.mark.gpu

BCC = np.array([[0.0, 0.0, 0.0], [0.5, 0.5, 0.5]])


def test_more_than_65535_chunks(gpu_lib):
    rc = 3.2
    b = fg.B2("chebyshev", "quadratic", [0, rc], [], [1, 2, 1])
    rng = np.random.default_rng(3)
    frame = fg.Structure(*synth.rattled(BCC, 3.0, (3, 3, 3), 0.2, rng), rc, [b])
    cd = fg.ClusterDescriptor(frame.descriptors[0])
    n = cd.n_clusters
    gp = fg.SparseGP([fg.NormalizedDotProduct(2.0, 2)], 0.01, 0.05, 0.006)
    gp.set_model(b, cd, rng.uniform(0.5, 1.5, size=n), R_inv=0.1 * np.eye(n),
                 L_inv=0.05 * np.eye(n))
    ref = None
    for reps in ((4, 4, 4), (128, 128, 128)):
        cell, sp, pos = synth.rattled(BCC, 3.0, reps, 0.0, rng)
        e, v, local = gp.predict_energy_uncertainty(fg.Structure(cell, sp, pos, rc))
        if ref is None:
            ref, small = (e, v, local[0]), len(sp)
    assert len(sp) == 64 * 65536
    k = len(sp) / small
    assert abs(e - k * ref[0]) <= 1e-10 * k * abs(ref[0])
    assert abs(v - k * k * ref[1]) <= 2e-10 * k * k * ref[1]
    np.testing.assert_allclose(local, ref[2], rtol=0, atol=1e-10 * 4.0)
