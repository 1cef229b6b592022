"""Predictions of a model without sparse environments, in memory that holds something else:
zero mean and SOR variance (R_inv^T K has no rows)."""
import numpy as np
import pytest

import flare_pp_gb300 as fg
from flare_pp_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cls", ["B2", "B3"])
def test_zero_mean(gpu_lib, cls):
    import torch
    b = getattr(fg, cls)("chebyshev", "quadratic", [0, 4.0], [], [1, 2, 2])
    gp = fg.SparseGP([fg.NormalizedDotProduct(2.0, 2)], 0.01, 0.05, 0.006)
    cd = fg.ClusterDescriptor()
    cd.initialize_cluster(1, b.n_descriptors)
    cd.descriptors[0], cd.descriptor_norms[0] = np.zeros((0, b.n_descriptors)), np.zeros(0)
    cd.cutoff_values[0] = np.zeros(0)
    cd.n_clusters_by_type, cd.cumulative_type_count, cd.n_clusters = [0], [0], 0
    gp.set_model(b, cd, np.zeros(0), R_inv=np.zeros((0, 0)), L_inv=np.zeros((0, 0)))
    s = fg.Structure(*synth.rattled(synth.FCC_BASIS, 4.05, (2, 2, 2), 0.1,
                                    np.random.default_rng(1)), 4.0, [b])
    for size in (10, 14, 18, 22, 26):  # the sizes that device allocations are cut from
        held = [torch.full((1 << (size - 3),), 5.0, dtype=torch.float64, device="cuda")
                for _ in range(8)]
        torch.cuda.synchronize()
        del held
    torch.cuda.empty_cache()
    gp.predict_SOR(s)
    assert (s.mean_efs == 0).all()
    assert (s.variance_efs == 0).all()
    gp.predict_mean(s)
    assert (s.mean_efs == 0).all()
    gp.predict_SOR(s)
    assert (s.mean_efs == 0).all() and (s.variance_efs == 0).all()
