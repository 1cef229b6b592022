"""The neighbor build's one-block scan at its limit and the library's scan past it, and
energy_forces_stress with and without something watching the autograd graph: the same
numbers, and no_grad refused as the graph refuses it."""
import numpy as np
import pytest

import flare_pp_gb300 as fg
from flare_pp_gb300 import synth

pytestmark = pytest.mark.gpu

BCC = np.array([[0.0, 0.0, 0.0], [0.5, 0.5, 0.5]])


@pytest.mark.parametrize("reps", [(2, 2, 2), (16, 16, 16), (16, 16, 17)])  # 8,192: the limit
def test_neighbor_counts(gpu_lib, reps):
    """Every atom of the BCC lattice has 8 + 6 neighbors within 1.33 a."""
    cell, sp, pos = synth.rattled(BCC, 3.0, reps, 0.0, np.random.default_rng(0))
    s = fg.Structure(cell, sp, pos, 4.0)
    assert s.noa == 2 * int(np.prod(reps))
    assert (np.asarray(s.neighbor_count) == 14).all()


def test_energy_forces_stress_paths(gpu_lib):
    import torch
    from flare_pp_gb300.autograd import energy_forces_stress
    b = fg.B2("chebyshev", "quadratic", [0, 5.0], [], [1, 4, 2])
    b.store_dervs = False
    cell, sp, pos = synth.rattled(synth.FCC_BASIS, 4.05, (2, 2, 2), 0.1,
                                  np.random.default_rng(4))
    s = fg.Structure(cell, sp, pos, 5.0, [b])
    cd = fg.ClusterDescriptor(s.descriptors[0])
    cd.descriptor_calculator = b
    gp = fg.SparseGP([fg.NormalizedDotProduct(2.0, 2)], 0.01, 0.05, 0.006)
    gp.set_model(b, cd, np.random.default_rng(5).uniform(-1, 2, size=cd.n_clusters))
    x = torch.as_tensor(pos, device="cuda")
    for precision in ("fp64", "mixed"):
        plain = energy_forces_stress(gp, s, x, precision)
        seen = []
        with torch.autograd.graph.saved_tensors_hooks(lambda t: seen.append(1) or t,
                                                      lambda t: t):
            graph = energy_forces_stress(gp, s, x, precision)
        assert seen  # through the graph, where the hooks see the saved forces
        for p, g in zip(plain, graph):
            assert p.shape == g.shape and not p.requires_grad and (p == g).all()
        e, f, st = gp.predict_mapped(s, precision)
        assert plain[0].item() == e and (plain[1].cpu().numpy() == f).all()
        with torch.no_grad(), pytest.raises(RuntimeError):
            energy_forces_stress(gp, s, x, precision)
