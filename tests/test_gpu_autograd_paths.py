"""energy_forces_stress where the autograd graph does more than pass the forces on: anomaly
detection, positions that the graph refuses, and positions of another shape."""
import numpy as np
import pytest

import flare_pp_gb300 as fg
from flare_pp_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case(gpu_lib):
    import torch
    b = fg.B2("chebyshev", "quadratic", [0, 5.0], [], [1, 4, 2])
    b.store_dervs = False
    cell, sp, pos = synth.rattled(synth.FCC_BASIS, 4.05, (2, 2, 2), 0.1,
                                  np.random.default_rng(4))
    s = fg.Structure(cell, sp, pos, 5.0, [b])
    cd = fg.ClusterDescriptor(s.descriptors[0])
    cd.descriptor_calculator = b

    def model():
        gp = fg.SparseGP([fg.NormalizedDotProduct(2.0, 2)], 0.01, 0.05, 0.006)
        gp.set_model(b, cd, np.random.default_rng(5).uniform(-1, 2, size=cd.n_clusters))
        return gp
    return s, torch.as_tensor(pos, device="cuda"), model


@pytest.mark.filterwarnings("ignore:Error detected in")
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_anomaly_detection(case, precision):
    import torch
    from flare_pp_gb300.autograd import energy_forces_stress
    s, x, model = case
    gp = model()
    plain = energy_forces_stress(gp, s, x, precision)
    with torch.autograd.set_detect_anomaly(True):
        for p, g in zip(plain, energy_forces_stress(gp, s, x, precision)):
            assert (p == g).all()
    nd = gp._model.n_descriptors
    gp._model.set_beta(2, np.full(nd * (nd + 1) // 2, np.nan))
    assert torch.isnan(energy_forces_stress(gp, s, x, precision)[1]).all()
    with torch.autograd.set_detect_anomaly(True), pytest.raises(RuntimeError, match="nan"):
        energy_forces_stress(gp, s, x, precision)


def test_refused_positions(case):
    import torch
    from flare_pp_gb300.autograd import energy_forces_stress
    s, x, model = case
    gp = model()
    with torch.inference_mode():
        inference = x.clone()
    for bad in (x.flatten(), x.long(), inference):
        with pytest.raises(RuntimeError):
            energy_forces_stress(gp, s, bad, "fp64")
    for bad in (x.float(), x.cpu()):
        with pytest.raises(TypeError):
            energy_forces_stress(gp, s, bad, "fp64")


def test_other_forms(case):
    import torch
    from flare_pp_gb300.autograd import energy_forces_stress
    s, x, model = case
    gp = model()
    plain = energy_forces_stress(gp, s, x, "fp64")
    for same in (x.t().contiguous().t(), torch.nn.Parameter(x), x.clone().requires_grad_()):
        for p, g in zip(plain, energy_forces_stress(gp, s, same, "fp64")):
            assert p.shape == g.shape and not g.requires_grad and (p == g).all()
