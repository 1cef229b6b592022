"""Device memory that a model keeps between calls: below the limit it stays (the next call
finds it), above it is given back, and the results are the same."""
import numpy as np
import pytest

import flare_pp_gb300 as fg
from flare_pp_gb300 import synth
from flare_pp_gb300._lib import check, ptr

pytestmark = pytest.mark.gpu

MB = 1 << 20


def test_given_back_above_the_limit(gpu_lib):
    import torch
    rc = 3.2
    b = fg.B2("chebyshev", "quadratic", [0, rc], [], [1, 4, 2])
    b.store_dervs = False
    rng = np.random.default_rng(8)
    bcc = np.array([[0.0, 0.0, 0.0], [0.5, 0.5, 0.5]])
    cd = fg.ClusterDescriptor(fg.Structure(*synth.rattled(bcc, 3.0, (6, 6, 6), 0.1, rng), rc,
                                           [b]).descriptors[0])
    n = cd.n_clusters
    gp = fg.SparseGP([fg.NormalizedDotProduct(2.0, 2)], 0.01, 0.05, 0.006)
    gp.set_model(b, cd, rng.uniform(0.5, 1.5, size=n), R_inv=0.1 * np.eye(n),
                 L_inv=0.05 * np.eye(n))
    s = fg.Structure(*synth.rattled(bcc, 3.0, (16, 16, 8), 0.1, rng), rc)

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    def sor():
        gp.predict_SOR(s)
        return s.mean_efs.copy(), s.variance_efs.copy()

    def mean():
        gp.predict_mean(s)
        return (s.mean_efs.copy(),)

    def uncert():
        return gp.predict_energy_uncertainty(s)

    def envs():
        K = np.empty((n, 1 + 3 * s.noa + 6))
        check(gpu_lib.fpp_envs_struc(gp._model.handle, s.handle, ptr(K), None))
        return (K,)

    # bytes of the kernel matrix of the structure, and of its atoms
    k_struc, k_atoms = 8 * n * (3 * s.noa + 7), 8 * n * s.noa
    assert k_atoms > 13 * MB
    for call, held in ((sor, 3 * k_struc), (envs, k_struc), (mean, k_atoms),
                       (uncert, 2 * k_atoms)):
        check(gpu_lib.fpp_model_set_workspace_limits(gp._model.handle, 0, 0, 0))
        want = call()
        f0 = free()
        got = call()
        assert free() == f0  # kept, and enough for the same call
        check(gpu_lib.fpp_model_set_workspace_limits(gp._model.handle, 0, 0, 1))
        again = call()
        assert free() - f0 >= held, (call.__name__, free() - f0, held)
        for w, g, a in zip(want, got, again):
            assert (np.asarray(w) == g).all() and (np.asarray(w) == a).all()


@pytest.mark.parametrize("ns", [1, 3])
def test_fp64_contraction_in_blocks(gpu_lib, ns):
    """Rows of phat in blocks of 128 and of 1,024: less memory, the same bits (each row's
    products are exact integer sums)."""
    import torch
    rc = 4.0
    b = fg.B2("chebyshev", "quadratic", [0, rc], [], [ns, 8 // ns, 3])
    b.store_dervs = False
    rng = np.random.default_rng(9)
    bcc = np.array([[0.0, 0.0, 0.0], [0.5, 0.5, 0.5]])
    cd = fg.ClusterDescriptor(fg.Structure(
        *synth.rattled(bcc, 3.0, (4, 4, 4), 0.1, rng, n_species=ns), rc, [b]).descriptors[0])
    gp = fg.SparseGP([fg.NormalizedDotProduct(2.0, 2)], 0.01, 0.05, 0.006)
    gp.set_model(b, cd, rng.uniform(0.5, 1.5, size=cd.n_clusters))
    frame = synth.rattled(bcc, 3.0, (16, 16, 13), 0.1, rng, n_species=ns)
    row = 16 * -(-b.n_descriptors // 64) * 64  # bytes of a row's planes
    want, used = None, []
    gp.predict_mapped(fg.Structure(*frame, rc), "fp64")  # the model's own buffers
    for keep in (0, row * 1024, 1):
        check(gpu_lib.fpp_model_set_workspace_limits(gp._model.handle, 0, 0, keep))
        s = fg.Structure(*frame, rc)
        torch.cuda.synchronize()
        f0 = torch.cuda.mem_get_info()[0]
        got = gp.predict_mapped(s, "fp64")
        torch.cuda.synchronize()
        used.append(f0 - torch.cuda.mem_get_info()[0])
        if want is None:
            want = got
        for w, g in zip(want, got):
            assert (np.asarray(w) == np.asarray(g)).all(), keep
    planes = row * len(frame[1])
    assert used[0] - used[1] >= planes // 2 and used[0] - used[2] >= planes // 2, (used, planes)
