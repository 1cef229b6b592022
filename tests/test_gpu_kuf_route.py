"""The count of sparse environments from which fpp_kuf_batched takes the GEMM form (its tile
is 32 environments, the adjoint form's at most 16), by descriptors and structures, and the
two forms' columns on both sides of it.

Tolerance: an entry is a sum over at most 50 pairs of products of K <= 1120 terms, each operand
within 2^-55 of its row's largest entry: 2^-55 * 1120 * 50 = 2e-12 of the largest product
a * dp * dhat, which is itself of the order of the largest kernel entry; 1e-10 of that."""
import ctypes

import numpy as np
import pytest

import flare_pp_gb300 as fg
from flare_pp_gb300 import synth
from flare_pp_gb300._lib import check, ptr
from flare_pp_gb300.api import _Model

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,lmax,n_structures,line", [
    (2, 2, 3, 64), (2, 2, 4, 24),      # 9 descriptors
    (3, 2, 3, 24), (3, 2, 4, 10),      # 18
    (8, 3, 3, 20), (8, 3, 4, 10),      # 144
    (15, 8, 3, 20), (15, 8, 4, 16),    # 1080
])
def test_line(gpu_lib, N, lmax, n_structures, line):
    rc = 4.0
    rng = np.random.default_rng(N)
    b = fg.B2("chebyshev", "quadratic", [0, rc], [], [1, N, lmax])
    frame = fg.Structure(*synth.rattled(synth.FCC_BASIS, 4.05, (4, 2, 2), 0.1, rng), rc, [b])
    strucs = [fg.Structure(*synth.rattled(synth.FCC_BASIS, 4.05, (1, 1, 1), 0.1, rng), rc)
              for _ in range(n_structures)]
    hs = (ctypes.c_void_p * n_structures)(*[s.handle for s in strucs])
    mask = np.full(n_structures, 7, np.int32)
    rows = np.asarray(frame.descriptors[0].descriptors[0])
    out = []
    for n in (line - 1, line):
        sd = fg.ClusterDescriptor()
        sd.initialize_cluster(1, b.n_descriptors)
        sd.descriptors[0], sd.descriptor_norms[0] = rows[:n], np.linalg.norm(rows[:n], axis=1)
        sd.cutoff_values[0] = np.ones(n)
        sd.n_clusters_by_type, sd.cumulative_type_count, sd.n_clusters = [n], [0], n
        model = _Model(b, 1.7, 2, sd)
        K = np.empty((n, n_structures * 19))
        check(gpu_lib.fpp_kuf_batched(model.handle, hs, n_structures, ptr(mask), None, None,
                                      ptr(K), K.shape[1], None))
        ks, threads = ctypes.c_int32(), ctypes.c_int32()
        check(gpu_lib.fpp_model_kuf_tiles(model.handle, ctypes.byref(ks), ctypes.byref(threads),
                                          None, None))
        assert (ks.value == 32) == (n == line), (n, ks.value)
        out.append(K)
    np.testing.assert_allclose(out[1][:-1], out[0], rtol=0, atol=1e-10 * np.abs(out[0]).max())
