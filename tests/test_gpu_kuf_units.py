"""Kuf by one GEMM in several chunks of structures, in a unit per species of a structure
that exceeds the limit, and in several slices, with species that have no sparse
environments and structures with some of the labels: against the oracle, and the same
bits whatever the limits (every product is an exact integer sum, every other sum runs
per atom or per structure).

Tolerance against the oracle: an entry is a sum over at most 100 pairs of products of
K <= 300 terms, each operand within 2^-55 of its row's largest entry: 2^-55 * 300 * 100 =
9e-13 of the largest product a * dp * dhat, which is itself of the order of the largest
kernel entry; 1e-10 of that."""
import ctypes

import numpy as np
import pytest

import flare_pp_gb300 as fg
from flare_pp_gb300 import synth
from flare_pp_gb300._lib import check, ptr
from flare_pp_gb300.api import _Model
from oracle.b2 import B2 as OB2
from oracle.b2 import ClusterDescriptor as OCD
from oracle.geometry import Structure as OStructure
from oracle.kernel import NormalizedDotProduct as ONDP

pytestmark = pytest.mark.gpu

RC, SIGMA = 4.5, 1.7


def case(ns, with_sparse):
    """Frames of 16, 24, 4 and 8 atoms; 12 sparse environments of each species listed."""
    rng = np.random.default_rng(21)
    b = fg.B2("chebyshev", "quadratic", [0, RC], [], [ns, 5, 3])
    cells = [synth.rattled(synth.FCC_BASIS, 4.05, reps, 0.1, rng, n_species=ns)
             for reps in ((2, 2, 1), (1, 2, 3), (1, 1, 1), (2, 1, 1))]
    strucs = [fg.Structure(c, s, p, RC, [b]) for c, s, p in cells]
    sd = fg.ClusterDescriptor()
    sd.initialize_cluster(ns, b.n_descriptors)
    for t in range(ns):
        rows = np.concatenate([st.descriptors[0].descriptors[t] for st in strucs[:2]])
        k = 12 if t in with_sparse else 0
        sd.descriptors[t] = rows[:k]
        assert len(sd.descriptors[t]) == k
        sd.descriptor_norms[t] = np.linalg.norm(rows[:k], axis=1)
        sd.cutoff_values[t] = np.ones(k)
        sd.n_clusters_by_type[t] = k
    sd.cumulative_type_count = [int(v) for v in
                                np.cumsum([0] + list(sd.n_clusters_by_type))[:ns]]
    sd.n_clusters = sum(sd.n_clusters_by_type)
    return b, cells, strucs, sd


MASKS = [7, 2, 5, 7]


def kuf(lib, model, strucs, rows):
    n = sum((m & 1) + (3 * s.noa if m & 2 else 0) + (6 if m & 4 else 0)
            for s, m in zip(strucs, MASKS))
    out = np.full((rows, n), 7.0)
    hs = (ctypes.c_void_p * len(strucs))(*[s.handle for s in strucs])
    mask = np.array(MASKS, np.int32)
    check(lib.fpp_kuf_batched(model.handle, hs, len(strucs), ptr(mask), None, None, ptr(out),
                              n, None))
    return out


@pytest.mark.parametrize("ns,with_sparse", [(2, (0, 1)), (2, (1,)), (2, (0,)), (3, (1, 2)),
                                            (3, (2,))])
def test_limits(gpu_lib, ns, with_sparse):
    b, cells, strucs, sd = case(ns, with_sparse)
    ob = OB2("chebyshev", "quadratic", [0, RC], [], [ns, 5, 3])
    osd = OCD()
    osd.initialize_cluster(ns, b.n_descriptors)
    osd.descriptors = [np.array(d) for d in sd.descriptors]
    osd.descriptor_norms = [np.array(v) for v in sd.descriptor_norms]
    osd.n_clusters_by_type = list(sd.n_clusters_by_type)
    osd.cumulative_type_count = list(sd.cumulative_type_count)
    osd.n_clusters = sd.n_clusters
    full = [ONDP(SIGMA, 2).envs_struc(osd, OStructure(c, s, p, RC, [ob]).descriptors[0])
            for c, s, p in cells]
    want = np.hstack([
        K[:, ([0] if m & 1 else []) + (list(range(1, 1 + 3 * s.noa)) if m & 2 else []) +
          (list(range(1 + 3 * s.noa, 7 + 3 * s.noa)) if m & 4 else [])]
        for K, s, m in zip(full, strucs, MASKS)])
    tol = 1e-10 * np.abs(want).max()
    whole = None
    # the defaults; a structure per chunk, species by species; chunks of some structures;
    # a structure per slice; both
    for chunk, pairs in ((0, 0), (1, 0), (3 << 20, 0), (0, 1), (1, 1)):
        model = _Model(b, SIGMA, 2, sd)
        check(gpu_lib.fpp_model_set_workspace_limits(model.handle, chunk, pairs, 0))
        got = kuf(gpu_lib, model, strucs, sd.n_clusters)
        np.testing.assert_allclose(got, want, rtol=0, atol=tol, err_msg=str((chunk, pairs)))
        if whole is None:
            whole = got
        assert (got == whole).all(), (chunk, pairs)
        for s, K in zip(strucs, full):  # a structure's full kernel matrix
            one = np.full(K.shape, 7.0)
            check(gpu_lib.fpp_envs_struc(model.handle, s.handle, ptr(one), None))
            np.testing.assert_allclose(one, K, rtol=0, atol=tol)
