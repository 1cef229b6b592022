"""Kuf of descriptor shapes whose derivative rows fill a block's shared memory to within
its static part (384 bytes): against the oracle.

Tolerance: an entry is a sum over at most 30 pairs of products of K <= 8127 terms, each
operand within 2^-55 of its row's largest entry: 2^-55 * 8127 * 30 = 7e-12 of the largest
product a * dp * dhat, which is itself of the order of the largest kernel entry; 1e-10 of
that."""
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


# eight, four warps of a block at the limit
@pytest.mark.parametrize("ns,N,lmax", [(7, 6, 5), (7, 6, 8)])
def test_full_block(gpu_lib, ns, N, lmax):
    rc = 3.5
    b = fg.B2("chebyshev", "quadratic", [0, rc], [], [ns, N, lmax])
    cell, _, pos = synth.rattled(synth.FCC_BASIS, 4.05, (1, 1, 1), 0.1,
                                 np.random.default_rng(2))
    sp = np.array([0, 2, 6, 2], np.int32)
    s = fg.Structure(cell, sp, pos, rc, [b])
    sd = s.descriptors[0]
    model = _Model(b, 1.3, 2, sd)
    K = np.full((sd.n_clusters, 1 + 3 * 4 + 6), 7.0)
    check(gpu_lib.fpp_envs_struc(model.handle, s.handle, ptr(K), None))
    od = OStructure(cell, sp, pos, rc, [OB2("chebyshev", "quadratic", [0, rc], [],
                                            [ns, N, lmax])]).descriptors[0]
    oc = OCD()
    oc.initialize_cluster(ns, b.n_descriptors)
    oc.descriptors = [np.array(d) for d in sd.descriptors]
    oc.descriptor_norms = [np.array(v) for v in sd.descriptor_norms]
    oc.n_clusters_by_type = list(sd.n_clusters_by_type)
    oc.cumulative_type_count = list(sd.cumulative_type_count)[:ns]
    oc.n_clusters = sd.n_clusters
    want = ONDP(1.3, 2).envs_struc(oc, od)
    np.testing.assert_allclose(K, want, rtol=0, atol=1e-10 * np.abs(want).max())
