"""The neighbor build's one-block scan at its limit and the library's scan past it."""
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
