"""The fused digit cut next to the edge of the 96-wide column tile: occupied
counts that, with the density columns, need one tile or two.  Against the
unfused exchange, and every repetition the same bits."""
import numpy as np
import pytest

from chem_gb300.fock import JKEngine
from chem_gb300.synthetic import occupied, synthetic_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nocc", [30, 56, 57, 96, 97, 130])
def test_fused_exchange(nocc):
    layout, decay = synthetic_layout(200, 230, seed=5)
    C = occupied(200, nocc, seed=5)
    K = {}
    for fuse in (False, True):
        eng = JKEngine(layout, None, None, None, fitted=True, synthetic=(9, decay),
                       precision="split")
        eng.set_split_fuse(fuse)
        K[fuse] = [eng.compute_jk(None, C)[1] for _ in range(3)]
        eng.close()
        assert all(np.array_equal(K[fuse][0], k) for k in K[fuse])
    scale = np.abs(K[False][0]).max()
    # both keep 39 bits of every row (or row segment) of the two factors
    assert np.abs(K[True][0] - K[False][0]).max() <= 2.0 ** -34 * scale
