"""gbjk_get_split_fuse after a build says which digit cut the builds run: the
one in the epilogue takes all columns of a row in one 96-wide tile."""
import pytest

from chem_gb300.fock import JKEngine
from chem_gb300.synthetic import occupied, synthetic_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nocc,fused", [(30, True), (97, False)])
def test_get_split_fuse(nocc, fused):
    layout, decay = synthetic_layout(200, 230, seed=5)
    eng = JKEngine(layout, None, None, None, fitted=True, synthetic=(9, decay), precision="split")
    eng.set_split_fuse(True)
    assert eng.get_split_fuse()
    eng.compute_jk(None, occupied(200, nocc, seed=5))
    assert eng.get_split_fuse() == fused
    # the next plan is free to fuse again
    eng.compute_jk(None, occupied(200, 30, seed=5))
    assert eng.get_split_fuse()
    eng.set_split_fuse(False)
    assert not eng.get_split_fuse()
    eng.close()
