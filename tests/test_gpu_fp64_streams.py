"""FP64 J on the side stream beside K: the bits of the phases in order, whole
and in batches, and a K plan that cannot be had leaves the engine as it was."""
import numpy as np
import pytest

from chem_gb300.fock import JKEngine
from chem_gb300.layout import build_layout
from chem_gb300.synthetic import occupied, synthetic_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [None, "aux", "occ"])
def test_beside_is_in_order(batch, water):
    rng = np.random.default_rng(11)
    if batch == "aux":
        layout, decay = synthetic_layout(60, 130, seed=5)
        eng = JKEngine(layout, None, None, None, fitted=True, synthetic=(9, decay), aux_batch=64)
        C = occupied(60, 7, seed=5)
    else:
        eng = JKEngine(water.layout, water.B, np.tril(water.Linv), water.Vinv, eps=1e-10)
        C = np.linalg.qr(rng.standard_normal((water.nbf, 5)))[0]
        if batch == "occ":
            eng.set_occ_batch(2)
    P = [rng.standard_normal((eng.nbf, eng.nbf)) for _ in range(3)]
    P = [p + p.T for p in P]
    eng.set_overlap(-1)
    ref = [eng.compute_jk(p, C) for p in P]
    eng.set_overlap(0)
    # direct launches, then the replayed graph, a new density each time
    for _ in range(4):
        for p, (J, K) in zip(P, ref):
            J1, K1 = eng.compute_jk(p, C)
            assert np.array_equal(J, J1) and np.array_equal(K, K1)
    eng.close()


def test_plan_without_memory():
    """The half transform of one batch would take more than the device has (32
    functions, 25568 auxiliary rows, 47000 orbitals: 308 GB), so the build
    reports it; J before and after are the same."""
    layout = build_layout([32], [25600], lambda i, j: np.array([True]))
    eng = JKEngine(layout, None, None, None, fitted=True, synthetic=(3, 0.1), aux_batch=25568)
    P = np.random.default_rng(2).standard_normal((32, 32))
    P = P + P.T
    J = eng.compute_jk(P)[0]
    held = eng.device_bytes
    with pytest.raises(RuntimeError, match="OOM|memory"):
        eng.compute_jk(2 * P, np.ones((32, 47000)))
    for _ in range(2):
        assert np.array_equal(eng.compute_jk(P)[0], J)
    assert eng.device_bytes < held + (1 << 30)
    J4, K4 = eng.compute_jk(P, np.ones((32, 4)))
    assert np.array_equal(J4, J) and K4.shape == (32, 32)
    eng.close()
