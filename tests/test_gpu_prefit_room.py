"""The mixed path's prefit with little memory for its operand digits: it works in
smaller parts and gives the same bits, or reports that memory ran out and
leaves the engine usable."""
import numpy as np
import pytest

from chem_gb300.fock import JKEngine
from chem_gb300.layout import build_layout

pytestmark = pytest.mark.gpu


def _system(bsizes, naux, dense_to_panels):
    rng = np.random.default_rng(naux)
    lay = build_layout(bsizes, [naux], lambda i, j: np.array([j - i <= 1]))
    n = lay.nbf
    T = rng.standard_normal((naux, n, n)) * 2.0 ** rng.integers(-12, 3, (naux, 1, 1))
    B, _ = dense_to_panels(lay, T + T.transpose(0, 2, 1))
    L = np.tril(rng.standard_normal((naux, naux)))
    P = rng.standard_normal((n, n))
    return lay, B, L, P + P.T, rng.standard_normal((n, 2))


@pytest.mark.parametrize("naux", [47, 97, 257])
def test_parts_give_the_same_bits(naux, dense_to_panels):
    lay, B, L, P, C = _system([9, 40, 14, 30, 1], naux, dense_to_panels)
    part = -(-naux // 32) * 24576  # digits of 48 rows of L^-1
    ref = None
    for room in (-1, 0, part, 2 * part, 5 * part):
        eng = JKEngine(lay, B, L, L.T @ L, precision="split")
        eng.test_prefit_room(room)
        J, K = eng.compute_jk(P, C)
        eng.close()
        if ref is None:
            ref = J, K
        assert np.array_equal(J, ref[0]) and np.array_equal(K, ref[1])


def test_too_little_for_one_part(dense_to_panels):
    lay, B, L, P, C = _system([1], 257, dense_to_panels)
    eng = JKEngine(lay, B, L, L.T @ L, precision="split")
    ref = eng.compute_jk(P, C)
    eng.close()
    eng = JKEngine(lay, B, L, L.T @ L, precision="split")
    eng.test_prefit_room(0)
    with pytest.raises(RuntimeError, match="OOM|memory"):
        eng.compute_jk(P, C)
    eng.test_prefit_room(-1)
    J, K = eng.compute_jk(P, C)
    eng.close()
    assert np.array_equal(J, ref[0]) and np.array_equal(K, ref[1])
