"""Integer half transforms: a row's exponent follows the columns that the row
has, however far below the others of its tile they lie.  Against dense FP64
products, with the bound relative to the norms of the rows."""
import numpy as np
import pytest

from chem_gb300.fock import JKEngine
from chem_gb300.layout import build_layout

pytestmark = pytest.mark.gpu

NAUX = 45


def _tensor(rng, n):
    T = rng.standard_normal((NAUX, n, n))
    return T + T.transpose(0, 2, 1)


def _layout():
    return build_layout([14, 5, 30, 9, 3], [NAUX], lambda i, j: np.array([j - i <= 3]))


def _half(D, C):
    """Rows H[mu] = (Y, i) of D C."""
    n = D.shape[1]
    return (D.reshape(-1, n) @ C).reshape(NAUX, n, -1).transpose(1, 0, 2).reshape(n, -1)


@pytest.mark.parametrize("su,sv", [(1e-16, 1.0), (1.0, 1e-16), (1e-25, 1.0), (1.0, 1e-25),
                                   (1e-25, 1e-25)])
@pytest.mark.parametrize("nocc", [1, 4, 31, 47, 49])
def test_small_vectors(nocc, su, sv, dense_to_panels):
    """The non-symmetric exchange is linear in either side: an odd number of
    vectors leaves a zero column after each side."""
    rng = np.random.default_rng(nocc)
    lay = _layout()
    B, D = dense_to_panels(lay, _tensor(rng, lay.nbf))
    U = su * rng.standard_normal((lay.nbf, nocc))
    Vt = sv * rng.standard_normal((nocc, lay.nbf))
    eng = JKEngine(lay, B, None, None, fitted=True, precision="split")
    K = eng.compute_k_lmo_asym(U, Vt)
    eng.close()
    Hu, Hv = _half(D, U), _half(D, Vt.T)
    # three operands of 39 bits below their rows' exponents
    bound = 2.0 ** -33 * np.outer(np.linalg.norm(Hu, axis=1), np.linalg.norm(Hv, axis=1))
    assert (np.abs(K + Hu @ Hv.T) <= bound).all()


@pytest.mark.parametrize("scale", [1e-3, 1e-16, 1e-25])
@pytest.mark.parametrize("nocc", [2, 33, 70])
@pytest.mark.parametrize("call", ["dfmo", "asym"])
def test_rows_without_the_large_columns(call, nocc, scale, dense_to_panels):
    """Functions whose integrals with the first orbital's functions are all
    zero: their rows hold the other orbitals alone, `scale` times as large."""
    rng = np.random.default_rng(nocc)
    lay = _layout()
    n = lay.nbf
    T = _tensor(rng, n)
    big, rows = np.arange(16, 20), np.array([3, 20, 47, 60])
    T[:, rows[:, None], big] = 0.0
    T[:, big[:, None], rows] = 0.0
    B, D = dense_to_panels(lay, T)
    C = scale * rng.standard_normal((n, nocc))
    C[:, 0] = 0.0
    C[big, 0] = rng.standard_normal(4)
    eng = JKEngine(lay, B, None, None, fitted=True, precision="split")
    K = eng.compute_jk(None, C)[1] if call == "dfmo" else eng.compute_k_lmo_asym(C, C.T.copy())
    eng.close()
    H = _half(D, C)
    norm = np.linalg.norm(H, axis=1)
    assert (np.abs(K + H @ H.T) <= 2.0 ** -33 * np.outer(norm, norm)).all()
