"""The mixed path's prefit under a rescaled auxiliary basis: function Y taken
2^s_Y times as large multiplies the tensor's row Y and divides the column Y of
L^-1, and leaves L^-1 B, J and K as they are."""
import numpy as np
import pytest

from chem_gb300.fock import JKEngine
from chem_gb300.layout import build_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spread", [4, 20, 60])
@pytest.mark.parametrize("naux", [5, 48, 130, 257])
def test_auxiliary_scale(naux, spread, dense_to_panels):
    rng = np.random.default_rng(naux + spread)
    lay = build_layout([3, 9, 30, 5], [naux], lambda i, j: np.array([j - i <= 1]))
    n = lay.nbf
    T = rng.standard_normal((naux, n, n))
    B, D = dense_to_panels(lay, T + T.transpose(0, 2, 1))
    L = np.tril(rng.standard_normal((naux, naux)))
    L[np.diag_indices(naux)] += 3.0
    s = 2.0 ** rng.integers(-spread, spread + 1, naux)
    Bs = dense_to_panels(lay, D * s[:, None, None])[0]
    C = np.linalg.qr(rng.standard_normal((n, 3)))[0]
    P = rng.standard_normal((n, n))
    P = P + P.T
    out = []
    for b, linv in ((B, L), (Bs, L / s)):
        eng = JKEngine(lay, b, linv, linv.T @ linv, precision="split")
        out.append(eng.compute_jk(P, C))
        eng.close()
    F = np.einsum("xy,ymn->xmn", L, D)
    H = np.einsum("xmn,ni->mxi", F, C).reshape(n, -1)
    Jr = np.einsum("xmn,x->mn", F, np.einsum("xmn,mn->x", F, P))
    A = np.einsum("xmn,x->mn", np.abs(F), np.einsum("xmn,mn->x", np.abs(F), np.abs(P)))
    for J, K in out:
        # 39-bit operands below the rows' exponents
        assert np.abs(K + H @ H.T).max() <= 2.0 ** -33 * np.linalg.norm(H, axis=1).max() ** 2
        assert np.abs(J - Jr).max() <= 2.0 ** -36 * A.max()
    # powers of two change no digit
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
