"""Operand rows of the split builds, exponents and digits in one launch: orbital
counts around the 8-row groups that the coefficient and density rows share, a
zero orbital, panels of ragged widths, and the tensor's own rows in one batch
and in several.  Against dense FP64 products."""
import numpy as np
import pytest

from chem_gb300.fock import JKEngine
from chem_gb300.layout import build_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("aux_batch", [0, 32])
@pytest.mark.parametrize("nocc", [1, 7, 8, 9, 15, 32, 33])
def test_operand_rows(nocc, aux_batch):
    rng = np.random.default_rng(300 + nocc)
    bsizes, naux = [14, 5, 30, 9, 40, 3], 75
    lay = build_layout(bsizes, [naux], lambda i, j: np.array([j - i <= 3]))
    n, off = lay.nbf, lay.boff
    T = rng.standard_normal((naux, n, n))
    T = T + T.transpose(0, 2, 1)
    B, D = np.zeros(lay.nnz), np.zeros_like(T)
    for i, cols in enumerate(lay.column_map()):
        b, k, o = int(lay.bsizes[i]), len(cols), int(lay.panel_off[i])
        blk = T[:, off[i]:off[i + 1]][:, :, cols]
        B[o:o + b * naux * k] = blk.transpose(1, 0, 2).ravel()
        D[:, off[i]:off[i + 1], cols] = blk
    C = rng.standard_normal((n, nocc))
    if nocc > 1:
        C[:, nocc // 2] = 0.0
    P = rng.standard_normal((n, n))
    P = P + P.T
    eng = JKEngine(lay, B, None, None, fitted=True, precision="split", aux_batch=aux_batch)
    J, K = eng.compute_jk(P, C)
    _, K1 = eng.compute_jk(None, C)  # without density rows
    eng.close()
    H = (D.reshape(-1, n) @ C).reshape(naux, n, nocc).transpose(1, 0, 2).reshape(n, -1)
    # two operands of 39 bits below their rows' exponents, summed over rows of
    # up to 75 * 33 terms: 2^-34 of the row norms' product
    bound = 2.0 ** -34 * np.linalg.norm(H, axis=1).max() ** 2
    assert np.abs(K + H @ H.T).max() <= bound
    assert np.abs(K1 + H @ H.T).max() <= bound
    Jr = np.einsum("xmn,x->mn", D, np.einsum("xmn,mn->x", D, P))
    Ja = np.einsum("xmn,x->mn", np.abs(D), np.einsum("xmn,mn->x", np.abs(D), np.abs(P)))
    # 39 bits of each operand row, 40 of the tensor copy's elements
    assert np.abs(J - Jr).max() <= 2.0 ** -36 * Ja.max()
