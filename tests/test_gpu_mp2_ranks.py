"""The MP2 batch's factors as they come in: ranks that differ from point to
point around the 32-row blocks of the operand images, a zero column, and a
second set through the buffers of the first.  Against dense FP64 products."""
import numpy as np
import pytest

from chem_gb300.fock import JKEngine
from chem_gb300.layout import build_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "split"])
@pytest.mark.parametrize("ranks", [[(1, 1)], [(33, 40), (1, 7), (8, 65)],
                                   [(31, 32), (32, 31), (3, 101), (33, 2)]])
def test_ranks(ranks, precision):
    rng = np.random.default_rng(400 + len(ranks))
    bsizes, naux = [14, 5, 30, 9, 40, 3], 35
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
    eng = JKEngine(lay, B, None, None, fitted=True, precision=precision)
    for call in range(2):
        Lo = [rng.standard_normal((n, r)) for r, _ in ranks]
        Lv = [rng.standard_normal((n, r)) for _, r in ranks]
        Lo[-1][:, 0] *= call  # zero the first time
        e, Z = eng.mp2_laplace(Lo, Lv, want_z=True)
        for t in range(len(ranks)):
            W = np.einsum("xmi,ma->xia", D @ Lo[t], Lv[t]).reshape(naux, -1)
            Wa = np.einsum("xmi,ma->xia", np.abs(D) @ np.abs(Lo[t]), np.abs(Lv[t])).reshape(naux, -1)
            Zr, Za = W @ W.T, Wa @ Wa.T
            # three chained products of 39-bit operands, each row's largest value a
            # few times its mean: 2^-32 of the sums of absolute values
            assert np.abs(Z[t] - Zr).max() <= 2.0 ** -32 * Za.max()
            assert abs(e[t] - (Zr * Zr).sum()) <= 2.0 ** -31 * (Za * Za).sum()
    eng.close()
