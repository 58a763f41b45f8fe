"""The non-symmetric exchange's half transform over the columns [u | v] of one
operand: vector counts around the 96-wide column tile and its halves, and
sides of very different scale (each keeps its own row exponents).  Against
dense FP64 products."""
import numpy as np
import pytest

from chem_gb300.fock import JKEngine
from chem_gb300.layout import build_layout

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [1.0, 1e-9])
@pytest.mark.parametrize("nocc", [1, 2, 17, 47, 48, 49, 95, 96, 97])
def test_column_tiles(nocc, scale):
    rng = np.random.default_rng(100 + nocc)
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
    U = rng.standard_normal((n, nocc))
    Vt = scale * rng.standard_normal((nocc, n))
    eng = JKEngine(lay, B, None, None, fitted=True, precision="split")
    K = eng.compute_k_lmo_asym(U, Vt)
    eng.close()
    Hu = (D.reshape(-1, n) @ U).reshape(naux, n, nocc).transpose(1, 0, 2).reshape(n, -1)
    Hv = (D.reshape(-1, n) @ Vt.T).reshape(naux, n, nocc).transpose(1, 0, 2).reshape(n, -1)
    Kr = -(Hu @ Hv.T)
    # three operands of 39 bits below their rows' exponents, summed over rows
    # of up to 75 * 97 terms: 2^-34 of the row norms' product
    assert np.abs(K - Kr).max() <= 2.0 ** -34 * np.linalg.norm(Hu, axis=1).max() * \
        np.linalg.norm(Hv, axis=1).max()
