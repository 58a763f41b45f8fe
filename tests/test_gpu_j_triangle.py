"""The mixed path's J column sums over the upper block triangle: a tensor
whose off-diagonal block pairs hold the same bits twice is read once and J
mirrored; any other tensor or column order is read whole.  Against dense
FP64 sums of the same tensor."""
import copy

import numpy as np
import pytest

from chem_gb300.fock import JKEngine
from chem_gb300.layout import build_layout

pytestmark = pytest.mark.gpu


def _tensor(bsizes, naux, kept, rng):
    """Layout and panel array of a symmetric random tensor."""
    lay = build_layout(bsizes, [naux], lambda i, j: np.array([kept(i, j)]))
    n = lay.nbf
    T = rng.standard_normal((naux, n, n))
    T = T + T.transpose(0, 2, 1)
    off = lay.boff
    B = np.zeros(lay.nnz)
    for i, cols in enumerate(lay.column_map()):
        b, k, o = int(lay.bsizes[i]), len(cols), int(lay.panel_off[i])
        B[o:o + b * naux * k] = T[:, off[i]:off[i + 1]][:, :, cols].transpose(1, 0, 2).ravel()
    return lay, B


def _reverse_columns(lay, B):
    """The same tensor with every panel's blocks in descending order."""
    out = copy.copy(lay)
    out.nbr = [list(reversed(v)) for v in lay.nbr]
    off, C = lay.boff, np.zeros_like(B)
    for i, (old, new) in enumerate(zip(lay.column_map(), out.column_map())):
        b, k, o = int(lay.bsizes[i]), len(old), int(lay.panel_off[i])
        P = B[o:o + b * lay.naux * k].reshape(b, lay.naux, k)
        C[o:o + b * lay.naux * k] = P[:, :, np.searchsorted(old, new)].ravel()
    return out, C


@pytest.mark.parametrize("form", ["symmetric", "one_element", "descending"])
@pytest.mark.parametrize("bsizes,naux", [([3], 33), ([5, 14, 5], 31), ([14, 14, 5, 9, 1, 14], 129),
                                         ([40, 30, 18, 9, 40], 260)])
def test_j_columns(form, bsizes, naux):
    rng = np.random.default_rng(17)
    lay, B = _tensor(bsizes, naux, lambda i, j: j - i <= 2, rng)
    if form == "one_element" and len(bsizes) > 1:
        B[int(lay.panel_off[1])] += 0.5  # an element below the diagonal
    if form == "descending":
        lay, B = _reverse_columns(lay, B)
    n = lay.nbf
    P = rng.standard_normal((n, n))
    P = P + P.T
    C = np.linalg.qr(rng.standard_normal((n, 2)))[0]
    eng = JKEngine(lay, B, None, None, fitted=True, precision="split")
    J, _ = eng.compute_jk(P, C)
    eng.close()
    dense = np.zeros((naux, n, n))
    off = lay.boff
    for i, cols in enumerate(lay.column_map()):
        b, k, o = int(lay.bsizes[i]), len(cols), int(lay.panel_off[i])
        dense[:, off[i]:off[i + 1], cols] = \
            B[o:o + b * naux * k].reshape(b, naux, k).transpose(1, 0, 2)
    Jr = np.einsum("xmn,x->mn", dense, np.einsum("xmn,mn->x", dense, P))
    # operands keep 39 bits below each row's exponent, J's tensor copy 40 bits
    # per element: 2^-36 of the sums of absolute values
    bound = np.einsum("xmn,x->mn", np.abs(dense), np.einsum("xmn,mn->x", np.abs(dense),
                                                            np.abs(P)))
    assert np.all(np.abs(J - Jr) <= 2.0 ** -36 * bound.max())
    if form == "symmetric":
        offd = np.ones((n, n), bool)
        for i in range(lay.nblk):
            offd[off[i]:off[i + 1], off[i]:off[i + 1]] = False
        assert np.array_equal(J[offd], J.T[offd])
