"""The mixed path's prefit L^-1 B on the tensor cores at the edges of its tiles
(48 metric rows, 128 tensor columns, 32 k per stage, 128 k per exact chunk):
K and J of an engine with a graded metric factor against dense FP64 sums, and
the FP64 MP2 batch, which keeps its own in-order prefit, before and after."""
import numpy as np
import pytest

from chem_gb300.fock import JKEngine
from chem_gb300.layout import build_layout

pytestmark = pytest.mark.gpu


def _system(naux, bsizes, seed):
    rng = np.random.default_rng(seed)
    lay = build_layout(bsizes, [naux], lambda i, j: np.array([j - i <= 1]))
    n, off = lay.nbf, lay.boff
    T = rng.standard_normal((naux, n, n)) * 2.0 ** rng.integers(-12, 3, (naux, 1, 1))
    T = T + T.transpose(0, 2, 1)
    B, D = np.zeros(lay.nnz), np.zeros_like(T)
    for i, cols in enumerate(lay.column_map()):
        b, k, o = int(lay.bsizes[i]), len(cols), int(lay.panel_off[i])
        blk = T[:, off[i]:off[i + 1]][:, :, cols]
        B[o:o + b * naux * k] = blk.transpose(1, 0, 2).ravel()
        D[:, off[i]:off[i + 1], cols] = blk
    L = np.tril(rng.standard_normal((naux, naux)) * 2.0 ** rng.integers(-8, 1, (naux, 1)))
    return lay, B, D, L, rng


@pytest.mark.parametrize("naux", [1, 31, 32, 33, 47, 48, 49, 96, 97, 127, 128, 129, 160, 257])
@pytest.mark.parametrize("bsizes", [[3, 9, 5], [40, 14, 30, 1]])
def test_k_and_j(naux, bsizes):
    lay, B, D, L, rng = _system(naux, bsizes, 1000 + naux)
    n = lay.nbf
    C = np.linalg.qr(rng.standard_normal((n, 3)))[0]
    P = rng.standard_normal((n, n))
    P = P + P.T
    eng = JKEngine(lay, B, L, L.T @ L, precision="split")
    J, K = eng.compute_jk(P, C)
    eng.close()
    F = np.einsum("xy,ymn->xmn", L, D)
    H = np.einsum("xmn,ni->mxi", F, C).reshape(n, -1)
    Kr = -(H @ H.T)
    Jr = np.einsum("xmn,x->mn", F, np.einsum("xmn,mn->x", F, P))
    # 39-bit operands below the rows' exponents (see the exchange's own tests)
    A = np.einsum("xmn,x->mn", np.abs(F), np.einsum("xmn,mn->x", np.abs(F), np.abs(P)))
    assert np.abs(K - Kr).max() <= 2.0 ** -33 * np.linalg.norm(H, axis=1).max() ** 2
    assert np.abs(J - Jr).max() <= 2.0 ** -36 * A.max()


def test_fp64_mp2_keeps_its_prefit():
    lay, B, D, L, rng = _system(70, [9, 14, 5], 3)
    n = lay.nbf
    Lo, Lv = [rng.standard_normal((n, 4))], [rng.standard_normal((n, 11))]

    def fp64(eng):
        eng.set_precision("fp64")
        e, Z = eng.mp2_laplace(Lo, Lv, want_z=True)
        return e, Z

    eng = JKEngine(lay, B, L, L.T @ L)
    e0, Z0 = fp64(eng)
    eng.set_precision("split")
    es, _ = eng.mp2_laplace(Lo, Lv)
    e1, Z1 = fp64(eng)
    eng.mp2_release()
    e2, Z2 = fp64(eng)
    eng.close()
    assert np.array_equal(Z0, Z1) and np.array_equal(Z0, Z2)
    assert e0[0] == e1[0] == e2[0]
    assert abs(es[0] - e0[0]) <= 1e-8 * e0[0]
