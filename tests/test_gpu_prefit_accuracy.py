"""The tensor-core prefit L^-1 B, element by element, against double-double sums:
its digits' own bound, at the edges of its tiles, for operands without structure,
for sums that cancel to 2^-20 of their terms (where an FP64 chain is off by
2^-53 of the terms) and for auxiliary functions of very different scale."""
import numpy as np
import pytest

from chem_gb300.fock import JKEngine
from chem_gb300.layout import build_layout

pytestmark = pytest.mark.gpu


def _two_sum(a, b):
    s = a + b
    t = s - a
    return s, (a - (s - t)) + (b - t)


def _split(a):
    t = 134217729.0 * a
    h = t - (t - a)
    return h, a - h


def _dd_product(L, B):
    """L @ B as (hi, lo), every product and sum exact to about 2^-104."""
    hi = np.zeros((L.shape[0], B.shape[1]))
    lo = np.zeros_like(hi)
    for y in range(L.shape[1]):
        a, b = L[:, y:y + 1], B[y:y + 1]
        p = a * b
        (ah, al), (bh, bl) = _split(a), _split(b)
        e = ((ah * bh - p) + ah * bl + al * bh) + al * bl
        hi, t = _two_sum(hi, p)
        lo += t + e
    return _two_sum(hi, lo)


def _exponent(a, axis):
    """e with |a| < 2^e."""
    return np.frexp(np.abs(a).max(axis))[1]


def _check(eng, lay, L, D, dense_to_panels):
    """Every element of the engine's prefitted tensor against L D."""
    naux, n = D.shape[0], D.shape[1]
    with pytest.raises(RuntimeError):
        eng.download_fitted()
    eng.compute_jk(None, np.eye(n)[:, :2].copy())
    F = eng.download_fitted()
    eng.close()
    Dm = D.reshape(naux, n * n)
    hi, lo = _dd_product(L, Dm)
    hi, lo = (dense_to_panels(lay, x.reshape(naux, n, n))[0] for x in (hi, lo))
    # exponents of the operands with the columns of L taken to 1
    ey = _exponent(L, 0)
    Ls, Ds = np.ldexp(L, -ey[None]), np.ldexp(Dm, ey[:, None])
    ed = _exponent(Ds, 0)
    E = np.where(np.abs(Dm).max(0) > 0, _exponent(Ls, 1)[:, None] + ed, -1000)
    # per term: 2 operands rounded at half a unit of 2^-63 and the 7 dropped digit
    # pairs of 2^-64 (6 of 2^-72, ..); one rounding of the result
    bound = naux * 9.1 * np.ldexp(1.0, E - 64)
    bound = dense_to_panels(lay, bound.reshape(naux, n, n))[0] + 2.0 ** -53 * np.abs(hi)
    assert (np.abs((F - hi) - lo) <= bound).all()


@pytest.mark.parametrize("kind", ["plain", "cancelling", "scaled"])
@pytest.mark.parametrize("naux", [1, 32, 33, 48, 49, 128, 129, 257])
def test_prefit_elements(naux, kind, dense_to_panels):
    rng = np.random.default_rng(naux)
    lay = build_layout([3, 14, 5], [naux], lambda i, j: np.array([j - i <= 1]))
    n = lay.nbf
    T = rng.standard_normal((naux, n, n))
    T = T + T.transpose(0, 2, 1)
    L = np.tril(rng.standard_normal((naux, naux)))
    if kind == "cancelling":
        # functions 2j and 2j + 1 are the same, with opposite factors but for 2^-20
        m = naux // 2 * 2
        T[1:m:2] = T[0:m:2]
        L[:, 1:m:2] = -L[:, 0:m:2] * (1.0 + 2.0 ** -20 * rng.standard_normal((naux, m // 2)))
        L = np.tril(L)
        L[np.arange(0, m, 2), np.arange(0, m, 2)] *= 2.0 ** -20
    elif kind == "scaled":
        s = 2.0 ** rng.integers(-30, 31, naux)
        T, L = T * s[:, None, None], L / s
    B, D = dense_to_panels(lay, T)
    eng = JKEngine(lay, B, L, L.T @ L, precision="split")
    _check(eng, lay, L, D, dense_to_panels)


@pytest.mark.parametrize("spread", [20, 60])
@pytest.mark.parametrize("naux", [33, 130])
def test_columns_keep_their_own_scale(naux, spread, dense_to_panels):
    """AO and auxiliary functions scaled over many powers of two and integrals that
    vanish for some of them: the bound holds in every column."""
    rng = np.random.default_rng(naux + spread)
    lay = build_layout([3, 9, 4], [naux], lambda i, j: np.array([True]))
    n = lay.nbf
    T = rng.standard_normal((naux, n, n))
    T[rng.random((naux, n, n)) < 0.5] = 0.0
    T = T + T.transpose(0, 2, 1)
    T[:5, :4] = 0.0
    T[:5, :, :4] = 0.0  # auxiliary functions without the first AO functions
    T[7] = 0.0          # .. without any
    a = 2.0 ** rng.integers(-spread, 1, n)
    s = 2.0 ** rng.integers(-spread, spread + 1, naux)
    L = np.tril(rng.standard_normal((naux, naux))) / s
    B, D = dense_to_panels(lay, T * (s[:, None, None] * a[:, None] * a[None]))
    eng = JKEngine(lay, B, L, L.T @ L, precision="split")
    _check(eng, lay, L, D, dense_to_panels)
