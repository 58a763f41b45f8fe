"""gbjk_mp2_release gives back every device buffer of the batch, and the next
batch gives the same bits."""
import numpy as np
import pytest

from chem_gb300.fock import JKEngine

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "split"])
def test_release_returns_the_memory(precision, water):
    ds = water
    rng = np.random.default_rng(1)
    Lo, Lv = [rng.standard_normal((ds.nbf, 4))], [rng.standard_normal((ds.nbf, 9))]
    eng = JKEngine(ds.layout, ds.B, np.tril(ds.Linv), ds.Vinv, precision=precision)
    if precision == "split":
        eng.compute_jk(None, Lo[0])  # the engine's own prefitted tensor
    held = eng.device_bytes
    first = eng.mp2_laplace(Lo, Lv, want_z=True)
    assert eng.device_bytes > held
    eng.mp2_release()
    # (fp64: the exchange's and the batch's buffers are separate)
    assert eng.device_bytes == held
    again = eng.mp2_laplace(Lo, Lv, want_z=True)
    eng.close()
    assert np.array_equal(first[0], again[0]) and np.array_equal(first[1], again[1])


@pytest.mark.parametrize("precision", ["fp64", "split"])
def test_batches_of_changing_shape(precision, water):
    """One engine, batches of other ranks and numbers of points in turn (the staging
    buffer of the factors stays and grows): the bits of an engine of its own."""
    ds = water
    rng = np.random.default_rng(5)
    batches = [([rng.standard_normal((ds.nbf, r)) for r in ro],
                [rng.standard_normal((ds.nbf, r)) for r in rv])
               for ro, rv in (([3, 5], [7, 9]), ([4], [11]), ([5, 2, 1], [13, 3, 8]))]

    def engine():
        return JKEngine(ds.layout, ds.B, np.tril(ds.Linv), ds.Vinv, precision=precision)

    want = []
    for b in batches:
        eng = engine()
        want.append(eng.mp2_laplace(*b, want_z=True))
        eng.close()
    eng = engine()
    for i in (0, 1, 0, 2, 2, 1, 0):
        e, Z = eng.mp2_laplace(*batches[i], want_z=True)
        assert np.array_equal(e, want[i][0]) and np.array_equal(Z, want[i][1]), i
    eng.close()
