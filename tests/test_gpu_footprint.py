"""The server's admission estimate against the bytes that an engine holds after
its first build: never below, and close enough that what fits is admitted."""
import numpy as np
import pytest

from chem_gb300.fock import JKEngine
from chem_gb300.serving import footprint_bytes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sysname", ["water", "butane", "decane", "c20h42"])
def test_estimate(sysname, request):
    ds = request.getfixturevalue(sysname)
    C = np.linalg.qr(np.random.default_rng(3).standard_normal((ds.nbf, ds.nocc)))[0]
    eng = JKEngine(ds.layout, ds.B, np.tril(ds.Linv), ds.Vinv, eps=1e-10, precision="split")
    eng.compute_jk(2.0 * C @ C.T, C)
    held = eng.device_bytes
    eng.close()
    est = footprint_bytes(ds.layout, ds.nocc, "split")
    # 5 % and 64 MB of slack, and the split-K partials at their upper bound
    assert held <= est <= 1.1 * held + 80e6
