"""convol and SUM_AmB at the edges of their tiles (16 outputs x 128 terms, 32 x 8 offsets, chunks of
2048 terms): direct cases and sums bit for bit against the oracle, exchange cases to 1e-13 of the
result's norm (the order of the offsets differs)."""
import numpy as np
import pytest

from oracle import oracle as O
from tests.conftest import rel_err
from tests.gpu_helpers import to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("icase", [1, 2, 3, 4])
@pytest.mark.parametrize("syms", ["ss", "nn", "ns", "sn"])
@pytest.mark.parametrize("ns,ks", [(7, 4), (16, 8), (17, 3), (33, 9), (64, 2), (70, 12)])
def test_convol(icase, syms, ns, ks):
    import bsr_b200 as bsr
    rng = np.random.default_rng(100 * ns + icase)
    rkb = np.asfortranarray(rng.standard_normal((ns, ns, 2 * ks - 1, 2 * ks - 1)))
    d = np.asfortranarray(rng.standard_normal((ns, max(ns, 2 * ks - 1))))
    ref = O.convol(ns, ks, d, rkb, icase, syms[0], syms[1])
    got = to_np(bsr.convol(ns, ks, d, rkb, icase, syms[0], syms[1]))
    if icase <= 2:
        w = min(got.shape[1], ref.shape[1])
        assert np.array_equal(got[:, :w], ref[:, :w])
    else:
        assert rel_err(got, ref) < 1e-13


@pytest.mark.parametrize("sym", ["s", "l", "n", "x"])
@pytest.mark.parametrize("ns,ks", [(3, 2), (45, 3), (46, 12), (64, 16), (65, 8), (181, 12), (256, 8)])
def test_sum_amb(sym, ns, ks):
    import bsr_b200 as bsr
    rng = np.random.default_rng(ns)
    n = max(ns, 2 * ks - 1)
    a = np.asfortranarray(rng.standard_normal((ns, n)))
    b = np.asfortranarray(rng.standard_normal((ns, n)))
    assert float(bsr.sum_amb(ns, ks, a, b, sym).cpu()[0]) == O.sum_amb(ns, ks, a, b, sym)
