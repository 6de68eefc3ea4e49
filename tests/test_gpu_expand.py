"""The table expansion kernels at orders and sizes off their tiles (32 x 64 elements, a band of
2 ks - 1 diagonals), bit for bit against the oracle: small and odd orders, a basis barely wider
than its order, sizes just below and above a tile, and moments that overflow (a high power at a
tiny first interval), where the terms outside the grid must not be formed."""
import numpy as np
import pytest

from tests.gpu_helpers import to_np

pytestmark = pytest.mark.gpu
SIZES = [(3, 35), (4, 5), (5, 41), (7, 64), (9, 97), (12, 33)]
CELLS = ["mrk_cell", "mmk_cell", "mnk_cell", "mtk_cell", "mvk_cell", "mwk_cell", "mqk_cell"]


def _knots(ks, ns, r0):
    inner = r0 * 1.2 ** np.arange(ns - ks)
    return np.concatenate([np.zeros(ks), inner, np.full(ks, inner[-1] * 1.2 if len(inner) else 1.0)])


def _both(ks, ns, r0, cell, k):
    import bsr_b200 as bsr
    from bsr_b200 import core
    from oracle import oracle as O
    t = _knots(ks, ns, r0)
    gb, ob = bsr.define_spline(t, ks), O.Basis(ks, t)
    if cell == "mrk_cell":
        return to_np(core.mrk_cell(gb, k)), ob.mrk_cell(k)
    return to_np(getattr(core, cell)(gb, k, fine=0.75)), getattr(ob, cell)(k, fine=0.75)


@pytest.mark.parametrize("cell", CELLS)
@pytest.mark.parametrize("ks,ns", SIZES)
def test_bitwise(ks, ns, cell):
    got, ref = _both(ks, ns, 0.01, cell, 2)
    assert np.array_equal(got, ref)


@pytest.mark.parametrize("cell", CELLS)
def test_overflowing_moments(cell):
    with np.errstate(all="ignore"):
        got, ref = _both(5, 70, 1e-6, cell, 62)
    assert not np.all(np.isfinite(ref))
    assert np.array_equal(got, ref, equal_nan=True)
