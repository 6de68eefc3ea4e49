"""mqk_cell into an array with more columns a side than the table has: the table where it belongs, zeros elsewhere."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ldp", [5, 6, 255, 256, 300])
def test_columns_past_the_table(ldp):
    import bsr_b200 as bsr
    ks, ns = 3, 12
    t = np.concatenate([[0.0] * (ks - 1), np.linspace(0.0, 4.0, ns - ks + 2), [4.0] * (ks - 1)])
    b = bsr.define_spline(t, ks)
    ref = bsr.mqk_cell(b, 1).cpu().numpy()
    assert ref.shape == (ns, ns, 2 * ks - 1, 2 * ks - 1) and np.any(ref != 0.0)
    got = bsr.mqk_cell(b, 1, ldp=ldp).cpu().numpy()
    p = 2 * ks - 1
    assert np.array_equal(got[:, :, :p, :p], ref)
    got[:, :, :p, :p] = 0.0
    assert not np.any(got)
