"""W_OUT's channel order where weights are equal, or NaN: the exchange sort's, as the oracle has it."""
import numpy as np
import pytest

from oracle import oracle as O

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nch", [1, 2, 5, 32, 129])
def test_channel_weights_ties(nch):
    import torch

    import bsr_b200 as bsr
    rng = np.random.default_rng(nch)
    ipsol = np.arange(0, 2 * nch + 1, 2, dtype=np.int32)
    khm = 2 * nch
    a = np.asfortranarray(rng.integers(-2, 3, (khm, khm)).astype(np.float64))      # few values: many equal weights
    a[:, 0] = 1.0
    a[:, khm - 1] = rng.standard_normal(khm)                                       # no equal ones
    if nch > 2:
        a[3, 1] = np.nan
    wt, isol, iprm = bsr.channel_weights(bsr.Context(), ipsol, torch.from_numpy(a).cuda().t().contiguous().t())
    wr, ir, pr = O.channel_weights(ipsol, a)
    assert np.array_equal(wt.cpu().numpy(), wr, equal_nan=True)
    assert np.array_equal(isol.cpu().numpy(), ir) and np.array_equal(iprm.cpu().numpy(), pr)
