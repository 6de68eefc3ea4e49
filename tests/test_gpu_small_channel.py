"""A channel whose matrix has a column with entries so small that their squares are subnormal or vanish (1e-150 ..
1e-170): the reflectors must stay orthogonal.  The bound is that of any channel, n eps cond(S) ||C||, as
C = L^-1 H L^-T carries the conditioning of the overlap."""
import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps
SIZES = (1e-150, 1e-155, 1e-158, 1e-160, 1e-161, 1e-162, 1e-165, 1e-170)


@pytest.mark.parametrize("s", SIZES)
@pytest.mark.parametrize("cfg", ["config1", "config2"])
def test_channel(cfg, s):
    """One channel whose first spline is coupled to the others, and to itself, by s: C = L^-1 H L^-T has that
    column as it is, since L^-1 is lower triangular."""
    import bsr_b200 as bsr
    from bsr_b200 import workload as W
    pw = W.partial_wave(cfg, nch=1)
    b = bsr.define_spline(pw["t"], pw["ks"])
    ns, ks = b.ns, b.ks
    sb = b.get("sb").cpu().numpy()
    S = np.zeros((ns, ns))
    for j in range(ks):
        o = ks - 1 - j                        # S(i, i - o)
        for i in range(o, ns):
            S[i, i - o] = S[i - o, i] = sb[i, j]
    rng = np.random.default_rng(ns)
    M = rng.standard_normal((ns, ns))
    H = (M + M.T) / 2
    H[1, :] *= s                              # l = 0: rows 1 .. ns-1 are the channel's
    H[2:, 1] = H[1, 2:]
    Hr, Sr = H[1:, 1:], S[1:, 1:]
    wr = sl.eigh(Hr, Sr, eigvals_only=True)
    ctx = bsr.Context()
    ctx.set_eigensolver("lib")
    r = bsr.diag_hd(ctx, b, [0], bsr.as_fortran(H[:, :, None].copy()), want_vectors=False)
    assert ctx.channel_fallbacks() == 0
    w = r["eval"].cpu().numpy()
    an = np.max(np.abs(wr))
    ref = wr[np.abs(wr) > 1e-3]               # the filter of channel solutions
    assert len(w) == len(ref)
    assert np.max(np.abs(w - ref)) <= len(wr) * EPS * np.linalg.cond(Sr) * an
    ctx.close()
