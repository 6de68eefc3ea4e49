"""The channel eigenproblems of diag_hd on the library's kernels, at the sizes where they can go wrong: one
chunk of 32 rows more or less, the panel widths of the back-transformation, each spline order."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _grid(ns, ks):
    """Knots of ns splines of order ks: multiple end knots, growing steps."""
    m = ns - ks + 2                                     # distinct knots
    x = np.linspace(0.0, 1.0, m) ** 2 * 40.0 + np.linspace(0.0, 1.0, m) * 2.0
    return np.concatenate([np.zeros(ks - 1), x, np.full(ks - 1, x[-1])])


@pytest.mark.parametrize("ns,ks,nch", [(9, 4, 3), (34, 4, 2), (35, 5, 3), (66, 8, 1), (67, 6, 40), (100, 3, 2),
                                       (131, 8, 4), (195, 10, 2), (208, 8, 3), (60, 16, 2), (97, 2, 2)])
def test_channel_solves(ns, ks, nch):
    """One block per channel, H = kinetic-like + potential (symmetric, banded and a dense low-rank part):
    the dense problem without coupling is the union of the channels' spectra.  The library's kernels against
    scipy's generalized solver, within 2 n eps times the norm times the condition number of S."""
    import scipy.linalg as sl

    import bsr_b200 as bsr
    t = _grid(ns, ks)
    b = bsr.define_spline(t, ks)
    assert b.ns == ns
    rng = np.random.default_rng(ns * 100 + ks)
    sb = b.get("sb").cpu().numpy()
    S = np.zeros((ns, ns))
    for i in range(ns):
        for q in range(ks):
            if i - q >= 0:
                S[i, i - q] = S[i - q, i] = sb[i, ks - 1 - q]
    lch = [c % min(3, ks - 1) for c in range(nch)]
    hcc = np.zeros((ns, ns, nch * (nch + 1) // 2))
    want, cond, norm = [], 1.0, 0.0
    for c in range(nch):
        A = rng.standard_normal((ns, ns))
        H = S @ (A + A.T) @ S
        hcc[:, :, (c + 1) * (c + 2) // 2 - 1] = H
        s0, s1 = min(lch[c], ks - 2) + 1, ns
        w = sl.eigh(H[s0:s1, s0:s1], S[s0:s1, s0:s1], eigvals_only=True)
        ev = np.linalg.eigvalsh(S[s0:s1, s0:s1])
        cond, norm = max(cond, ev[-1] / ev[0]), max(norm, np.abs(w).max())
        want.append(w)
    want = np.concatenate(want)
    want = np.sort(want[np.abs(want) >= 0.001])
    ctx = bsr.Context()
    for vec in (True, False):
        r = bsr.diag_hd(ctx, b, lch, bsr.as_fortran(torch.tensor(hcc, device="cuda")), want_vectors=vec)
        got = r["eval"].cpu().numpy()
        assert len(got) == len(want)
        assert np.abs(got - want).max() <= 2 * ns * 2.0 ** -52 * norm * cond
    assert ctx.channel_fallbacks() == 0
