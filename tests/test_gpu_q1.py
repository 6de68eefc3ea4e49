"""The back-transformation of the band reduction: its T factors on the second stream or on the solve's own."""
import ctypes

import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 64, 65, 288, 289, 545, 801])
def test_q1_streams(n, monkeypatch):
    """One panel, one group of eight panels and one more, three groups: the same bits either way, orthonormal
    vectors and residuals within 4 n eps of the norm."""
    import bsr_b200 as bsr
    ctx = bsr.Context()
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64)
    A = A + A.t()
    p = lambda x: ctypes.c_void_p(x.data_ptr())
    out = []
    for one in (False, True):
        if one:
            monkeypatch.setenv("BSRG_NO_LOOKAHEAD", "1")
        w, Z = torch.empty(n, device="cuda", dtype=torch.float64), torch.empty_like(A)
        assert bsr.lib().bsrg_dsyevd(ctx.handle, n, p(A), n, p(w), p(Z), n) == 0
        out.append((w, Z))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    w, V = out[0][0], out[0][1].t()
    tol = 4 * n * 2.0 ** -52
    assert float((A @ V - V * w[None]).abs().max()) <= tol * float(w.abs().max())
    assert float((V.t() @ V - torch.eye(n, device="cuda", dtype=torch.float64)).abs().max()) <= tol
