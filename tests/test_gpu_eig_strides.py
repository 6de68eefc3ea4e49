"""The dense eigensolver with leading dimensions above n: rows past n are neither read nor written, nor is A's upper
triangle, and Z may be A itself.  Bounds as everywhere: 8 n eps (times ||A||)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


@pytest.mark.parametrize("alias", [False, True])
@pytest.mark.parametrize("pad", [0, 1, 5])
@pytest.mark.parametrize("n", [1, 2, 33, 100, 321])
def test_dsyevd(n, pad, alias):
    import torch
    import bsr_b200 as bsr
    from bsr_b200._lib import call
    from bsr_b200.core import _ptr
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n))
    A = M + M.T
    X = np.full((n, n + pad), np.nan)                       # row j: column j of A
    X[:, :n] = np.where(np.tri(n, dtype=bool), A, np.nan).T
    ctx = bsr.Context()
    dA = torch.from_numpy(X).cuda()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    Z = dA if alias else torch.full((n, n + pad), float("nan"), dtype=torch.float64, device="cuda")
    call("bsrg_dsyevd", ctx.handle, n, _ptr(dA), n + pad, _ptr(w), _ptr(Z), n + pad)
    torch.cuda.synchronize()
    if not alias:
        assert np.array_equal(dA.cpu().numpy(), X, equal_nan=True)
    W, Z = w.cpu().numpy(), Z.cpu().numpy()
    assert np.all(np.isnan(Z[:, n:]))
    V, wr = Z[:, :n].T, np.linalg.eigvalsh(A)
    an, tol = np.max(np.abs(wr)), 8 * n * EPS
    assert np.max(np.abs(W - wr)) <= tol * an
    assert np.max(np.abs(A @ V - V * W[None, :])) <= tol * an
    assert np.max(np.abs(V.T @ V - np.eye(n))) <= tol
    ctx.close()
