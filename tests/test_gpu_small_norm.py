"""Tridiagonal and dense matrices of small norm: 2^-q times a matrix has 2^-q times its eigenvalues and the same
vectors.  The deflation's tolerance is eps ||T||: residuals and eigenvalues to 8 n eps ||A||, as at norm 1."""
import numpy as np
import pytest
from scipy.linalg import eigh_tridiagonal

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps
SCALES = (-4, -20, -60, -160)


def _check(T, wr, W, V, n):
    an, tol = np.max(np.abs(wr)), 8 * max(n, 16) * EPS
    assert np.all(np.diff(W) >= 0)
    assert np.max(np.abs(W - wr)) <= tol * an
    assert np.max(np.abs(T @ V - V * W[None, :])) <= tol * an
    assert np.max(np.abs(V.T @ V - np.eye(n))) <= tol


@pytest.mark.parametrize("q", SCALES)
@pytest.mark.parametrize("n", [65, 129, 1000])
def test_dstedc(n, q):
    import torch
    import bsr_b200 as bsr
    from bsr_b200._lib import call
    from bsr_b200.core import _ptr
    rng = np.random.default_rng(n)
    d, e = rng.standard_normal(n) * 2.0 ** q, rng.standard_normal(n - 1) * 2.0 ** q
    ctx = bsr.Context()
    dd, de = torch.from_numpy(d).cuda(), torch.from_numpy(e).cuda()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    Z = torch.empty((n, n), dtype=torch.float64, device="cuda")
    call("bsrg_dstedc", ctx.handle, n, _ptr(dd), _ptr(de), _ptr(w), _ptr(Z), n)
    torch.cuda.synchronize()
    _check(np.diag(d) + np.diag(e, 1) + np.diag(e, -1), eigh_tridiagonal(d, e, eigvals_only=True), w.cpu().numpy(),
           Z.cpu().numpy().T, n)
    ctx.close()


@pytest.mark.parametrize("q", SCALES)
@pytest.mark.parametrize("n", [100, 257])
def test_dsyevd(n, q):
    import torch
    import bsr_b200 as bsr
    from bsr_b200._lib import call
    from bsr_b200.core import _ptr
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n))
    A = (M + M.T) * 2.0 ** q
    ctx = bsr.Context()
    dA = torch.from_numpy(A.copy()).cuda()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    Z = torch.empty((n, n), dtype=torch.float64, device="cuda")
    call("bsrg_dsyevd", ctx.handle, n, _ptr(dA), n, _ptr(w), _ptr(Z), n)
    torch.cuda.synchronize()
    _check(A, np.linalg.eigvalsh(A), w.cpu().numpy(), Z.cpu().numpy().T, n)
    ctx.close()
