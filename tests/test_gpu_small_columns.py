"""Columns whose entries are so small that their squares are subnormal or vanish (1e-150 .. 1e-170) in a matrix of
ordinary size: the reflectors must stay orthogonal.  A dropped column of size s is a backward error of s, far
below the rounding, so the bounds are those of any matrix: 8 n eps (times ||A||), as the solver's backward errors
are a modest multiple of eps ||A||."""
import numpy as np
import pytest
import scipy.linalg as sl

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps
SIZES = (1e-150, 1e-155, 1e-158, 1e-160, 1e-161, 1e-162, 1e-165, 1e-170)


def _coupled(n, kind, s):
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n))
    A = (M + M.T) / 2
    i = np.arange(n)
    if kind == "blocks":                      # two blocks, every coupling of size s: whole panels are small
        h = n // 2 // 32 * 32
        A[h:, :h] *= s
        A[:h, h:] *= s
    elif kind == "band":                      # already a band: columns of the chase are small
        A[np.abs(i[:, None] - i[None, :]) > 32] = 0.0
        for c in (0, n // 3):
            A[c + 1:, :c + 1] *= s
            A[:c + 1, c + 1:] *= s
    return A


@pytest.mark.parametrize("s", SIZES)
@pytest.mark.parametrize("n,kind", [(64, "blocks"), (200, "blocks"), (700, "blocks"), (40, "band"), (130, "band")])
def test_dense(n, kind, s):
    import torch
    import bsr_b200 as bsr
    from bsr_b200._lib import call
    from bsr_b200.core import _ptr
    A = _coupled(n, kind, s)
    ctx = bsr.Context()
    dA = torch.from_numpy(np.tril(A).T.copy()).cuda()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    Z = torch.empty(n * n, dtype=torch.float64, device="cuda")
    d, e = torch.empty(n, dtype=torch.float64, device="cuda"), torch.empty(n - 1, dtype=torch.float64, device="cuda")
    call("bsrg_dsyevd", ctx.handle, n, _ptr(dA), n, _ptr(w), _ptr(Z), n)
    call("bsrg_dsytrd_2stage", ctx.handle, n, _ptr(dA), n, _ptr(d), _ptr(e))
    torch.cuda.synchronize()
    W, V = w.cpu().numpy(), Z.cpu().numpy().reshape(n, n).T
    wr = np.linalg.eigvalsh(A)
    an, tol = np.max(np.abs(wr)), 8 * n * EPS
    assert np.max(np.abs(sl.eigh_tridiagonal(d.cpu().numpy(), e.cpu().numpy(), eigvals_only=True) - wr)) <= tol * an
    assert np.max(np.abs(W - wr)) <= tol * an
    assert np.max(np.abs(A @ V - V * W[None, :])) <= tol * an
    assert np.max(np.abs(V.T @ V - np.eye(n))) <= tol
    ctx.close()
