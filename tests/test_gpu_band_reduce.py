"""The dense -> band stage at the edges of its splits: panels of a few rows, one row more or less than a
cluster CTA's share, clusters of 1, 2, 3 and 16 CTAs, and panels whose columns vanish (low rank, zero
blocks: reflectors with tau = 0).  Checked through the whole eigensolver: eigenvalues against numpy,
residual and orthogonality, each to 8 n eps (times ||A||)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _matrix(n, kind):
    rng = np.random.default_rng(7 * n)
    M = rng.standard_normal((n, n))
    A = (M + M.T) / 2
    if kind == "lowrank":
        U = rng.standard_normal((n, 3))
        A = U @ np.diag([3.0, -1.0, 0.5]) @ U.T
        A = (A + A.T) / 2
    elif kind == "zero-blocks":
        A[40:, :40] = 0.0
        A[:40, 40:] = 0.0
        A[n // 2:, : n // 2] = 0.0
        A[: n // 2, n // 2:] = 0.0
    return A


@pytest.mark.parametrize("n,kind", [(34, "random"), (63, "random"), (191, "random"), (192, "random"), (193, "random"),
                                    (353, "random"), (513, "random"), (674, "random"), (2593, "random"),
                                    (2594, "random"), (200, "lowrank"), (411, "lowrank"), (300, "zero-blocks"),
                                    (700, "zero-blocks")])
def test_whole_solver(n, kind):
    import torch
    import bsr_b200 as bsr
    from bsr_b200._lib import call
    from bsr_b200.core import _ptr
    A = _matrix(n, kind)
    ctx = bsr.Context()
    dA = torch.from_numpy(np.tril(A).T.copy()).cuda()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    Z = torch.empty(n * n, dtype=torch.float64, device="cuda")
    call("bsrg_dsyevd", ctx.handle, n, _ptr(dA), n, _ptr(w), _ptr(Z), n)
    torch.cuda.synchronize()
    W, V = w.cpu().numpy(), Z.cpu().numpy().reshape(n, n).T
    wr = np.linalg.eigvalsh(A)
    an, tol = np.max(np.abs(wr)), 8 * n * EPS
    assert np.max(np.abs(W - wr)) <= tol * an
    assert np.max(np.abs(A @ V - V * W[None, :])) <= tol * an
    assert np.max(np.abs(V.T @ V - np.eye(n))) <= tol
    ctx.close()
