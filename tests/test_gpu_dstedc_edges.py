"""The tridiagonal divide and conquer at the edges of its leaves (32 rows) and merges, and where deflation
does most of the work: sizes around multiples of a leaf, matrices whose halves share eigenvalues (every
pair rotates), decoupled and constant ones, and graded ones.  Eigenvalues against LAPACK's bisection,
residual and orthogonality to 8 n eps (times ||T||)."""
import numpy as np
import pytest
from scipy.linalg import eigh_tridiagonal

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _tridiagonal(n, kind):
    rng = np.random.default_rng(n)
    d, e = rng.standard_normal(n), rng.standard_normal(max(n - 1, 0))
    if kind == "wilkinson":
        d, e = np.abs(np.arange(n) - (n - 1) / 2.0), np.ones(max(n - 1, 0))
    elif kind == "glued":                    # copies of one block weakly coupled: equal eigenvalues everywhere
        b = 16
        d = np.tile(np.abs(np.arange(b) - (b - 1) / 2.0), n // b + 1)[:n]
        e = np.ones(max(n - 1, 0))
        e[b - 1::b] = 1e-11
    elif kind == "constant":
        d, e = np.full(n, 2.0), np.zeros(max(n - 1, 0))
    elif kind == "graded":
        d = np.logspace(-3, 7, n)
        e = 0.1 * np.sqrt(d[1:] * d[:-1]) if n > 1 else e
    return d, e


@pytest.mark.parametrize("kind", ["random", "wilkinson", "glued", "constant", "graded"])
@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 64, 65, 66, 127, 129, 257, 1000])
def test_dstedc(n, kind):
    import torch
    import bsr_b200 as bsr
    from bsr_b200._lib import call
    from bsr_b200.core import _ptr
    d, e = _tridiagonal(n, kind)
    ctx = bsr.Context()
    dd, de = torch.from_numpy(d).cuda(), torch.from_numpy(np.append(e, 0.0)).cuda()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    Z = torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda")
    for _ in range(2):                       # twice in a row: the second call's staging follows the first's
        call("bsrg_dstedc", ctx.handle, n, _ptr(dd), _ptr(de), _ptr(w), _ptr(Z), n)
    torch.cuda.synchronize()
    W, V = w.cpu().numpy(), Z.cpu().numpy().T
    wr = eigh_tridiagonal(d, e, eigvals_only=True) if n > 1 else d
    T = np.diag(d) + np.diag(e, 1) + np.diag(e, -1)
    an, tol = max(np.max(np.abs(wr)), 1e-300), 8 * max(n, 16) * EPS
    assert np.all(np.diff(W) >= 0)
    assert np.max(np.abs(W - wr)) <= tol * an
    assert np.max(np.abs(T @ V - V * W[None, :])) <= tol * an
    assert np.max(np.abs(V.T @ V - np.eye(n))) <= tol
    ctx.close()
