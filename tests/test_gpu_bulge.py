"""The bulge chasing (band -> tridiagonal) at the ends of its windows: sizes on both sides of
multiples of the window, where the last window has 2..32 rows or leaves one row over, with random
bands, bands that are already tridiagonal (every reflector is the identity) and bands with zero
rows in between.  The tridiagonal matrix has the eigenvalues of the input, to 8 n eps ||A|| (the
backward error of two orthogonal reductions)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIZES = (3, 4, 33, 34, 35, 36, 64, 65, 66, 67, 97, 98, 99, 129, 130, 161, 162, 193, 194)


def _matrix(n, kind):
    rng = np.random.default_rng(n)
    M = rng.standard_normal((n, n))
    A = (M + M.T) / 2
    i = np.arange(n)
    if kind == "band":
        A[np.abs(i[:, None] - i[None, :]) > 32] = 0.0
    elif kind == "tridiagonal":
        A[np.abs(i[:, None] - i[None, :]) > 1] = 0.0
    elif kind == "decoupled":
        A[np.abs(i[:, None] - i[None, :]) > 32] = 0.0
        A[n // 2:, : n // 2] = 0.0
        A[: n // 2, n // 2:] = 0.0
        A[n // 3, :] = A[:, n // 3] = 0.0
    return A


@pytest.mark.parametrize("kind", ["dense", "band", "tridiagonal", "decoupled"])
@pytest.mark.parametrize("n", SIZES)
def test_tridiagonal_has_the_same_spectrum(n, kind):
    import torch
    import bsr_b200 as bsr
    from bsr_b200._lib import call
    from bsr_b200.core import _ptr
    A = _matrix(n, kind)
    ctx = bsr.Context()
    dA = torch.from_numpy(np.tril(A).T.copy()).cuda()
    d = torch.empty(n, dtype=torch.float64, device="cuda")
    e = torch.empty(n - 1, dtype=torch.float64, device="cuda")
    call("bsrg_dsytrd_2stage", ctx.handle, n, _ptr(dA), n, _ptr(d), _ptr(e))
    torch.cuda.synchronize()
    dd, ee = d.cpu().numpy(), e.cpu().numpy()
    T = np.diag(dd) + np.diag(ee, 1) + np.diag(ee, -1)
    w = np.linalg.eigvalsh(A)
    tol = 8 * n * np.finfo(float).eps * max(np.max(np.abs(w)), 1e-300)
    assert np.max(np.abs(np.linalg.eigvalsh(T) - w)) <= tol
    if kind == "tridiagonal":
        assert np.array_equal(dd, np.diag(A))
    ctx.close()
