"""The back-transformation of the bulge chasing at the edges of its strips and rounds: widths that leave a
strip partly empty (n mod 8, and strips of 2 to 7 tiles), fewer groups than slots, and a last chunk of one
row.  Checked through the eigensolver: ||A Z - Z W|| and ||Z^T Z - I|| to 8 n eps (times ||A||); the
matrices' eigenvectors make every column of Z count."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 5, 9, 35, 36, 66, 67, 68, 98, 131, 200, 331, 2369, 3301, 3555, 4740])
def test_vectors(n):
    import torch
    import bsr_b200 as bsr
    from bsr_b200._lib import call
    from bsr_b200.core import _ptr
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64)
    A = (A + A.t()) / 2
    ctx = bsr.Context()
    w = torch.empty(n, dtype=torch.float64, device="cuda")
    Z = torch.full((n, n), float("nan"), dtype=torch.float64, device="cuda")
    call("bsrg_dsyevd", ctx.handle, n, _ptr(A), n, _ptr(w), _ptr(Z), n)
    torch.cuda.synchronize()
    an, tol = float(w.abs().max()), 8 * max(n, 16) * np.finfo(float).eps
    V = Z.t()
    assert float((A @ V - V * w).abs().max()) <= tol * an
    assert float((V.t() @ V - torch.eye(n, device="cuda", dtype=torch.float64)).abs().max()) <= tol
    ctx.close()
