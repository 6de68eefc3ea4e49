"""diag_hd without eigenvectors on the library's eigensolver (reduction and bisection), and what the
dense solver gives for scaled and non-finite matrices."""
import ctypes

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

EPS = 2.0 ** -52


def _dsyevd(ctx, A):
    import bsr_b200 as bsr
    n = A.shape[0]
    w, Z = torch.empty(n, dtype=torch.float64, device="cuda"), torch.empty_like(A)
    p = lambda x: ctypes.c_void_p(x.data_ptr())
    assert bsr.lib().bsrg_dsyevd(ctx.handle, n, p(A), n, p(w), p(Z), n) == 0
    return w, Z


@pytest.mark.parametrize("cfg,nch", [("config1", 1), ("config1", 3), ("config1", 6), ("config2", 1), ("config2", 4)])
def test_values_only(cfg, nch):
    """The eigenvalues of both solvers without vectors, n eps ||A|| apart at most (each is backward
    stable with a bound well inside n eps ||A||), ascending, and also those of the library's with vectors."""
    import bsr_b200 as bsr
    from bsr_b200 import workload as W
    pw = W.partial_wave(cfg, nch=nch)
    b = bsr.define_spline(pw["t"], pw["ks"])
    ctx = bsr.Context()
    H = bsr.assemble(ctx, b, pw["z"], pw["lch"], pw["ech"], pw["P"], pw["kmax"], pw["coefs"])["hcc"]
    out = {}
    for which, vec in (("own", False), ("lib", False), ("own", True), ("auto", False)):
        ctx.set_eigensolver(which)
        r = bsr.diag_hd(ctx, b, pw["lch"], H, want_vectors=vec)
        out[which, vec] = r["eval"].cpu().numpy()
    ref = out["lib", False]
    n, norm = len(ref), np.abs(ref).max()
    for k, e in out.items():
        assert np.all(np.diff(e) >= 0.0), k
        assert np.abs(e - ref).max() <= n * EPS * norm, k
    ctx.set_eigensolver("own")
    for bad in (float("nan"), float("inf")):
        if nch == 1:
            break                                           # no coupling block
        h = H.clone()
        h[5, 6, 1] = h[6, 5, 1] = bad                       # H(2,1)
        for vec in (False, True):
            with pytest.raises(Exception):
                bsr.diag_hd(ctx, b, pw["lch"], bsr.as_fortran(h), want_vectors=vec)
    # the context goes on as before
    assert np.array_equal(bsr.diag_hd(ctx, b, pw["lch"], H, want_vectors=False)["eval"].cpu().numpy(),
                          out["own", False])


@pytest.mark.parametrize("sign", [1, -1])
@pytest.mark.parametrize("nch", [1, 3])
def test_values_only_one_sign(sign, nch):
    """Spectra on one side of zero (the channel solutions filtered by their energies), as cuSOLVER's."""
    import bsr_b200 as bsr
    from bsr_b200 import workload as W
    pw = W.partial_wave("config1", nch=nch)
    b = bsr.define_spline(pw["t"], pw["ks"])
    ctx = bsr.Context()
    H = bsr.assemble(ctx, b, pw["z"], pw["lch"], pw["ech"], pw["P"], pw["kmax"], pw["coefs"])["hcc"]
    flt = dict(Egap=1e3) if sign > 0 else dict(Edmax=-0.5)
    out = []
    for which in ("own", "lib"):
        ctx.set_eigensolver(which)
        out.append(bsr.diag_hd(ctx, b, pw["lch"], H, want_vectors=False, **flt)["eval"].cpu().numpy())
    a, ref = out
    assert len(a) == len(ref) and np.all(ref * sign > 0) and np.all(np.diff(a) >= 0.0)
    assert np.abs(a - ref).max() <= len(ref) * EPS * np.abs(ref).max()


@pytest.mark.parametrize("n", [1, 2, 33, 100, 257])
@pytest.mark.parametrize("q", [-1000, -400, 400, 1000])
def test_dsyevd_scaled(n, q):
    """2^q A has 2^q times the eigenvalues of A and the same vectors (residuals within n eps ||A||)."""
    import bsr_b200 as bsr
    g = torch.Generator(device="cuda").manual_seed(n)
    A = torch.randn(n, n, generator=g, device="cuda", dtype=torch.float64)
    A = A + A.t()
    ctx = bsr.Context()
    w0, _ = _dsyevd(ctx, A)
    s = 2.0 ** q
    w, Z = _dsyevd(ctx, A * s)
    norm = float(w0.abs().max())
    assert float((w / s - w0).abs().max()) <= n * EPS * norm + 1e-300
    Z = Z.t()                                               # column-major
    assert float((A @ Z - Z * (w / s)[None]).abs().max()) <= 8 * n * EPS * norm


@pytest.mark.parametrize("n", [2, 40, 129])
@pytest.mark.parametrize("bad", [float("nan"), float("inf"), float("-inf")])
def test_dsyevd_non_finite(n, bad):
    import bsr_b200 as bsr
    ctx = bsr.Context()
    A = torch.eye(n, dtype=torch.float64, device="cuda")
    A[n // 2, 0] = A[0, n // 2] = bad
    w, Z = _dsyevd(ctx, A)
    assert bool(torch.isnan(w).all()) and bool(torch.isnan(Z).all())
    w, _ = _dsyevd(ctx, torch.eye(n, dtype=torch.float64, device="cuda"))
    assert bool((w == 1.0).all())
