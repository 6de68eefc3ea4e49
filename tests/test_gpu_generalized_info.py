"""An overlap that is not positive definite, or not finite, stops the generalized branch with the factorisation's
error at every size and with either eigensolver, also where the reduced matrix comes out non-finite."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bad", ["indefinite", "nan"])
@pytest.mark.parametrize("nch,vectors", [(2, True), (10, False), (14, True)])
@pytest.mark.parametrize("which", ["auto", "lib"])
def test_cholesky_error(bad, nch, vectors, which):
    import bsr_b200 as bsr
    from bsr_b200 import workload as W
    pw = W.partial_wave("config1", nch=nch)
    b = bsr.define_spline(pw["t"], pw["ks"])
    ctx = bsr.Context()
    ctx.set_eigensolver(which)
    H = bsr.assemble(ctx, b, pw["z"], pw["lch"], pw["ech"], pw["P"], pw["kmax"], pw["coefs"], want_s=True)
    scc = H["scc"].cpu().numpy().copy()
    scc[:, :, 1] = 2.0 * scc[:, :, 0] if bad == "indefinite" else np.nan
    with pytest.raises(bsr.BsrgError, match="Cholesky"):
        bsr.diag_hd(ctx, b, pw["lch"], H["hcc"], want_vectors=vectors, scc=bsr.as_fortran(scc))
    ctx.close()
