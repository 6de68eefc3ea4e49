"""diag_hd on a device with too little memory left for the library eigensolver's workspace, but enough for
cuSOLVER's: the automatic choice turns to cuSOLVER, also on later calls, and the context serves other sizes as before."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _wave(nch):
    import bsr_b200 as bsr
    from bsr_b200 import workload as W
    pw = W.partial_wave("config1", nch=nch)
    b = bsr.define_spline(pw["t"], pw["ks"])
    with_ctx = bsr.Context()
    H = bsr.assemble(with_ctx, b, pw["z"], pw["lch"], pw["ech"], pw["P"], pw["kmax"], pw["coefs"])["hcc"]
    with_ctx.close()
    return b, pw["lch"], H


def test_falls_back_to_cusolver():
    import torch
    import bsr_b200 as bsr
    large, small = _wave(40), _wave(2)

    def solve(ctx, wave):
        r = bsr.diag_hd(ctx, *wave)
        return r["eval"].cpu().numpy(), r["khm"]

    def context(which):
        ctx = bsr.Context()
        ctx.set_eigensolver(which)
        solve(ctx, small)                     # the libraries' handles take what they need
        torch.cuda.synchronize()
        return ctx

    def free():
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    used, out = {}, {}
    for which in ("lib", "own", "lib", "own"):              # the second time with the modules loaded
        ctx = context(which)
        before = free()
        out[which], khm = solve(ctx, large)
        used[which] = before - free()
        ctx.close()
    assert khm >= 640 and not np.array_equal(out["own"], out["lib"])
    assert used["own"] > used["lib"] + (64 << 20)
    ctx = context("auto")
    ref_small = solve(ctx, small)[0]
    filler = torch.empty(free() - (used["own"] + used["lib"]) // 2, dtype=torch.uint8, device="cuda")
    try:
        for _ in range(2):
            assert np.array_equal(solve(ctx, large)[0], out["lib"])
            assert np.array_equal(solve(ctx, small)[0], ref_small)
        # asked for, the library's solver has no room; the error is that call's alone
        ctx.set_eigensolver("own")
        with pytest.raises(bsr.BsrgError, match="memory"):
            solve(ctx, large)
        ctx.set_eigensolver("auto")
        assert np.array_equal(solve(ctx, small)[0], ref_small)
        assert np.array_equal(solve(ctx, large)[0], out["lib"])
    finally:
        del filler
        torch.cuda.empty_cache()
    assert np.array_equal(solve(ctx, large)[0], out["own"])  # with the memory back, the library's again
    ctx.close()
