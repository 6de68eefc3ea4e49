"""rsol_out's batched launches: more channels than one launch takes (64), channels without solutions, and basis
columns past a channel's solutions, which are not read.  A product of m terms is within 2 m eps of sum |b| |a| (two
summation orders, each within m eps / 2 plus the products' roundings)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nch,ns", [(1, 9), (3, 33), (63, 12), (64, 7), (65, 7), (129, 40), (200, 3)])
@pytest.mark.parametrize("empty", [False, True])
def test_rsol_out(nch, ns, empty):
    import torch
    import bsr_b200 as bsr
    rng = np.random.default_rng(nch)
    m = rng.integers(1, ns + 1, nch)
    if empty:
        m[rng.integers(0, nch, (nch + 2) // 3)] = 0
        m[-1] = max(m[-1], 1)
    ip = np.concatenate([[0], np.cumsum(m)]).astype(np.int32)
    khm = int(ip[-1])
    a = rng.standard_normal((khm, khm))
    bb = rng.standard_normal((ns, nch * ns))
    ref, bound = np.zeros((nch * ns, khm)), np.zeros((nch * ns, khm))
    for i in range(nch):
        b, x = bb[:, i * ns:i * ns + m[i]], a[ip[i]:ip[i + 1]]
        ref[i * ns:(i + 1) * ns] = b @ x
        bound[i * ns:(i + 1) * ns] = 2 * max(m[i], 1) * np.finfo(float).eps * (np.abs(b) @ np.abs(x))
        bb[:, i * ns + m[i]:(i + 1) * ns] = np.nan
    v, w = bsr.rsol_out(bsr.Context(), ns, ip, bsr.as_fortran(bb), bsr.as_fortran(a))
    torch.cuda.synchronize()
    v, w = v.cpu().numpy(), w.cpu().numpy()
    assert np.all(np.abs(v - ref) <= bound)
    assert np.array_equal(w, v[ns - 1::ns])
