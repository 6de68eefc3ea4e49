"""Timed workloads of the library, through its public entry points.

Each case is one thing a BSR calculation has the library do:

  table      mrk_cell: the R^k table of one multipole on a B-spline basis
  breit      the six Breit-Pauli tables (N, M, T, V, W, Q) of one multipole
  integrals  Slater integrals between orbitals: density, convol (direct and exchange), SUM_AmB
  assemble   bsr_mat SUB1: the channel blocks of one partial wave from host coefficient records
  solve      one partial wave from host buffers to eigenvalues (bsr_mat + bsr_hd)
  dense      DSYEV on the device: every eigenvalue and eigenvector of a symmetric matrix
  solutions  what bsr_hd does after DSYEV: solutions in the B-spline basis, surface
             amplitudes, channel weights
  batch      several symmetries of one basis through the request server

Sizes come from the workload configurations of bsr_b200.workload (order 8 and 10, 60 to
200 splines, 8 to 40 channels); draw() spreads them over the range between.
"""
import ctypes
import math

import numpy as np
import torch

import bsr_b200 as bsr
from bsr_b200 import serve
from bsr_b200 import workload as W

F64 = torch.float64


# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------
def listed():
    return [
        # the smallest table a calculation builds (a bound-state basis): launches and latency
        dict(name="table_small", kind="table", ks=8, ns=60, rmax=20.0, k=2),
        # the production basis: the module array of one multipole, 32 MB
        dict(name="table_large", kind="table", ks=10, ns=200, rmax=40.0, k=4),
        # relativistic corrections on a mid-sized basis: all six operators of one multipole
        dict(name="breit_tables", kind="breit", ks=8, ns=150, rmax=30.0, k=1),
        # one direct and one exchange integral between orbitals, the inner loop of the radial codes
        dict(name="integrals", kind="integrals", ks=10, ns=200, rmax=40.0, k=2),
        # the interaction matrix of a large scattering symmetry, 137 thousand records
        dict(name="assemble_40ch", kind="assemble", ks=10, ns=200, rmax=40.0, kmax=8, norb=30, lmod=9, z=18.0,
             p=0.02, nch=40),
        # a small symmetry from host data to eigenvalues: latency
        dict(name="solve_8ch", kind="solve", ks=8, ns=60, rmax=20.0, kmax=4, norb=10, lmod=5, z=10.0, p=0.05, nch=8,
             vectors=True, mixed=False),
        # eigenvalues only (a scan of the spectrum), ordinary size
        dict(name="solve_15ch_values", kind="solve", ks=8, ns=150, rmax=30.0, kmax=6, norb=20, lmod=7, z=10.0, p=0.03,
             nch=15, vectors=False, mixed=False),
        # the mixed-precision form at an ordinary-to-large size
        dict(name="solve_30ch_mixed", kind="solve", ks=8, ns=150, rmax=30.0, kmax=6, norb=20, lmod=7, z=10.0, p=0.03,
             nch=30, vectors=True, mixed=True),
        # the production partial wave, 8000 rows, FP64
        dict(name="solve_40ch", kind="solve", ks=10, ns=200, rmax=40.0, kmax=8, norb=30, lmod=9, z=18.0, p=0.02,
             nch=40, vectors=True, mixed=False),
        # the eigensolver by itself on a matrix already on the device
        dict(name="dense_1713", kind="dense", n=1713),
        # post-processing of the solutions of a 20-channel symmetry
        dict(name="solutions_20ch", kind="solutions", ns=150, nch=20, lmod=7),
        # a batch of symmetries of one basis submitted together
        dict(name="batch_8sym", kind="batch", ks=8, ns=150, rmax=30.0, kmax=6, norb=20, lmod=7, z=10.0, p=0.03,
             nsym=8, nch_lo=4, nch_hi=30, streams=4),
    ]


def _log_int(rng, lo, hi):
    return int(math.floor(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))


def _basis_draw(rng):
    ks = rng.choice([8, 9, 10])
    return dict(ks=ks, ns=rng.randint(60, 200), rmax=round(rng.uniform(20.0, 40.0), 3))


def draw(rng):
    kind = rng.choice(["table", "breit", "integrals", "assemble", "solve", "solve", "dense", "dense", "solutions", "batch"])
    b = _basis_draw(rng)
    if kind == "table":
        return dict(kind=kind, k=rng.randint(0, 8), **b)
    if kind == "breit":
        b["ks"] = 8
        b["ns"] = rng.randint(60, 150)
        return dict(kind=kind, k=rng.randint(0, 4), **b)
    if kind == "integrals":
        return dict(kind=kind, k=rng.randint(0, 8), **b)
    if kind == "dense":
        return dict(kind=kind, n=_log_int(rng, 200, 5000))
    if kind == "solutions":
        return dict(kind=kind, ns=b["ns"], nch=_log_int(rng, 4, 24), lmod=rng.randint(4, 9))
    phys = dict(kmax=rng.randint(4, 8), norb=rng.randint(10, 30), lmod=rng.randint(5, 9), z=float(rng.randint(10, 18)),
                p=round(rng.uniform(0.02, 0.05), 4))
    if kind == "batch":
        b["ks"], b["ns"] = 8, rng.randint(100, 150)
        return dict(kind=kind, nsym=rng.randint(4, 8), nch_lo=4, nch_hi=rng.randint(12, 28), streams=4, **b, **phys)
    nch = _log_int(rng, 4, 40)
    b["ns"] = min(b["ns"], 7600 // nch)
    if kind == "assemble":
        return dict(kind=kind, nch=nch, **b, **phys)
    return dict(kind=kind, nch=nch, vectors=rng.random() < 0.75, mixed=rng.random() < 0.3, **b, **phys)


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
_PHYS = ("ks", "ns", "rmax", "kmax", "norb", "lmod", "z", "p")


def _wave(case, seed):
    return W.partial_wave("config4", seed=seed, nch=case["nch"], **{q: case[q] for q in _PHYS})


def _knots(case):
    return W.knot_grid(case["ks"], case["ns"], 1e-3, case["rmax"])[0]


def _batch(case, seed):
    """Symmetries of one basis and orbital set; channel counts spread evenly (in their
    logarithm) over nch_lo..nch_hi, so that every seed has the same amount of work."""
    base = W.partial_wave("config4", seed=seed, nch=1, **{q: case[q] for q in _PHYS})
    rng = np.random.default_rng(seed + 1)
    n, lo, hi = case["nsym"], math.log(case["nch_lo"]), math.log(case["nch_hi"])
    base["symmetries"] = []
    for q in range(n):
        nch = int(round(math.exp(lo + (hi - lo) * q / max(1, n - 1))))
        base["symmetries"].append(dict(
            nch=nch, lch=np.array([c % case["lmod"] for c in range(nch)], dtype=np.int32),
            ech=rng.uniform(-1.0, 0.0, size=nch),
            coefs=W.coefficients(rng, nch, case["norb"], case["kmax"], case["p"])))
    return base


class _Served:
    """A request server that ends with its owner."""

    def __init__(self, b, streams):
        self.server = serve.PartialWaveServer(b["t"], b["ks"], b["z"], b["P"], b["kmax"], n_streams=streams)
        self.server.warm(max(b["symmetries"], key=lambda s: s["nch"]))

    def __del__(self):
        server = self.__dict__.pop("server", None)
        if server is not None:
            server.close()


def _dense_matrix(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(case["n"], case["n"], generator=g, device="cuda", dtype=F64)
    return a + a.t()


def _solution_sizes(case):
    """Solutions kept per channel: one spline less than the basis for each of the first l + 1."""
    return [case["ns"] - (c % case["lmod"]) - 1 for c in range(case["nch"])]


def _solution_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    sizes = _solution_sizes(case)
    khm = sum(sizes)
    a = torch.randn(khm, khm, generator=g, device="cuda", dtype=F64) / math.sqrt(khm)
    bb = torch.randn(case["nch"] * case["ns"], case["ns"], generator=g, device="cuda", dtype=F64)
    ipsol = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int32)
    return a.t(), bb.t(), ipsol          # column-major, as diag_hd returns them


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case)
    if kind in ("table", "breit"):
        # another seed, other knots: the grid's end moves by up to 1 %
        s["basis"] = bsr.define_spline(_seeded_knots(case, seed), case["ks"])
    elif kind == "integrals":
        s["basis"] = bsr.define_spline(_knots(case), case["ks"])
        s["rkb"] = bsr.mrk_cell(s["basis"], case["k"])
        s["P"] = [bsr.as_fortran(p) for p in _orbital_set(case, seed)]
    elif kind == "assemble":
        pw = _wave(case, seed)
        s["pw"], s["ctx"] = pw, bsr.Context()
        s["basis"] = bsr.define_spline(pw["t"], pw["ks"])
        s["P"] = bsr.as_fortran(pw["P"])
    elif kind == "solve":
        s["pw"], s["ctx"] = _wave(case, seed), bsr.Context()
        s["ctx"].set_precision(case["mixed"])
    elif kind == "dense":
        n = case["n"]
        s["ctx"], s["A"] = bsr.Context(), _dense_matrix(case, seed)
        s["w"] = torch.empty(n, device="cuda", dtype=F64)
        s["Z"] = torch.empty(n, n, device="cuda", dtype=F64)
    elif kind == "solutions":
        s["ctx"] = bsr.Context()
        s["a"], s["bb"], s["ipsol"] = _solution_inputs(case, seed)
    elif kind == "batch":
        b = _batch(case, seed)
        s["symmetries"] = b["symmetries"]
        s["served"] = _Served(b, case["streams"])
    return s


def _seeded_knots(case, seed):
    t = _knots(case).copy()
    ks, f = case["ks"], 1.0 + 0.01 * np.random.default_rng(seed).random()
    t[ks:] *= f
    return t


def _orbital_set(case, seed):
    P = W.orbitals(np.random.default_rng(seed), _knots(case), case["ks"], 4)
    return [P[:, q] for q in range(4)]


# ---------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------
def run(s):
    return _RUN[s["kind"]](s)


def _run_table(s):
    return bsr.mrk_cell(s["basis"], s["k"])


def _run_breit(s):
    from bsr_b200 import core
    b, k = s["basis"], s["k"]
    return [f(b, k) for f in (core.mnk_cell, core.mmk_cell, core.mtk_cell, core.mvk_cell, core.mwk_cell, core.mqk_cell)]


def _run_integrals(s):
    ns, ks, rkb = s["ns"], s["ks"], s["rkb"]
    p1, p2, p3, p4 = s["P"]
    y = bsr.convol(ns, ks, bsr.density(ns, ks, p1, p3, "s"), rkb, 1, "s", "s")
    direct = bsr.sum_amb(ns, ks, y, bsr.density(ns, ks, p2, p4, "s"), "s")
    x = bsr.convol(ns, ks, bsr.density(ns, ks, p3, p2, "x"), rkb, 3, "s", "s")
    exchange = bsr.sum_amb(ns, ks, x, bsr.density(ns, ks, p1, p4, "x"), "x")
    return {"direct": direct, "exchange": exchange, "y": y, "x": x}


def _run_assemble(s):
    pw = s["pw"]
    return bsr.assemble(s["ctx"], s["basis"], pw["z"], pw["lch"], pw["ech"], s["P"], pw["kmax"], pw["coefs"])["hcc"]


def _run_solve(s):
    pw = s["pw"]
    return _spectrum(bsr.partial_wave_solve(s["ctx"], pw, want_vectors=s["vectors"]), pw["nch"], pw["ns"])


def _spectrum(e, nch, ns):
    """Eigenvalues in an array of the declared length nch * ns, zeros after the last: how many
    channel solutions the energy filter keeps depends on the inputs."""
    out = np.zeros(nch * ns)
    out[:len(e)] = e
    return out


def _run_dense(s):
    n, w, Z = s["n"], s["w"], s["Z"]
    p = lambda x: ctypes.c_void_p(x.data_ptr())  # noqa: E731
    rc = bsr.lib().bsrg_dsyevd(s["ctx"].handle, n, p(s["A"]), n, p(w), p(Z), n)
    if rc != 0:
        raise bsr.BsrgError("bsrg_dsyevd", rc, bsr.lib().bsrg_last_error().decode())
    return {"w": w, "Z": _phases(Z)}


def _phases(Z):
    """Eigenvectors (the rows of Z) with their largest component positive, in a new tensor:
    a vector's sign is not determined."""
    top = Z.gather(1, Z.abs().argmax(dim=1, keepdim=True))
    return Z * torch.sign(top)


def _run_solutions(s):
    from bsr_b200 import core
    v, wmat = core.rsol_out(s["ctx"], s["ns"], s["ipsol"], s["bb"], s["a"])
    wt, isol, iprm = core.channel_weights(s["ctx"], s["ipsol"], s["a"])
    return {"v": v, "wmat": wmat, "wt": wt, "isol": isol, "iprm": iprm}


def _run_batch(s):
    server = s["served"].server
    requests = [server.submit(q) for q in s["symmetries"]]
    return [_spectrum(r.wait(600.0)["eval"], q["nch"], s["ns"]) for r, q in zip(requests, s["symmetries"])]


_RUN = dict(table=_run_table, breit=_run_breit, integrals=_run_integrals, assemble=_run_assemble, solve=_run_solve,
            dense=_run_dense, solutions=_run_solutions, batch=_run_batch)


# ---------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------
def _dense_flops(n, vectors):
    """Reduction to tridiagonal form 4/3 n^3; with vectors the tridiagonal eigenvectors and
    the back-transformation, 4/3 n^3 + 2 n^3."""
    return (4.0 / 3.0 + (10.0 / 3.0 if vectors else 0.0)) * float(n) ** 3


def _assembly_work(c, nch):
    """Tables of every multipole and the blocks written once; per multipole the direct
    contraction of one density a channel pair and the exchange products of the orbitals."""
    ns, ks, nblk, nk = c["ns"], c["ks"], nch * (nch + 1) // 2, c["kmax"] + 1
    direct = 2.0 * (ns * ks) ** 2 * nblk
    exchange = 2.0 * ns * ns * ((2 * ks - 1) * c["norb"] ** 2 + nblk * c["p"] * c["norb"] * (c["norb"] + 1) / 2)
    return 8.0 * (nblk * ns * ns), nk * (direct + exchange)


def _solve_work(c, nch, vectors):
    ns = c["ns"]
    khm = nch * ns - sum((q % c["lmod"]) + 1 for q in range(nch))
    b, f = _assembly_work(c, nch)
    f += 2.0 * nch * (nch + 1) * float(ns) ** 3 + _dense_flops(khm, vectors)      # block transforms, DSYEV
    if vectors:
        f += 2.0 * float(khm) ** 3                                                # residuals of the refinement
    return 8.0 * khm * khm * (3 if vectors else 1) + b, f


def work(case):
    kind = case["kind"]
    if kind == "table":
        ns, ks = case["ns"], case["ks"]
        return dict(bytes=8.0 * (ns * ks) ** 2, flops=float(ns * ks) ** 2)
    if kind == "breit":
        ns, ks = case["ns"], case["ks"]
        return dict(bytes=8.0 * ns * ns * (2 * ks * ks + 4 * (2 * ks - 1) ** 2), flops=6.0 * ns * ns * (2 * ks - 1) ** 2)
    if kind == "integrals":
        ns, ks = case["ns"], case["ks"]
        return dict(bytes=8.0 * ((ns * ks) ** 2 + 4 * ns * ns), flops=2.0 * (ns * ks) ** 2 * 5)
    if kind == "assemble":
        b, f = _assembly_work(case, case["nch"])
        return dict(bytes=b, flops=f)
    if kind == "solve":
        b, f = _solve_work(case, case["nch"], case["vectors"])
        return dict(bytes=b, flops=f)
    if kind == "dense":
        return dict(bytes=16.0 * case["n"] ** 2, flops=_dense_flops(case["n"], True))
    if kind == "solutions":
        khm, n = sum(_solution_sizes(case)), case["ns"] * case["nch"]
        return dict(bytes=8.0 * (khm * khm + n * khm + 2.5 * case["nch"] * khm), flops=2.0 * khm * khm * case["ns"])
    n, lo, hi = case["nsym"], math.log(case["nch_lo"]), math.log(case["nch_hi"])
    each = [_solve_work(case, int(round(math.exp(lo + (hi - lo) * q / max(1, n - 1)))), True) for q in range(n)]
    return dict(bytes=sum(e[0] for e in each), flops=sum(e[1] for e in each))


# ---------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------------------
def _dev(x):
    return torch.as_tensor(np.ascontiguousarray(x)).to("cuda", F64)


def _gauss(n):
    """Gauss-Legendre rule on [0, 1]."""
    x, w = np.polynomial.legendre.leggauss(n)
    return _dev((x + 1) / 2), _dev(w / 2)


def _splines(t, k, x, cell, orders=1):
    """B-splines of order k at the points x of the knot intervals cell (0-based, from the
    first non-empty one), and of the orders below: a list of (points, splines) arrays."""
    v = torch.zeros(x.numel(), t.numel() - 1, device=x.device, dtype=F64)
    v.scatter_(1, (cell.reshape(-1, 1) + k - 1), 1.0)
    x, out = x.reshape(-1, 1), []
    for q in range(2, k + 1):
        if q > k - orders + 1:
            out.insert(0, v)
        m = t.numel() - q
        dl, dr = t[q - 1:q - 1 + m] - t[:m], t[q:q + m] - t[1:1 + m]
        il, ir = torch.where(dl > 0, 1 / dl, 0 * dl), torch.where(dr > 0, 1 / dr, 0 * dr)
        v = (x - t[:m]) * il * v[:, :m] + (t[q:q + m] - x) * ir * v[:, 1:1 + m]
    return [v] + out


def _derivative(t, q, low):
    """Derivatives of the splines of order q from the coefficients' splines of order q - 1."""
    m = t.numel() - q
    dl, dr = t[q - 1:q - 1 + m] - t[:m], t[q:q + m] - t[1:1 + m]
    il, ir = torch.where(dl > 0, 1 / dl, 0 * dl), torch.where(dr > 0, 1 / dr, 0 * dr)
    return (q - 1) * (il * low[:, :m] - ir * low[:, 1:1 + m])


class _Quadrature:
    """The k-point Gauss rule of every knot interval and the splines at its points."""

    def __init__(self, t, ks):
        self.t, self.ks, self.ns = _dev(t), ks, len(t) - ks
        self.nv = self.ns - ks + 1
        gx, gw = _gauss(ks)
        self.gx, self.gw = gx, gw
        left, right = self.t[ks - 1:self.ns], self.t[ks:self.ns + 1]
        self.left = left
        self.x = (left[:, None] + (right - left)[:, None] * gx).reshape(-1)
        self.w = ((right - left)[:, None] * gw).reshape(-1)
        self.cell = torch.arange(self.nv, device="cuda").repeat_interleave(ks)
        low = _splines(self.t, ks, self.x, self.cell, orders=3)
        self.b = low[0]
        self.d2 = _derivative(self.t, ks, _derivative(self.t, ks - 1, low[2]))

    def pairs(self, b):
        """B_i B_{i+ip} as (..., ns, ks), zero past the last spline."""
        pad = torch.nn.functional.pad(b, (0, self.ks))
        return torch.stack([b * pad[..., p:p + self.ns] for p in range(self.ks)], dim=-1)

    def table(self, k):
        """R^k(i, j, ip, jp): the outer rule over r1, the inner one over the whole intervals
        below r1 and the part of r1's own, r2 < r1; then the same with the electrons exchanged."""
        ks, ns, nv = self.ks, self.ns, self.nv
        outer = self.pairs(self.b) * (self.w * self.x ** -(k + 1))[:, None, None]
        whole = (self.pairs(self.b) * (self.w * self.x ** k)[:, None, None]).reshape(nv, ks, ns, ks).sum(1)
        below = torch.cumsum(whole, 0) - whole
        span = self.x - self.left[self.cell]
        xi = self.left[self.cell][:, None] + span[:, None] * self.gx
        wi = span[:, None] * self.gw * xi ** k
        inner = []
        for q in range(0, xi.shape[0], 256):
            c = self.cell[q:q + 256]
            b = _splines(self.t, ks, xi[q:q + 256].reshape(-1), c.repeat_interleave(ks))[0]
            b = b.reshape(-1, ks, ns)
            part = torch.einsum("pm,pmsq->psq", wi[q:q + 256], self.pairs(b))
            inner.append(part + below[c])
        half = outer.reshape(-1, ns * ks).t() @ torch.cat(inner).reshape(-1, ns * ks)
        return (half + half.t()).reshape(ns, ks, ns, ks).permute(0, 2, 1, 3)


def _both_sides(R):
    """The table over offsets -(ks-1)..ks-1 of both electrons."""
    ns, ks = R.shape[0], R.shape[2]
    X = torch.zeros(ns, ns, 2 * ks - 1, 2 * ks - 1, device=R.device, dtype=F64)
    X[:, :, ks - 1:, ks - 1:] = R
    for e in range(1, ks):                       # element (i, i - e) is element (i - e, i)
        X[:, :, ks - 1 - e] = torch.roll(X[:, :, ks - 1 + e], e, 0)
        X[:e, :, ks - 1 - e] = 0
    for f in range(1, ks):
        X[:, :, :, ks - 1 - f] = torch.roll(X[:, :, :, ks - 1 + f], f, 1)
        X[:, :f, :, ks - 1 - f] = 0
    return X


def _exchange_products(R, P):
    """K[a, b](i, j') = sum R(i i'; j j') P(i', a) P(j, b) for every orbital pair."""
    ns, ks, no = R.shape[0], R.shape[2], P.shape[1]
    X, pad = _both_sides(R), torch.nn.functional.pad(P, (0, 0, ks - 1, ks - 1))
    win = torch.stack([pad[e:e + ns] for e in range(2 * ks - 1)], 1)          # P(i + e, a): (ns, 2ks-1, no)
    Y = torch.einsum("ijef,iea->aijf", X, win)
    K = torch.zeros(no, no, ns, ns, device=R.device, dtype=F64)
    for f in range(1 - ks, ks):
        lo, hi = max(0, -f), min(ns, ns - f)
        K[:, :, :, lo + f:hi + f] += Y[:, None, :, lo:hi, f + ks - 1] * P[lo:hi].t()[None, :, None, :]
    return K


def _blocks(pw):
    """The channel blocks (nblk, ns, ns) of a partial wave."""
    q = _Quadrature(pw["t"], pw["ks"])
    ns, ks, nch, P, c = q.ns, q.ks, len(pw["lch"]), _dev(pw["P"]), pw["coefs"]
    nblk, no = nch * (nch + 1) // 2, P.shape[1]
    H = torch.zeros(nblk, ns * ns, device="cuda", dtype=F64)
    blk = c["ich"].astype(np.int64) * (c["ich"] - 1) // 2 + c["jch"] - 1
    for k in range(pw["kmax"] + 1):
        R = q.table(k)
        for ty in (0, 1):
            m = np.nonzero((c["k"] == k) & (c["type"] == ty))[0]
            if not len(m):
                continue
            C = torch.zeros(nblk, no * no, device="cuda", dtype=F64)
            at = torch.as_tensor(np.stack([blk[m], c["a"][m].astype(np.int64) * no + c["b"][m]])).cuda()
            C.index_put_((at[0], at[1]), _dev(c["c"][m]), accumulate=True)
            if ty == 0:
                pad = torch.nn.functional.pad(P, (0, 0, 0, ks))
                D = torch.stack([P[:, :, None] * pad[p:p + ns][:, None, :] for p in range(ks)], 1)
                D[:, 1:] += torch.stack([pad[p:p + ns][:, :, None] * P[:, None, :] for p in range(1, ks)], 1)
                A = R.permute(0, 2, 1, 3).reshape(ns * ks, ns * ks) @ D.reshape(ns * ks, no * no) @ C.t()
                A = A.reshape(ns, ks, nblk)
                V = H.view(nblk, ns, ns)
                for p in range(ks):
                    i = torch.arange(ns - p, device="cuda")
                    V[:, i, i + p] += A[:ns - p, p].t()
                    if p:
                        V[:, i + p, i] += A[:ns - p, p].t()
            else:
                H += C @ _exchange_products(R, P).reshape(no * no, ns * ns)
    V = H.view(nblk, ns, ns)
    wb = q.w[:, None] * q.b
    S, rm1, rm2 = wb.t() @ q.b, (wb / q.x[:, None]).t() @ q.b, (wb / q.x[:, None] ** 2).t() @ q.b
    D2 = torch.tril(wb.t() @ q.d2)
    D2 = D2 + torch.tril(D2, -1).t()
    last = q.cell == q.nv - 1
    edge = (wb[last, ns - 2] * q.d2[last, ns - 1]).sum() - D2[ns - 1, ns - 2]       # Bloch term
    D2[ns - 1, ns - 2] += edge
    D2[ns - 2, ns - 1] += edge
    D2[ns - 1, ns - 1] -= edge
    for i in range(nch):
        b, l = i * (i + 1) // 2 + i, int(pw["lch"][i])
        V[b] += -0.5 * (D2 - l * (l + 1) * rm2 + 2 * pw["z"] * rm1) + float(pw["ech"][i]) * S
        V[b] = (V[b] + V[b].t()) / 2
    return V, S


def _eigenvalues(pw):
    """bsr_hd: channel eigenbases with the first l + 1 splines dropped and |E| < 0.001 left
    out, then the whole matrix in them."""
    V, S = _blocks(pw)
    nch, ns, ks = len(pw["lch"]), V.shape[1], pw["ks"]
    H = torch.zeros(nch * ns, nch * ns, device="cuda", dtype=F64)
    cols = []
    for i in range(nch):
        for j in range(i + 1):
            b = V[i * (i + 1) // 2 + j]
            H[i * ns:(i + 1) * ns, j * ns:(j + 1) * ns] = b
            H[j * ns:(j + 1) * ns, i * ns:(i + 1) * ns] = b.t()
        f = min(int(pw["lch"][i]), ks - 2) + 1
        L = torch.linalg.cholesky(S[f:, f:])
        C = torch.linalg.solve_triangular(L, V[i * (i + 1) // 2 + i][f:, f:], upper=False)
        C = torch.linalg.solve_triangular(L, C.t().contiguous(), upper=False)
        e, u = torch.linalg.eigh((C + C.t()) / 2)
        u = torch.linalg.solve_triangular(L.t(), u, upper=True)[:, e.abs() >= 0.001]
        cols.append((i * ns + f, u))
    B = torch.zeros(nch * ns, sum(u.shape[1] for _, u in cols), device="cuda", dtype=F64)
    at = 0
    for row, u in cols:
        B[row:row + u.shape[0], at:at + u.shape[1]] = u
        at += u.shape[1]
    A = B.t() @ (H @ B)
    return _spectrum(torch.linalg.eigvalsh((A + A.t()) / 2).cpu().numpy(), nch, ns)


def exact(case, seed):
    kind = case["kind"]
    if kind == "table":
        return _Quadrature(_seeded_knots(case, seed), case["ks"]).table(case["k"])
    if kind == "integrals":
        R = _Quadrature(_knots(case), case["ks"]).table(case["k"])
        ns, ks = case["ns"], case["ks"]
        p1, p2, p3, p4 = [_dev(p) for p in _orbital_set(case, seed)]

        def band(a, b):
            d = torch.zeros(ns, ks, device="cuda", dtype=F64)
            for p in range(ks):
                d[:ns - p, p] = a[:ns - p] * b[p:] + (a[p:] * b[:ns - p] if p else 0)
            return d
        y = torch.einsum("ijpq,jq->ip", R, band(p1, p3))
        x = _exchange_products(R, torch.stack([p3, p2], 1))[0, 1]
        return {"direct": (y * band(p2, p4)).sum().reshape(1), "exchange": (p1 @ x @ p4).reshape(1), "y": y, "x": x}
    if kind == "assemble":
        return _blocks(_wave(case, seed))[0].permute(1, 2, 0)
    if kind == "solve":
        return _eigenvalues(_wave(case, seed))
    if kind == "dense":
        w, Z = torch.linalg.eigh(_dense_matrix(case, seed))
        return {"w": w, "Z": _phases(Z.t().contiguous())}
    if kind == "solutions":
        a, bb, ipsol = _solution_inputs(case, seed)
        ns, nch = case["ns"], case["nch"]
        v = torch.cat([bb[:, c * ns:c * ns + int(ipsol[c + 1] - ipsol[c])] @ a[int(ipsol[c]):int(ipsol[c + 1])]
                       for c in range(nch)])
        wt = torch.stack([(a[int(ipsol[c]):int(ipsol[c + 1])] ** 2).sum(0) for c in range(nch)])
        return {"v": v, "wmat": v[ns - 1::ns], "wt": wt, "isol": None, "iprm": None}
    if kind == "batch":
        b = _batch(case, seed)
        return [_eigenvalues({**b, "lch": s["lch"], "ech": s["ech"], "coefs": s["coefs"]}) for s in b["symmetries"]]
    return None
