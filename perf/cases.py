"""Performance cases of the lDGA ladder path: what a user's program has the library do, through its
C ABI entry points (``Context.call``), over the sizes the repository's configurations, tests and
benchmark use and over generic ones between them.

Kinds of work (``case["kind"]``):

* ``chain``  -- one parameter point's whole lambda_m chain (``ldga_chain_m``; ``graph``: captured and
  replayed), or several points of uneven box size in one ``ldga_batch_chain_m`` call (``points`` > 1);
* ``bubble`` -- the lattice G of a new Sigma_loc and the bubble chi_0 (``ldga_gloc``, ``ldga_bubble``);
* ``chi``    -- the Bethe-Salpeter step of both channels (``ldga_bse`` for m and d), the vertices given;
* ``sigma``  -- one residual of the lambda correction: lambda_0, the equation of motion at (lambda_m,
  lambda_d), the mu fit, G_ladder and the energies (``ldga_lambda0``, ``ldga_eom``, ``ldga_g_ladder``);
* ``adjoint`` -- the vector-Jacobian product of the whole chain at fixed lambda (``ldga_chain_vjp``).

Chains use an RPA-like local vertex with 20 % noise at half-bandwidth units (t = 0.25 in 2D,
t = 1/sqrt(24) in 3D), where the lambda_m root is well conditioned; the single stages use the
repository's seeded generator (``ladderdga_b200.synthetic``).
"""
import ctypes as C
import dataclasses
import math

import numpy as np
import torch

import ladderdga_b200 as L
from ladderdga_b200 import _lib
from ladderdga_b200 import synthetic as S

T3 = 0.2041241452319315
PREC = {"fp64": L.PREC_FP64, "mixed": L.PREC_MIXED}
# k-grids and box sizes of the library's configurations, tests and benchmark, small to large
NS = {2: (6, 8, 10, 12, 16, 20, 24, 32, 40, 48, 64), 3: (4, 6, 8, 10, 12, 16, 20, 24, 32)}
N_IV = (4, 5, 6, 7, 8, 9, 10, 12, 13, 15, 17, 18, 20, 23, 25, 27, 30, 33, 40, 47, 60)


def listed():
    return [
        # a single DMFT point of a parameter scan on a small 2D grid, host buffers, graph replayed
        dict(name="chain 2d16 n20", kind="chain", dim=2, ns=16, beta=10.0, U=1.0, n_iv=10, n_iw=10, prec="mixed",
             graph=True, points=1),
        # the headline box (3D 32^3, 969 irreducible q) as one whole call
        dict(name="chain 3d32 n40", kind="chain", dim=3, ns=32, beta=8.0, U=1.5, n_iv=20, n_iw=20, prec="mixed",
             graph=True, points=1),
        # an uneven (U, beta) scan: eight 2D 32^2 points of three box sizes in one call
        dict(name="scan 2d32 8 points", kind="chain", dim=2, ns=32, beta=10.0, U=2.0, n_iv=30, n_iw=30, prec="mixed",
             graph=True, points=8),
        # G and bubble of a new self-energy (the start of every chain and of each self-consistent step)
        dict(name="bubble 3d32 n40", kind="bubble", dim=3, ns=32, beta=20.0, U=1.5, n_iv=20, n_iw=20, prec="mixed"),
        # Bethe-Salpeter at the headline box, MIXED mode
        dict(name="chi 3d32 n40 mixed", kind="chi", dim=3, ns=32, beta=20.0, U=1.5, n_iv=20, n_iw=20, prec="mixed"),
        # FP64 mode (the default of setup_LDGA) on the adjoint configuration's grid
        dict(name="chi 2d48 n40 fp64", kind="chi", dim=2, ns=48, beta=20.0, U=1.5, n_iv=20, n_iw=20, prec="fp64"),
        # the lambda_dm configuration's box, MIXED
        dict(name="chi 2d64 n60 mixed", kind="chi", dim=2, ns=64, beta=30.0, U=2.0, n_iv=30, n_iw=30, prec="mixed"),
        # the lowest temperature of the uneven scan: the largest matrices
        dict(name="chi 2d32 n120 mixed", kind="chi", dim=2, ns=32, beta=40.0, U=1.5, n_iv=60, n_iw=60, prec="mixed"),
        # a box size no configuration was tuned for, FP64 mode
        dict(name="chi 3d12 n34 fp64", kind="chi", dim=3, ns=12, beta=12.0, U=1.2, n_iv=17, n_iw=13, prec="fp64"),
        # one residual of the lambda correction at the headline box
        dict(name="sigma 3d32 n40", kind="sigma", dim=3, ns=32, beta=20.0, U=1.5, n_iv=20, n_iw=20, prec="mixed",
             lam_m=1.5, lam_d=0.0),
        # one residual of the 2-D lambda_dm Newton at its configuration's box
        dict(name="sigma 2d64 n60", kind="sigma", dim=2, ns=64, beta=30.0, U=2.0, n_iv=30, n_iw=30, prec="mixed",
             lam_m=2.0, lam_d=0.5),
        # gradient of a loss on Sigma_ladder with respect to both vertices and Sigma_loc
        dict(name="adjoint 2d48 n40", kind="adjoint", dim=2, ns=48, beta=20.0, U=1.5, n_iv=20, n_iw=20, prec="mixed",
             lam_m=1.0, lam_d=0.0),
    ]


def _nq(case):
    m = case["ns"] // 2 + 1
    return m * (m + 1) // 2 if case["dim"] == 2 else m * (m + 1) * (m + 2) // 6


def _cost(case):
    """Rough floating-point work of a case; bounds the drawn ones."""
    n, nw, nq = 2 * case["n_iv"], 2 * case["n_iw"] + 1, _nq(case)
    solve = 2 * nq * nw * n**3 if case["kind"] in ("chi", "chain", "adjoint") else 0
    return case.get("points", 1) * (solve + 400 * nq * nw * n)


def draw(rng):
    kind = rng.choice(("chain", "chain", "bubble", "chi", "chi", "chi", "sigma", "sigma", "adjoint"))
    top = max(_cost(c) for c in listed())
    while True:
        dim = rng.choice((2, 3))
        ns = rng.choice(NS[dim])
        n_iv = rng.choice(N_IV)
        if kind == "adjoint":       # the adjoint's solves are built for these boxes
            n_iv = rng.choice((4, 5, 6, 8, 10, 15, 20))
        n_iw = max(2, int(n_iv * rng.uniform(0.4, 1.1)))
        case = dict(kind=kind, dim=dim, ns=ns, n_iv=n_iv, n_iw=n_iw)
        if kind == "chain":
            case.update(beta=round(rng.uniform(5.0, 10.0), 2), U=round(rng.uniform(0.5, 2.0), 3),
                        prec=rng.choice(("mixed", "mixed", "fp64")), graph=rng.random() < 0.7,
                        points=rng.choice((1, 1, 3, 5)))
            case["n_iw"] = max(n_iv * 3 // 4, 4)
        else:
            case.update(beta=round(n_iv * rng.uniform(0.6, 1.0), 2), U=round(rng.uniform(0.5, 2.0), 3),
                        prec=rng.choice(("mixed", "fp64")))
        if kind in ("sigma", "adjoint"):
            case.update(lam_m=round(rng.uniform(0.0, 2.0), 3), lam_d=round(rng.choice((0.0, rng.uniform(0.0, 1.0))), 3))
        # host time of the inputs and the reference values bounds n_iv^3 n_iw per point as well
        if _cost(case) <= 0.7 * top and case["n_iv"] ** 3 * case["n_iw"] * case.get("points", 1) <= 60**3 * 61:
            return case


# ------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------
def _boxes(case):
    """(n_iv, n_iw) of every point: the given box, then smaller ones in turn."""
    out = []
    for p in range(case.get("points", 1)):
        f = (1.0, 0.5, 4.0 / 15.0)[p % 3]
        out.append((max(2, round(case["n_iv"] * f)), max(2, round(case["n_iw"] * f))))
    return out


def _gimp_at(inp, n):
    g = inp.gimp
    return np.where(n >= 0, g[np.maximum(n, 0)], np.conj(g[np.maximum(-n - 1, 0)]))


def _chi0_loc(inp, w):
    n = np.arange(2 * inp.n_iv) - inp.n_iv
    return -inp.beta * _gimp_at(inp, n) * _gimp_at(inp, n + w - inp.n_iw)


def _input(case, seed, point=0):
    """The impurity solution of one parameter point (sizes and scalars of the case, U shifted by the
    seed by at most 5 %, vertex noise from the seed)."""
    n_iv, n_iw = _boxes(case)[point]
    sd = (seed * 1009 + point * 77 + 13) & 0x7FFFFFFF
    U = case["U"] * (0.95 + 0.1 * float(S.uniform01(sd, 1)[0]))
    t = 1.0
    if case["kind"] == "chain":
        t = 0.25 if case["dim"] == 2 else T3
        U *= 1.0 - 0.08 * point
    inp = S.make_input(case["dim"], case["ns"], case["beta"], U, n_iv, n_iw, seed=sd, t=t)
    if case["kind"] != "chain":
        return inp
    nnu, nw = 2 * n_iv, 2 * n_iw + 1
    n = np.arange(nnu)
    g = S.complex_gaussian(sd + 1, nnu * nnu * nw).reshape((nnu, nnu, nw), order="F")
    g = g / (1.0 + np.abs(n[:, None] - n[None, :]))[:, :, None]
    g = 1.0 + 0.1 * (g + np.conj(g.transpose(1, 0, 2)))
    new = {}
    for r, s in (("m", -1.0), ("d", 1.0)):
        gam = np.asfortranarray((s * U / inp.beta**2) * g)
        chi = np.empty_like(gam)
        for w in range(nw):
            chi[:, :, w] = np.linalg.inv(gam[:, :, w] + np.diag(1.0 / _chi0_loc(inp, w)))
        new["gamma_" + r], new["chi_loc_" + r] = gam, chi
    return dataclasses.replace(inp, **new)


def _local_sums(inp):
    """(imp_density, sum_w of the local chi_m) with the 1/(i w)^2 tail of the kinetic energy."""
    b, c2 = inp.beta, inp.Ekin_DMFT
    xm, xd = (np.real(x.sum(axis=(0, 1))) / b**2 for x in (inp.chi_loc_m, inp.chi_loc_d))
    w = 2 * np.arange(-inp.n_iw, inp.n_iw + 1) * math.pi / b
    tail = np.where(w != 0, -c2 / np.where(w != 0, w, 1.0) ** 2, 0.0)
    return (float(np.sum(0.5 * (xm + xd) - tail) / b - c2 * b / 12), float(np.sum(xm - tail) / b - c2 * b / 12))


def _numax(case):
    """Fermionic frequencies of the self-energy: n_iv, or the lambda_dm correction's smaller box."""
    n = case["n_iv"]
    return n if case.get("lam_d", 0.0) == 0.0 else max(1, min(n, (3 * (2 * case["n_iw"] + 1)) // 8))


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a, dtype=np.complex128).reshape(-1, order="F"))).cuda()


def _pin(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a, dtype=np.complex128).reshape(-1, order="F"))).pin_memory()


def _p(t):
    return C.c_void_p(t.data_ptr())


def _arr(*shape, dtype=torch.complex128):
    """A device array of the library's layout: shape (slowest index first)."""
    return torch.zeros(shape, dtype=dtype, device="cuda")


def _upstream(case, inp, nq, numax):
    """dL/dSigma_ladder [nu, q] of a loss on Sigma_ladder: complex noise of the seed."""
    g = S.complex_gaussian(inp.seed + 5, nq * numax).reshape(numax, nq)
    return g / (1.0 + np.arange(numax))[:, None]


def prepare(case, seed):
    if case["kind"] == "chain":
        pts = []
        for p in range(case["points"]):
            inp = _input(case, seed, p)
            h = L.setup_synthetic(inp, precision=PREC[case["prec"]])
            ctx = h.ctx
            dens, msum = _local_sums(inp)
            src = [_pin(x) for x in (inp.sigma_loc, inp.gamma_m, inp.gamma_d, inp.chi_loc_m, h.gImp)]
            out = {"sigma": torch.zeros((inp.n_iv, ctx.Nq), dtype=torch.complex128).pin_memory(),
                   "chi_m": torch.zeros((ctx.Nw, ctx.Nq), dtype=torch.float64).pin_memory(),
                   "chi_d": torch.zeros((ctx.Nw, ctx.Nq), dtype=torch.float64).pin_memory()}
            sc = torch.zeros(8, dtype=torch.float64).pin_memory()
            io = _lib.ChainIO(src[0].data_ptr(), len(inp.sigma_loc), src[1].data_ptr(), src[2].data_ptr(),
                              src[3].data_ptr(), src[4].data_ptr(), len(h.gImp), dens, msum, out["sigma"].data_ptr(),
                              out["chi_m"].data_ptr(), out["chi_d"].data_ptr(), sc.data_ptr())
            # lambda_m, mu, E_kin, E_pot1, E_pot2, sum rule | filling (without the Newton's step count)
            res = dict(out, scalars=sc[:6], n=sc[7:])
            pts.append(dict(h=h, src=src, out=out, sc=sc, io=io, dens=dens, msum=msum, res=res))
        n = len(pts)
        return dict(case=case, pts=pts, ios=(_lib.ChainIO * n)(*[x["io"] for x in pts]),
                    handles=(C.c_void_p * n)(*[x["h"].ctx.h.value for x in pts]), status=(C.c_int32 * n)())
    inp = _input(case, seed)
    h = L.setup_synthetic(inp, precision=PREC[case["prec"]])
    ctx = h.ctx
    nq, nnu, nw, nf, numax = ctx.Nq, ctx.Nnu, ctx.Nw, ctx.Nf, _numax(case)
    st = dict(case=case, inp=inp, h=h, ctx=ctx, numax=numax, sums=_local_sums(inp))
    if case["kind"] == "bubble":
        st.update(sig=_dev(inp.sigma_loc), out=dict(G=_arr(nf, nq), chi0=_arr(nw, nnu, nq)))
    else:
        ctx.call("ldga_bubble", None)
        st["gam"] = [_dev(inp.gamma_m), _dev(inp.gamma_d)]
    if case["kind"] == "chi":
        st["out"] = {k + r: _arr(nw, nnu, nq) if k == "gamma_" else _arr(nw, nq, dtype=torch.float64)
                     for r in "md" for k in ("chi_", "gamma_")}
    if case["kind"] in ("sigma", "adjoint"):
        for ch in (L.CH_M, L.CH_D):
            ctx.call("ldga_bse", ch, _p(st["gam"][ch]), None, None, None)
        ctx.call("ldga_lambda0", None, None)
    if case["kind"] == "sigma":
        st["out"] = dict(lambda0=_arr(nw, nnu, nq), sigma=_arr(numax, nq), G=_arr(nf, nq))
    if case["kind"] == "adjoint":
        n_sigma = len(inp.sigma_loc)
        st.update(sbar=torch.from_numpy(_upstream(case, inp, nq, numax)).cuda().contiguous(),
                  out=dict(gamma_m=_arr(nw, nnu, nnu), gamma_d=_arr(nw, nnu, nnu), sigma_loc=_arr(n_sigma),
                           chi0=_arr(nw, nnu, nq)))
    torch.cuda.synchronize()
    return st


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "chain":
        pts, graph = state["pts"], int(case["graph"])
        if len(pts) == 1:
            x = pts[0]
            s, gm, gd, xl, gi = x["src"]
            x["h"].ctx.call("ldga_chain_m", _p(s), s.numel(), _p(gm), _p(gd), _p(xl), _p(gi), gi.numel(), x["dens"],
                            x["msum"], graph, *[_p(x["out"][k]) for k in ("sigma", "chi_m", "chi_d")], _p(x["sc"]))
        else:
            if _lib.load().ldga_batch_chain_m(len(pts), state["handles"], state["ios"], graph, state["status"]):
                raise RuntimeError("ldga_batch_chain_m failed")
        return [x["res"] for x in pts]
    ctx, out = state["ctx"], state["out"]
    if kind == "bubble":
        ctx.call("ldga_gloc", _p(state["sig"]), state["sig"].numel(), _p(out["G"]))
        ctx.call("ldga_bubble", _p(out["chi0"]))
        return out
    if kind == "chi":
        nf = C.c_int32()
        for ch, r in ((L.CH_M, "m"), (L.CH_D, "d")):
            ctx.call("ldga_bse", ch, _p(state["gam"][ch]), _p(out["chi_" + r]), _p(out["gamma_" + r]), C.byref(nf))
        return out
    if kind == "sigma":
        mu, ek, ep, n = (C.c_double() for _ in range(4))
        ctx.call("ldga_lambda0", None, _p(out["lambda0"]))
        ctx.call("ldga_eom", case["lam_m"], case["lam_d"], state["numax"], 1, state["sums"][1], _p(out["sigma"]))
        ctx.call("ldga_g_ladder", None, 0, 1, state["h"].mP.μ, C.byref(mu), _p(out["G"]), C.byref(ek), C.byref(ep),
                 C.byref(n))
        return dict(out, mu=mu.value, E_kin=ek.value, E_pot=ep.value, n=n.value)
    nf = C.c_int32()
    ctx.call("ldga_chain_vjp", _p(state["sbar"]), case["lam_m"], case["lam_d"], state["numax"], 1, _p(out["gamma_m"]),
             _p(out["gamma_d"]), out["sigma_loc"].numel(), _p(out["sigma_loc"]), _p(out["chi0"]), C.byref(nf))
    return out


def work(case):
    """Bytes: every input array read once and every output written once.  Flops: k-space convolutions as
    FFTs (5 N log2 N per transform), one LU solve (8/3 N^3 + 8 N^2) per (q, w) and channel."""
    tot = dict(bytes=0.0, flops=0.0)
    nk = case["ns"] ** case["dim"]
    fft = 5.0 * nk * math.log2(max(nk, 2))
    nq = _nq(case)
    for n_iv, n_iw in _boxes(case):
        n, nw = 2 * n_iv, 2 * n_iw + 1
        nf = 4 * (n_iv + n_iw) + 1
        qvw, vvw, qw = 16.0 * nq * n * nw, 16.0 * n * n * nw, 8.0 * nq * nw
        solve = nq * nw * (8.0 / 3.0 * n**3 + 8.0 * n**2)
        numax = n_iv if case["kind"] == "chain" else _numax(case)
        eom = (numax * nw + numax) * fft
        k = case["kind"]
        if k == "bubble":
            tot["bytes"] += 16.0 * nf * nq + qvw
            tot["flops"] += (nf + n * nw) * fft
        elif k == "chi":
            tot["bytes"] += 2 * (qvw + vvw + qw + qvw)
            tot["flops"] += 2 * solve
        elif k == "sigma":
            used = 16.0 * nq * numax * nw
            tot["bytes"] += vvw + 2 * qvw + 2 * qw + 3 * used + 16.0 * nq * (numax + 2 * nf)
            tot["flops"] += eom + 8.0 * nq * n * nw
        elif k == "adjoint":
            tot["bytes"] += 4 * qvw + 4 * vvw + 2 * qw
            tot["flops"] += 2 * solve + 2 * nq * nw * 8.0 * n * n + (2 * numax * nw + n * nw + 2 * nf) * fft
        else:
            tot["bytes"] += 3 * vvw + 2 * qw + 16.0 * nq * numax
            tot["flops"] += 2 * solve + (nf + n * nw) * fft + eom
    return tot


# ------------------------------------------------------------------------------------------------
# the same values in plain torch, complex128, on the full k-grid with FFTs
# ------------------------------------------------------------------------------------------------
class _Exact:
    def __init__(self, case, inp):
        self.case, self.inp = case, inp
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        d, ns = inp.dim, inp.ns
        self.d, self.ns, self.nk = d, ns, ns**d
        self.b, self.U, self.mu, self.n = inp.beta, inp.U, inp.mu, inp.n
        self.n_iv, self.n_iw = inp.n_iv, inp.n_iw
        self.nnu, self.nw = 2 * inp.n_iv, 2 * inp.n_iw + 1
        self.Lf = 2 * (inp.n_iv + inp.n_iw)
        k = 2.0 * math.pi * np.arange(ns) / ns
        c = [np.cos(k).reshape([-1 if a == i else 1 for a in range(d)]) for i in range(d)]
        eps = -2.0 * inp.t * sum(c) + np.zeros((ns,) * d)
        m = ns // 2 + 1
        wedge = ([(a, b) for a in range(m) for b in range(a + 1)] if d == 2 else
                 [(a, b, e) for a in range(m) for b in range(a + 1) for e in range(b + 1)])
        place = {w: i for i, w in enumerate(wedge)}
        fold = np.minimum(np.arange(ns), (ns - np.arange(ns)) % ns)
        grids = np.stack(np.meshgrid(*[fold] * d, indexing="ij"), -1).reshape(-1, d)
        full = np.array([place[tuple(sorted(x, reverse=True))] for x in grids.tolist()])
        self.full = torch.from_numpy(full).to(self.dev)
        irr = np.array([np.ravel_multi_index(w, (ns,) * d) for w in wedge])
        self.irr = torch.from_numpy(irr).to(self.dev)
        self.kmult = torch.from_numpy(np.bincount(full).astype(np.float64)).to(self.dev)
        self.eps = torch.from_numpy(eps.reshape(-1)).to(self.dev)
        self.eps_q = self.eps[self.irr]

    def t(self, a):
        a = np.asarray(a)
        if a.ndim == 3:
            a = a.transpose(2, 1, 0)        # Julia [nu, nu', w] -> [w, nu', nu]
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)

    def iv(self, n):
        return (2.0 * n + 1.0) * math.pi / self.b

    def fft(self, x):
        return torch.fft.fftn(x.reshape((-1,) + (self.ns,) * self.d), dim=tuple(range(1, self.d + 1)))

    def conv(self, ahat, bhat):
        """(1/N_k) sum_k A(k) B(k + q) of even functions, at the irreducible q."""
        y = torch.fft.ifftn(ahat * bhat, dim=tuple(range(1, self.d + 1)))
        return y.reshape(y.shape[0], -1)[:, self.irr] / self.nk

    def lattice(self, sigma_loc):
        n = torch.arange(-self.Lf, self.Lf + 1, device=self.dev)
        s = torch.where(n >= 0, sigma_loc[n.clamp(min=0)], sigma_loc[(-n - 1).clamp(min=0)].conj())
        z = torch.complex(torch.full_like(s.real, self.mu), self.iv(n.double())) - s
        return 1.0 / (z[:, None] - self.eps[None, :])            # [Nf, k]

    def bubble(self, ghat):
        v = torch.arange(self.nnu, device=self.dev) - self.n_iv + self.Lf
        out = []
        for w in range(self.nw):
            out.append(-self.b * self.conv(ghat[v], ghat[v + w - self.n_iw]))
        return torch.stack(out)                                   # [w, nu, q]

    def bse(self, gamma, chi0, s):
        """gamma [w, nu', nu] = Gamma[nu, nu', w]; the left solve 1^T A^-1."""
        chi, gam = [], []
        one = torch.ones(self.nnu, dtype=torch.complex128, device=self.dev)
        for w in range(self.nw):
            B = gamma[w][None] + torch.diag_embed(1.0 / chi0[w].T)   # A^T: rows nu', columns nu
            y = torch.linalg.solve(B, one.expand(B.shape[0], -1))
            x = y.sum(1).real / self.b**2
            chi.append(x)
            gam.append((y / (chi0[w].T * (1.0 + s * self.U * x)[:, None])).T)
        return torch.stack(chi), torch.stack(gam)

    def colsum_F(self):
        """sum over nu of F_m[nu, nu', w]."""
        inp, out = self.inp, []
        n = np.arange(self.nnu) - self.n_iv
        for w in range(self.nw):
            gg = _gimp_at(inp, n) * _gimp_at(inp, n + w - self.n_iw)
            num = inp.chi_loc_m[:, :, w] + np.diag(self.b * gg)
            out.append(-(num / gg[:, None] / gg[None, :]).sum(0))
        return self.t(np.stack(out))                              # [w, nu']

    def lambda0(self, chi0):
        return chi0 * self.colsum_F()[:, :, None] / self.b**2

    def sum_kw(self, chi):
        w = 2.0 * torch.arange(-self.n_iw, self.n_iw + 1, device=self.dev, dtype=torch.float64) * math.pi / self.b
        c2 = self.inp.Ekin_DMFT
        tail = torch.where(w != 0, -c2 / torch.where(w != 0, w, torch.ones_like(w)) ** 2, torch.zeros_like(w))
        return ((chi @ self.kmult / self.nk - tail).sum() - self.b**2 / 12 * c2) / self.b

    def sigma(self, xm, gm, xd, gd, l0, ghat, lam_m, lam_d, numax, msum):
        """Sigma_ladder [nu, q]."""
        U = self.U
        xm, xd = xm / (lam_m * xm + 1.0), xd / (lam_d * xd + 1.0)
        acc = 0.0
        v = self.n_iv + torch.arange(numax, device=self.dev)
        g0 = torch.arange(numax, device=self.dev) + self.Lf
        for w in range(self.nw):
            K = U * (gm[w][v] * 1.5 * (1.0 + U * xm[w]) - gd[w][v] * 0.5 * (1.0 - U * xd[w]) - 1.0 + l0[w][v])
            acc = acc + self.conv(self.fft(K[:, self.full]), ghat[g0 + w - self.n_iw])
        wn = self.iv(torch.arange(numax, device=self.dev, dtype=torch.float64))
        tail = -U * (self.sum_kw(xm) - msum) / (1j * wn)
        return acc / self.b + tail[:, None] + self.n * U / 2.0

    def lambda_m(self, xm, rhs):
        """The root of sum_kw(chi_m/(lam chi_m + 1)) = rhs between lam_min and the first pole."""
        lo = float(-(1.0 / xm[self.n_iw]).min())
        neg = xm[xm < 0]
        hi = float((-1.0 / neg).min()) if neg.numel() else 1e3
        f = lambda x: float(self.sum_kw(xm / (x * xm + 1.0))) - rhs  # noqa: E731
        a, b = lo, hi
        for _ in range(200):
            c = 0.5 * (a + b)
            a, b = (c, b) if f(c) > 0 else (a, c)
        return 0.5 * (a + b)

    def g_ladder(self, sig, numax, sigma_loc):
        """(mu, G_ladder [Nf, q], E_kin, E_pot, filling)."""
        b, U, n0 = self.b, self.U, self.n
        nn = torch.arange(numax, device=self.dev, dtype=torch.float64)
        w = self.iv(nn)
        N = numax + 1
        j = np.arange(N, 4_000_000, dtype=np.float64)
        # trigamma(N + 1/2) - trigamma(1/2 - N), trigamma(1/2 - N) = pi^2 - trigamma(N + 1/2)
        tri = float(np.sum(1.0 / (j + 0.5) ** 2)) + 1.0 / 4_000_000
        shell = (2.0 * tri - math.pi**2) * b / (4 * math.pi**2) + b / 4

        def fill(mu):
            z = torch.complex(torch.full_like(w, mu), w)[:, None] - self.eps_q[None] - sig
            g = 1.0 / z
            s, ds = (float((x @ self.kmult.to(torch.complex128)).sum().real) / self.nk for x in (g, -g * g))
            return (2 * (2 * s / b + 0.5 + mu * shell) / (1 + U * shell) - n0,
                    2 * (2 * ds / b + shell) / (1 + U * shell), g)

        mu = self.mu
        for _ in range(60):
            f, df, g = fill(mu)
            step = f / df
            mu -= step
            if abs(step) < 1e-15 * (1 + abs(mu)):
                break
        f, _, g = fill(mu)
        full = torch.arange(self.Lf + 1, device=self.dev, dtype=torch.float64)
        s_all = sigma_loc[: self.Lf + 1][:, None].expand(-1, sig.shape[1]).clone()
        s_all[:numax] = sig[: self.Lf + 1]
        gp = 1.0 / (torch.complex(torch.full_like(full, mu), self.iv(full))[:, None] - self.eps_q[None] - s_all)
        G = torch.cat([gp[: self.Lf].conj().flip(0), gp])
        har = n0 * U / 2
        e = self.eps_q
        ek_c, ep_c = e + har - mu, U * U * 0.5 * n0 * (1 - 0.5 * n0) + har * (e + har - mu)
        tail = (-1.0 / w**2)[:, None]
        ek = 4 * (e * (g.real - ek_c * tail)).sum(0) + b / 2 * e * (1 - b * ek_c)
        ep = 2 * ((g * sig).real - ep_c * tail).sum(0) + b / 2 * har - b * b / 4 * ep_c
        k = self.kmult / self.nk
        return mu, G, float((ek * k).sum()) / b, float((ep * k).sum()) / b, f + n0


def _exact_point(case, seed, point):
    """The lattice G, its transform and the bubble of one point."""
    inp = _input(case, seed, point)
    e = _Exact(case, inp)
    e.sl = e.t(inp.sigma_loc)
    e.G = e.lattice(e.sl)
    e.ghat = e.fft(e.G)
    e.chi0 = e.bubble(e.ghat)
    return e


def exact(case, seed):
    kind = case["kind"]
    if kind == "chain":
        res = []
        for p in range(case["points"]):
            e = _exact_point(case, seed, p)
            dens, msum = _local_sums(e.inp)
            xm, gm = e.bse(e.t(e.inp.gamma_m), e.chi0, 1.0)
            xd, gd = e.bse(e.t(e.inp.gamma_d), e.chi0, -1.0)
            xds = float(e.sum_kw(xd))
            lam = e.lambda_m(xm, 2.0 * dens - xds)
            sig = e.sigma(xm, gm, xd, gd, e.lambda0(e.chi0), e.ghat, lam, 0.0, e.n_iv, msum)
            mu, _, ek, ep, n = e.g_ladder(sig, e.n_iv, e.sl)
            xms = float(e.sum_kw(xm / (lam * xm + 1.0)))
            ep2 = e.U / 2 * (xds - xms) + e.U * e.n * e.n / 4
            res.append(dict(sigma=sig, chi_m=xm, chi_d=xd, n=torch.tensor([n], dtype=torch.float64),
                            scalars=torch.tensor([lam, mu, ek, ep, ep2, (xds + xms) / 2], dtype=torch.float64)))
        return res
    if kind == "bubble":
        e = _exact_point(case, seed, 0)
        return dict(G=e.G[:, e.irr], chi0=e.chi0)
    e = _exact_point(case, seed, 0)
    gam = [e.t(e.inp.gamma_m), e.t(e.inp.gamma_d)]
    if kind == "chi":
        out = {}
        for r, g, s in (("m", gam[0], 1.0), ("d", gam[1], -1.0)):
            out["chi_" + r], out["gamma_" + r] = e.bse(g, e.chi0, s)
        return out
    numax, msum = _numax(case), _local_sums(e.inp)[1]
    if kind == "sigma":
        xm, gm = e.bse(gam[0], e.chi0, 1.0)
        xd, gd = e.bse(gam[1], e.chi0, -1.0)
        l0 = e.lambda0(e.chi0)
        sig = e.sigma(xm, gm, xd, gd, l0, e.ghat, case["lam_m"], case["lam_d"], numax, msum)
        mu, G, ek, ep, n = e.g_ladder(sig, numax, e.sl)
        return dict(lambda0=l0, sigma=sig, G=G, mu=mu, E_kin=ek, E_pot=ep, n=n)
    # adjoint: reverse mode through the same chain; the gradient convention is dL/dRe + i dL/dIm
    e.sl.requires_grad_()
    for g in gam:
        g.requires_grad_()
    ghat = e.fft(e.lattice(e.sl))
    chi0 = e.bubble(ghat)
    chi0.retain_grad()
    xm, gm = e.bse(gam[0], chi0, 1.0)
    xd, gd = e.bse(gam[1], chi0, -1.0)
    sig = e.sigma(xm, gm, xd, gd, e.lambda0(chi0), ghat, case["lam_m"], case["lam_d"], numax, msum)
    sbar = torch.from_numpy(_upstream(case, e.inp, sig.shape[1], numax)).to(e.dev)
    (sbar.conj() * sig).real.sum().backward()
    return dict(gamma_m=gam[0].grad, gamma_d=gam[1].grad, sigma_loc=e.sl.grad, chi0=chi0.grad)
