"""The grouped iteration (MIXED, Nnu = 60) over its splits into groups: of 32 q where the launch leaves SMs idle, of 64
elsewhere, the last group smaller; every matrix through the list of the pivoted solve; shards of the w.

Tolerance: solutions are accepted at a backward error of 1e-14 of their rows' norm (pivoted: 1e-15), so the error is
at most 2 kappa 1e-14 of the largest component, kappa the matrix's condition number, and rebuilding y
from gamma adds a few roundings (16 u).  A matrix has the same group in a shard: equal bits (tolerance 0); in a launch of one channel
and of both the groups are the same, and the bits, but where only the former has groups of 32 (the sum over y is then
off by at most the two solutions' errors).
"""
import ctypes as C

import numpy as np
import pytest

import ladderdga_b200 as L
from ladderdga_b200 import _lib
from ladderdga_b200 import synthetic as S

pytestmark = pytest.mark.gpu


# q x w: 15 x 3 (two warps), 28 x 5, 66 x 3 (three of 22), 66 x 51 (two of 33), 84 x 3, 153 x 3 (five of 31),
# 153 x 17 (five of 31, both channels three of 51), 153 x 31 (three of 51), 231 x 37 (four of 58)
@pytest.mark.parametrize("dim,ns,n_iw,sweeps", [(2, 8, 1, None), (2, 12, 2, None), (2, 20, 1, None), (2, 20, 25, None),
                                                (3, 12, 1, None), (2, 32, 1, None), (2, 32, 8, None), (2, 32, 15, None),
                                                (2, 40, 18, None), (2, 20, 1, "0"), (2, 32, 15, "0")])
def test_every_split(dim, ns, n_iw, sweeps, require_gpu, monkeypatch):
    if sweeps is not None:
        monkeypatch.setenv("LDGA_ITER_SWEEPS", sweeps)
    L.tune_reset()
    inp = S.make_input(dim=dim, ns=ns, beta=22.0, U=1.0, n_iv=30, n_iw=n_iw, seed=990 + ns)
    h = L.setup_synthetic(inp, precision=L.PREC_MIXED)
    ctx = h.ctx
    assert _lib.load().ldga_bse_config(ctx.h) == b"iterg64"
    chi0 = L.calc_bubble(h)
    c0 = np.asarray(chi0.data if hasattr(chi0, "data") else chi0)
    rng, one, bound = np.random.default_rng(ns), {}, {}
    for r, s in (("m", 1.0), ("d", -1.0)):
        x, g = L.calc_χγ(r, h, chi0)
        if sweeps is not None:
            assert x.n_fallback == ctx.Nq * ctx.Nw, r
        one[r] = np.array(x.data)
        G = h.Γ_m if r == "m" else h.Γ_d
        bound[r] = 0.0                # of the error of sum y: 60 components, both solutions'
        for w in range(ctx.Nw) if (ns, n_iw) == (32, 8) else ():
            B = G[:, :, w].T + np.einsum("qi,ij->qij", 1 / c0[:, :, w], np.eye(60))
            y = np.abs(g.data[:, :, w] * c0[:, :, w] * (1 + s * inp.U * x.data[:, w])[:, None]).max(axis=1)
            bound[r] = max(bound[r], float((120 * 2e-14 * np.linalg.cond(B, np.inf) * y).max()))
        for w in sorted({0, ctx.Nw // 2, ctx.Nw - 1}):
            for q in {0, ctx.Nq - 1, *rng.choice(ctx.Nq, min(ctx.Nq, 12), replace=False).tolist()}:
                B = G[:, :, w].T + np.diag(1 / c0[q, :, w])
                y = np.linalg.solve(B, np.ones(60))
                got = g.data[q, :, w] * c0[q, :, w] * (1 + s * inp.U * x.data[q, w])
                tol = 2e-14 * np.linalg.cond(B, np.inf) + 16 * 1.2e-16
                assert np.abs(got - y).max() < tol * np.abs(y).max(), (r, q, w)
    if sweeps is not None:
        return
    for lo, hi in ((0, 1), (1, ctx.Nw)):
        ctx.call("ldga_set_omega_shard", lo, hi, 1)
        for ch in (_lib.CH_M, _lib.CH_D):
            ctx.call("ldga_bse", ch, None, None, None, None)
    ctx.call("ldga_set_omega_shard", 0, ctx.Nw, 1)
    for ch, r in ((_lib.CH_M, "m"), (_lib.CH_D, "d")):
        out = np.zeros((ctx.Nq, ctx.Nw), order="F")
        ctx.call("ldga_get", 1, ch, _lib.ptr(out))
        assert np.array_equal(out, one[r]), r
    x = [np.zeros((ctx.Nq, ctx.Nw), order="F") for _ in "md"]
    ctx.call("ldga_chain_m", _lib.ptr(_lib.as_fc(h.Σ_loc)), len(h.Σ_loc), _lib.ptr(_lib.as_fc(h.Γ_m)),
             _lib.ptr(_lib.as_fc(h.Γ_d)), _lib.ptr(_lib.as_fc(h.χDMFT_m)), _lib.ptr(_lib.as_fc(h.gImp)), len(h.gImp),
             h.imp_density, h.χloc_m_sum, 0, None, _lib.ptr(x[0]), _lib.ptr(x[1]), (C.c_double * 8)())
    for a, r in zip(x, "md"):
        if (ns, n_iw) != (32, 8):
            assert np.array_equal(a, one[r]), r
        else:
            assert np.abs(a - one[r]).max() < bound[r] / inp.beta**2, r
