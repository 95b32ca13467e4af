"""Both channels' Bethe-Salpeter solve in one launch (the chain) against one launch per channel, and the list
of matrices that a launch hands to the pivoted solve.

Each matrix is solved by the same instructions in either launch, so chi_m and chi_d agree bit for bit
(tolerance 0).  A matrix whose first pivot is zero (Gamma chosen to cancel 1/chi0 there; the matrix itself
is well conditioned, its 2 x 2 block is [[0, a], [a, b]]) reaches the pivoted solve by the list in either
launch, and agrees with a dense solve in numpy to 1e-10 of sum |y| / beta^2.
"""
import ctypes as C

import numpy as np
import pytest

import ladderdga_b200 as L
from ladderdga_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def chain_chi(h):
    import torch

    def pinned(a):
        v = np.ascontiguousarray(np.asarray(a, dtype=np.complex128).reshape(-1, order="F")).view(np.float64)
        return torch.from_numpy(v.copy()).pin_memory()

    c = h.ctx
    src = [pinned(a) for a in (h.Σ_loc, h.Γ_m, h.Γ_d, h.χDMFT_m, h.gImp)]
    S_out = torch.zeros(c.Nq * h.sP.n_iν * 2, dtype=torch.float64).pin_memory()
    x = [torch.zeros(c.Nq * c.Nw, dtype=torch.float64).pin_memory() for _ in "md"]
    p = [C.c_void_p(t.data_ptr()) for t in src]
    c.call("ldga_chain_m", p[0], len(h.Σ_loc), p[1], p[2], p[3], p[4], len(h.gImp), h.imp_density, h.χloc_m_sum, 0,
           C.c_void_p(S_out.data_ptr()), C.c_void_p(x[0].data_ptr()), C.c_void_p(x[1].data_ptr()), (C.c_double * 8)())
    return {r: t.numpy().reshape((c.Nq, c.Nw), order="F") for r, t in zip("md", x)}


@pytest.mark.parametrize("prec", [L.PREC_FP64, L.PREC_MIXED])
@pytest.mark.parametrize("n_iv", [1, 2, 5, 8, 10, 13, 15, 20, 22, 30, 33, 50])
def test_both_channels_in_one_launch(n_iv, prec, require_gpu):
    inp = S.make_input(dim=2, ns=8, beta=max(4.0, 0.7 * n_iv), U=1.0, n_iv=n_iv, n_iw=2, seed=700 + n_iv)
    step = L.setup_synthetic(inp, precision=prec)
    chi0 = L.calc_bubble(step)
    want = {r: np.array(L.calc_χγ(r, step, chi0)[0].data) for r in "md"}
    got = chain_chi(L.setup_synthetic(inp, precision=prec))
    for r in "md":
        assert np.array_equal(got[r], want[r]), r


@pytest.mark.parametrize("prec", [L.PREC_FP64, L.PREC_MIXED])
@pytest.mark.parametrize("n_iv", [2, 10, 20, 22])
def test_zero_pivot_reaches_the_pivoted_solve(n_iv, prec, require_gpu):
    inp = S.make_input(dim=2, ns=8, beta=max(4.0, 0.7 * n_iv), U=1.0, n_iv=n_iv, n_iw=2, seed=720 + n_iv)
    h = L.setup_synthetic(inp, precision=prec)
    chi0 = L.calc_bubble(h)
    c0 = np.asarray(chi0.data if hasattr(chi0, "data") else chi0)
    q0, w0 = 1, 0                                             # an edge frequency
    a = 1.0 / c0[q0, 0, w0]
    for G in (h.Γ_m, h.Γ_d):
        G[0, 0, w0] = -a
        G[0, 1, w0] = G[1, 0, w0] = a
    want = {}
    for r in "md":
        x, _ = L.calc_χγ(r, h, chi0)
        want[r] = np.array(x.data)
        if n_iv <= 15 or prec == L.PREC_FP64:                 # the iterations (MIXED above 30) need no pivot
            assert x.n_fallback >= 1, r
        G = h.Γ_m if r == "m" else h.Γ_d
        y = np.linalg.solve(G[:, :, w0].T + np.diag(1.0 / c0[q0, :, w0]), np.ones(G.shape[0]))
        b2 = inp.beta ** 2
        assert abs(want[r][q0, w0] - y.sum().real / b2) < 1e-10 * np.abs(y).sum() / b2, r
    h2 = L.setup_synthetic(inp, precision=prec)
    for G2, G in ((h2.Γ_m, h.Γ_m), (h2.Γ_d, h.Γ_d)):
        G2[:] = G
    got = chain_chi(h2)
    for r in "md":
        assert np.array_equal(got[r], want[r]), r
