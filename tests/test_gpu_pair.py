"""Both channels' Bethe-Salpeter solve in one launch (the chain) against one launch per channel.

Each matrix is solved by the same instructions in either launch, so chi_m and chi_d agree bit for bit
(tolerance 0).
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
