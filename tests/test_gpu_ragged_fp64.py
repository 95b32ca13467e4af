"""MIXED at box sizes without kernels of their own solves in FP64, by the same elimination as the FP64 mode.

The two modes' chi and gamma agree bit for bit (tolerance 0), one channel at a time and both together.
"""
import ctypes as C

import numpy as np
import pytest

import ladderdga_b200 as L
from ladderdga_b200 import _lib
from ladderdga_b200 import synthetic as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_iv", [1, 9, 17, 21, 23, 25, 27, 29, 31, 33, 47])
def test_mixed_is_fp64_between_the_tiles(n_iv, require_gpu):
    inp = S.make_input(dim=2, ns=10, beta=max(4.0, 0.7 * n_iv), U=1.0, n_iv=n_iv, n_iw=2, seed=930 + n_iv)
    got = {}
    for prec in (L.PREC_FP64, L.PREC_MIXED):
        h = L.setup_synthetic(inp, precision=prec)
        chi0 = L.calc_bubble(h)
        got[prec] = [a for r in "md" for x, g in [L.calc_χγ(r, h, chi0)] for a in (np.array(x.data), np.array(g.data))]
        x = [np.zeros((h.ctx.Nq, h.ctx.Nw), order="F") for _ in "md"]
        h.ctx.call("ldga_chain_m", _lib.ptr(_lib.as_fc(h.Σ_loc)), len(h.Σ_loc), _lib.ptr(_lib.as_fc(h.Γ_m)),
                   _lib.ptr(_lib.as_fc(h.Γ_d)), _lib.ptr(_lib.as_fc(h.χDMFT_m)), _lib.ptr(_lib.as_fc(h.gImp)),
                   len(h.gImp), h.imp_density, h.χloc_m_sum, 0, None, _lib.ptr(x[0]), _lib.ptr(x[1]), (C.c_double * 8)())
        got[prec] += x
    for a, b in zip(got[L.PREC_FP64], got[L.PREC_MIXED]):
        assert np.array_equal(a, b)
