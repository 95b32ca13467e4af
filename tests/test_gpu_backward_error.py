"""MIXED by the preconditioned iterations: Nnu = 30 on grids with many q, as accurate as the elimination with refinement
that small grids keep, and the grouped iteration of Nnu = 60, also where it needs many sweeps.

The backward error of every solution, |1 - B y| / (|B| |y| + 1) with y rebuilt from gamma, is formed in extended
precision.  Tolerance: the iterations go on to 1e-15 and 4e-15; y = gamma chi0 (1 + s U chi) and gamma's own three
products are off by at most 8 u of |y|, which enters |1 - B y| with the factor |B|.
"""
import numpy as np
import pytest

import ladderdga_b200 as L
from ladderdga_b200 import synthetic as S

pytestmark = pytest.mark.gpu

STOP = {15: 1e-15, 30: 4e-15}


def rpa(inp, seed):
    """A local vertex of one sign with 20 % noise: rows of one size, so that errors do not average out."""
    nnu, nw = 2 * inp.n_iv, 2 * inp.n_iw + 1
    n = np.arange(nnu)
    g = S.complex_gaussian(seed, nnu * nnu * nw).reshape((nnu, nnu, nw), order="F")
    g = g / (1.0 + np.abs(n[:, None] - n[None, :]))[:, :, None]
    return (inp.U / inp.beta**2) * (1.0 + 0.1 * (g + np.conj(g.transpose(1, 0, 2))))


@pytest.mark.parametrize("n_iv,dim,ns", [(15, 2, 32), (15, 3, 16), (15, 2, 48), (30, 2, 16), (30, 2, 32), (30, 2, 48),
                                         (30, 3, 12)])
@pytest.mark.parametrize("vertex", ["noise", "rpa"])
def test_backward_error(n_iv, dim, ns, vertex, require_gpu):
    t = 1.0 if vertex == "noise" else (0.25 if dim == 2 else 0.2041241452319315)
    inp = S.make_input(dim=dim, ns=ns, beta=0.75 * n_iv if vertex == "noise" else 8.0, U=1.5, n_iv=n_iv, n_iw=3,
                       seed=950 + ns, t=t)
    h = L.setup_synthetic(inp, precision=L.PREC_MIXED)
    if vertex == "rpa":
        g = rpa(inp, 951 + ns)
        h.Γ_m[:], h.Γ_d[:] = -g, g
    chi0 = L.calc_bubble(h)
    c0 = np.asarray(chi0.data if hasattr(chi0, "data") else chi0)
    rng = np.random.default_rng(ns)
    for r, s in (("m", 1.0), ("d", -1.0)):
        x, g = L.calc_χγ(r, h, chi0)
        G = h.Γ_m if r == "m" else h.Γ_d
        for w in range(c0.shape[2]):
            q = rng.choice(c0.shape[0], min(60, c0.shape[0]), replace=False)
            d = 1 / c0[q, :, w].astype(np.clongdouble)
            y = g.data[q, :, w] * c0[q, :, w].astype(np.clongdouble) * (1 + s * inp.U * x.data[q, w])[:, None]
            B = G[:, :, w].T.astype(np.clongdouble)
            res = np.abs(1 - (y @ B.T + d * y)).max(axis=1)
            row = np.abs(B[None] + np.eye(2 * n_iv)[None] * d[:, :, None]).sum(axis=2).max(axis=1)
            assert float((res / (row * np.abs(y).max(axis=1) + 1)).max()) < STOP[n_iv] + 8 * 1.2e-16, (r, w)
