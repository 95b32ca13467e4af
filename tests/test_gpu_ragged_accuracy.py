"""Box sizes without kernels of their own at a matrix with a small pivot: as accurate as a pivoted elimination.

Gamma makes the first pivot of one (q, w) 1e-5 of its neighbours; the matrix itself has a condition number
kappa below 1e2.  An elimination without pivoting is off by up to 1e-12 there, so the matrix has to
reach the pivoted solve.  The solution, rebuilt from gamma, is compared with an 80-bit elimination.

Tolerance: a solution is accepted at a backward error eta = max(2.2e-16, 5.5e-17 sqrt(Nnu)) of its rows'
norm, so its error is at most 2 kappa eta of the largest component, and rebuilding it from gamma
adds a few roundings (16 u).
"""
import numpy as np
import pytest

import ladderdga_b200 as L
from ladderdga_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def solve80(B):
    """B y = 1 by partial pivoting in extended precision."""
    n = len(B)
    A = np.concatenate([B.astype(np.clongdouble), np.ones((n, 1), np.clongdouble)], axis=1)
    for k in range(n):
        p = k + int(np.argmax(np.abs(A[k:, k])))
        A[[k, p]] = A[[p, k]]
        A[k + 1:] -= (A[k + 1:, k] / A[k, k])[:, None] * A[k]
    y = np.zeros(n, np.clongdouble)
    for k in range(n - 1, -1, -1):
        y[k] = (A[k, n] - A[k, k + 1:n] @ y[k + 1:]) / A[k, k]
    return y


@pytest.mark.parametrize("prec", [L.PREC_FP64, L.PREC_FP64_INV, L.PREC_MIXED])
@pytest.mark.parametrize("n_iv", [1, 7, 9, 17, 21, 25, 31, 33, 47, 55])
def test_small_pivot_between_the_tiles(n_iv, prec, require_gpu):
    inp = S.make_input(dim=2, ns=8, beta=max(4.0, 0.7 * n_iv), U=1.0, n_iv=n_iv, n_iw=2, seed=740 + n_iv)
    h = L.setup_synthetic(inp, precision=prec)
    chi0 = L.calc_bubble(h)
    c0 = np.asarray(chi0.data if hasattr(chi0, "data") else chi0)
    q0, w0 = 1, 0
    a = 1.0 / c0[q0, 0, w0]
    for G in (h.Γ_m, h.Γ_d):
        G[0, 0, w0] = -a * (1.0 - 1e-5)
        G[0, 1, w0] = G[1, 0, w0] = a
    for r, s in (("m", 1.0), ("d", -1.0)):
        x, g = L.calc_χγ(r, h, chi0)
        G = h.Γ_m if r == "m" else h.Γ_d
        B = G[:, :, w0].T.astype(np.clongdouble) + np.diag(1 / c0[q0, :, w0].astype(np.clongdouble))
        want = solve80(B)
        got = g.data[q0, :, w0] * c0[q0, :, w0] * (1.0 + s * inp.U * x.data[q0, w0])
        eta = max(2.2e-16, 5.5e-17 * np.sqrt(2 * n_iv))
        tol = 2 * np.linalg.cond(B.astype(complex), np.inf) * eta + 16 * 1.1e-16
        assert float(np.abs(got - want).max() / np.abs(want).max()) < tol, r
        assert x.n_fallback >= 1, r
