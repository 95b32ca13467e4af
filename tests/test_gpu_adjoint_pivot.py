"""The Bethe-Salpeter adjoint at a matrix whose unpivoted elimination meets a zero pivot.

Gamma is chosen to cancel 1/chi0 at one (q, w), in the first row (the exact zero first pivot of
tests/test_gpu_pair.py); the matrix itself is well conditioned.  The gradients at that w are compared with
the same formulas on dense numpy solves.

Tolerance 1e-9 of the largest value: a solve is accepted at a backward error of 1e-12 (pivoted: a few
roundings), the condition numbers here stay below 1e2, and a gradient holds two solutions and three
factors that are at most a few roundings off.
"""
import ctypes as C

import numpy as np
import pytest

import ladderdga_b200 as L
from ladderdga_b200 import _lib
from ladderdga_b200 import synthetic as S

pytestmark = pytest.mark.gpu


def reference(G, c0, chi, gam, beta, U, s, xbar, gbar):
    """Gamma_bar [Nnu, Nnu] and chi0_bar [Nq, Nnu] at one w: G [Nnu, Nnu], c0, gam, gbar [Nq, Nnu], chi, xbar [Nq]."""
    n = G.shape[0]
    Gb, cb = np.zeros((n, n), complex), np.zeros_like(c0)
    for q in range(c0.shape[0]):
        d, rf = 1.0 / c0[q], 1.0 / (1.0 + s * U * chi[q])
        y = gam[q] * c0[q] / rf
        x = xbar[q] - s * U * rf**2 * np.sum((np.conj(gbar[q]) * y * d).real)
        yb = np.conj(d * rf) * gbar[q] + x / beta**2
        z = np.conj(np.linalg.solve(G + np.diag(d), np.conj(yb)))
        Gb -= np.outer(np.conj(y), z)
        cb[q] = -np.conj(d * d) * (np.conj(y * rf) * gbar[q] - z * np.conj(y))
    return Gb, cb


@pytest.mark.parametrize("n_iv,prec,sweeps", [(2, L.PREC_FP64, None), (10, L.PREC_FP64, None), (20, L.PREC_FP64, None),
                                              (30, L.PREC_FP64, None), (10, L.PREC_MIXED, None),
                                              (20, L.PREC_MIXED, "0")])
def test_adjoint_at_a_zero_pivot(n_iv, prec, sweeps, require_gpu, monkeypatch):
    if sweeps is not None:          # the iteration hands every matrix to the LU adjoint
        monkeypatch.setenv("LDGA_ITER_SWEEPS", sweeps)
    inp = S.make_input(dim=2, ns=8, beta=max(4.0, 0.7 * n_iv), U=1.0, n_iv=n_iv, n_iw=2, seed=720 + n_iv)
    h = L.setup_synthetic(inp, precision=prec)
    chi0 = L.calc_bubble(h)
    c0 = np.asarray(chi0.data if hasattr(chi0, "data") else chi0)
    q0, w0 = 1, 0
    a = 1.0 / c0[q0, 0, w0]
    for G in (h.Γ_m, h.Γ_d):
        G[0, 0, w0] = -a
        G[0, 1, w0] = G[1, 0, w0] = a
    ctx, rng = h.ctx, np.random.default_rng(n_iv)
    nq, nnu, nw = c0.shape
    for ch, r, s in ((_lib.CH_M, "m", 1.0), (_lib.CH_D, "d", -1.0)):
        G = h.Γ_m if r == "m" else h.Γ_d
        x, g = L.calc_χγ(r, h, chi0)
        xbar = np.asfortranarray(rng.standard_normal((nq, nw)))
        gbar = np.asfortranarray(rng.standard_normal((nq, nnu, nw)) + 1j * rng.standard_normal((nq, nnu, nw)))
        Gb, cb = _lib.cplx_out((nnu, nnu, nw)), _lib.cplx_out((nq, nnu, nw))
        nf = C.c_int32(-1)
        ctx.call("ldga_bse_vjp", ch, _lib.ptr(xbar), _lib.ptr(gbar), _lib.ptr(Gb), _lib.ptr(cb), C.byref(nf))
        assert nf.value == 0, r
        assert np.isfinite(Gb).all() and np.isfinite(cb).all(), r
        want_G, want_c = reference(G[:, :, w0], c0[:, :, w0], x.data[:, w0], g.data[:, :, w0], inp.beta, inp.U, s,
                                   xbar[:, w0], gbar[:, :, w0])
        assert np.abs(Gb[:, :, w0] - want_G).max() < 1e-9 * np.abs(want_G).max(), r
        assert np.abs(cb[:, :, w0] - want_c).max() < 1e-9 * np.abs(want_c).max(), r
