"""The k-space kernels with several vectors per CTA and several steps per CTA, at every grid size: the bubble and the
equation of motion against the FP64 oracle's full-grid FFTs.

The launches' shapes are restated here (TransformPlan, pairs_per_cta, eom_shape) so that each grid is run where a
CTA of the bubble takes several vectors, and the equation of motion at a number of nu (more than n_iv: the rest are
empty) whose CTAs take several steps of w with a smaller last one, if its plan has such.

Tolerance 1e-12 of the array's largest value: an axis sum of at most 33 terms is off by 33 u of the sum of absolute
values, three of them by 1.1e-14, two transforms by twice that; the inputs are a constant with 10 % noise, so
that sum stays below twice the largest result, and the sum over at most 121 w adds 121 u.
"""
import numpy as np
import pytest

import ladderdga_b200 as L
from ladderdga_b200 import _lib
from ladderdga_b200 import synthetic as S
from oracle import ldga_ref as R

pytestmark = pytest.mark.gpu

GRIDS = ([(2, n) for n in (2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 16, 17, 20, 21, 24, 25, 32, 33, 40, 41, 48, 49, 64)] +
         [(3, n) for n in (2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 16, 17, 20, 21, 24, 25, 32, 33)])
TOL = 1e-12


def up(a, b):
    return -(-a // b)


def plan(dim, ns):
    """(vectors per CTA, threads, bytes of a vector's buffers, wedge points)."""
    m = ns // 2 + 1
    p2 = m * (m + 1) // 2
    nq = p2 if dim == 2 else m * (m + 1) * (m + 2) // 6
    per = 16 * (nq + m * m if dim == 2 else max(nq, p2 * m) + m * p2)
    cols, best, beff = (m if dim == 2 else p2), 1, 0.0
    for k in range(1, 17):
        items, nt = 2 * k * cols, 32 * up(2 * k * cols, 32)
        if k > 1 and (nt > 320 or k * per > 112 * 1024):
            break
        eff = items / nt * (0.5 if nt < 96 else 1.0)
        if eff > beff + 0.02:
            best, beff = k, eff
    nt_i = 32 * up(2 * best * cols, 32)
    nt_l = 32 * up(up(best * nq, 3 if dim == 3 else 4), 32)
    return best, nt_l if nt_i < nt_l <= 352 else nt_i, per, nq


def eom_shape(dim, ns, numax, nw):
    """(w per CTA, vectors per step)."""
    npm, nt, per, nq = plan(dim, ns)
    best, bt = (1, 1), 1e300
    for k in range(1, npm + 1):
        slots = 148 * max(1, min((704 if dim == 3 else 640) // nt, 227 * 1024 // (k * per + 16 * nq + 2048)))
        for w in range(k, max(nw, k) + 1):
            t = up(numax * up(nw, w), slots) * (up(w, k) * (1.0 + 0.5 * k) + 0.5)
            if t < bt:
                best, bt = (w, k), t
    return best


def far(a, b):
    return float(np.max(np.abs(np.asarray(a) - np.asarray(b))) / np.max(np.abs(np.asarray(b))))


def box(dim, ns):
    """The smallest of a few boxes, and the numbers of nu, where a CTA of the EoM takes several steps of w, the last
    with fewer vectors if the plan has more than one (the 2 and 3 point grids: several vectors in one step)."""
    npm = plan(dim, ns)[0]
    for n_iv, n_iw in ((12, 17), (20, 20), (25, 25), (30, 30), (40, 40), (50, 60), (60, 60)):
        nw = 2 * n_iw + 1
        for k in range(1, 2 * n_iv + 1):
            w, v = eom_shape(dim, ns, k, nw)
            if w > v and (npm == 1 or v > 1 and (w % v or nw % w % v)):
                return n_iv, n_iw, k
    return 60, 60, 120


@pytest.mark.parametrize("dim,ns", GRIDS)
def test_several_vectors_and_steps(dim, ns, require_gpu):
    n_iv, n_iw, numax = box(dim, ns)
    nnu, nw = 2 * n_iv, 2 * n_iw + 1
    npm, _, _, nq = plan(dim, ns)
    w, v = eom_shape(dim, ns, numax, nw)
    assert (w > v if ns > 3 else w > 1) and (v > 1 or npm == 1), (w, v)
    assert min(npm, up(nnu * nw // 2, 148)) > 1 or npm == 1       # the bubble's vectors per CTA
    inp = S.make_input(dim=dim, ns=ns, beta=10.0, U=1.0, n_iv=n_iv, n_iw=n_iw, seed=1000 + ns)
    h = L.setup_synthetic(inp)
    ctx = h.ctx
    assert ctx.Nq == nq
    kG = R.KGrid(dim, ns, inp.t)
    mP = R.ModelParameters(inp.U, inp.mu, inp.beta, inp.n, inp.sVk, inp.Epot_DMFT, inp.Ekin_DMFT)
    sP = R.SimulationParameters(n_iw, n_iv, 0, inp.shift, None, inp.fft_range, 0.0, False)
    ghat, grhat = R.G_fft(kG, R.lattice_G(kG, inp.sigma_loc, mP, sP.fft_range))
    some = (0, n_iw - 1, n_iw, nw - 2)
    want = R.calc_bubble(ghat, grhat, kG, mP, sP, w_subset=some)
    got = np.asarray(L.calc_bubble(h).data)
    for i in some:
        assert far(got[:, :, i], want[:, :, i]) < TOL, i
    rng = np.random.default_rng(ns)

    def noisy(*shape):
        return np.asfortranarray(1.0 + 0.1 * (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)))

    chi = {r: np.asfortranarray(noisy(nq, nw).real) for r in "md"}
    gam, l0 = {r: noisy(nq, nnu, nw) for r in "md"}, noisy(nq, nnu, nw)
    for ch, r in ((_lib.CH_M, "m"), (_lib.CH_D, "d")):
        ctx.call("ldga_set_chi", ch, _lib.ptr(chi[r]))
        ctx.call("ldga_set_gamma", ch, _lib.ptr(gam[r]))
    ctx.call("ldga_set_lambda0", _lib.ptr(l0))
    x = {r: R.ChiT(chi[r], mP.beta, tail_c=[0, 0, mP.Ekin_DMFT]) for r in "md"}
    for n in sorted({numax, min(numax, n_iv)}):
        out = _lib.cplx_out((nq, n))
        ctx.call("ldga_eom", 0.0, 0.0, n, 1, 0.3, _lib.ptr(out))
        want = R.calc_Sigma(x["m"], gam["m"], x["d"], gam["d"], 0.3, l0, grhat, kG, mP, sP, n)
        assert far(out, want) < TOL, (n, eom_shape(dim, ns, n, nw))
