"""The k-space transform at every grid size it is built for: the bubble and the equation of motion through
the C ABI against the FP64 oracle's full-grid FFTs.

The transform folds a column by its period's factors of two, so every N has its own split (odd N: no
fold; N = 2 odd, 4, 8, ... : one more level each), its own vectors per CTA and threads, and the EoM's
split of w over CTAs depends on the number of nu and w: odd counts leave remainders everywhere.

Tolerance 1e-12 of the array's largest value: each of the d <= 3 axis sums has at most 33 terms, so a
transform's error is below 3 * 33 unit roundoffs (1.1e-14) of the sum of absolute values, two transforms
and the product double it, and on these inputs that sum exceeds the result's largest value by less than 30.
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


def far(a, b):
    return float(np.max(np.abs(np.asarray(a) - np.asarray(b))) / np.max(np.abs(np.asarray(b))))


@pytest.mark.parametrize("dim,ns", GRIDS)
def test_bubble_and_eom_on_every_grid(dim, ns, require_gpu):
    n_iv, n_iw = (3, 2) if ns % 2 else (4, 3)
    inp = S.make_input(dim=dim, ns=ns, beta=6.0, U=1.0, n_iv=n_iv, n_iw=n_iw, seed=700 + ns)
    ref = R.run_chain(inp, lambda_type=None)
    h = L.setup_synthetic(inp)
    ctx = h.ctx
    chi0 = L.calc_bubble(h)
    assert far(chi0.data, ref["chi0"]) < TOL
    # the EoM alone: the oracle's arrays in, two numbers of nu (another split over CTAs each)
    for ch, r in ((_lib.CH_M, "m"), (_lib.CH_D, "d")):
        ctx.call("ldga_set_chi", ch, _lib.ptr(np.asfortranarray(ref[f"chi_{r}"].data)))
        ctx.call("ldga_set_gamma", ch, _lib.ptr(_lib.as_fc(ref[f"gamma_{r}"])))
    ctx.call("ldga_set_lambda0", _lib.ptr(_lib.as_fc(ref["lambda0"])))
    rh = ref["h"]
    for numax in (1, n_iv):
        out = _lib.cplx_out((ctx.Nq, numax))
        ctx.call("ldga_eom", 0.0, 0.0, numax, 1, rh.chiloc_m_sum, _lib.ptr(out))
        want = R.calc_Sigma(ref["chi_m"], ref["gamma_m"], ref["chi_d"], ref["gamma_d"], rh.chiloc_m_sum,
                            ref["lambda0"], rh.grhat, rh.kG, rh.mP, rh.sP, numax)
        assert far(out, want) < TOL, numax
