"""The Bethe-Salpeter step at box sizes without kernels of their own, which run on the next tile up (an
identity block below the box): around every tile edge, in every precision mode, against the oracle.

Tolerance: the parity bound of the other box sizes, relative 1e-10 (denominator max(|oracle|, 1e-6
max|oracle|)) for gamma and componentwise for chi: every solution is accepted at a backward error of 1e-12
(FP64) or 1e-14 (MIXED), and the matrices' condition numbers here stay below 1e2.
"""
import numpy as np
import pytest

import ladderdga_b200 as L
from ladderdga_b200 import synthetic as S
from oracle import ldga_ref as R

pytestmark = pytest.mark.gpu

RTOL = 1e-10


@pytest.mark.parametrize("n_iv", [1, 7, 9, 11, 13, 17, 19, 21, 23, 25, 27, 29, 31, 33, 39, 41, 47, 49, 55, 57])
def test_box_sizes_between_the_tiles(n_iv, require_gpu):
    inp = S.make_input(dim=2, ns=10, beta=max(4.0, 0.7 * n_iv), U=1.0, n_iv=n_iv, n_iw=1, seed=900 + n_iv)
    ref = R.run_chain(inp, lambda_type=None)
    beta2 = inp.beta ** 2
    for prec in (L.PREC_FP64, L.PREC_FP64_INV, L.PREC_MIXED):
        h = L.setup_synthetic(inp, precision=prec)
        chi0 = L.calc_bubble(h)
        for r, s in (("m", 1.0), ("d", -1.0)):
            x, g = L.calc_χγ(r, h, chi0)
            want = ref[f"gamma_{r}"]
            chi = ref[f"chi_{r}"].data
            y = want * ref["chi0"] * (1.0 + s * inp.U * chi)[:, None, :]
            scale = np.abs(y).sum(axis=1) / beta2
            assert float(np.max(np.abs(x.data - chi) / scale)) < RTOL, (prec, r)
            m = np.maximum(np.abs(want), 1e-6 * np.abs(want).max())
            assert float(np.max(np.abs(g.data - want) / m)) < RTOL, (prec, r)
