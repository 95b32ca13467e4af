"""The Bethe-Salpeter configuration of an untuned MIXED handle at Nnu = 30, on both sides of the line where the
default changes: what ldga_bse_config names, and the results of what runs, against the oracle.

Tolerance: the parity bound of the box sizes, relative 1e-10 (denominator max(|oracle|, 1e-6 max|oracle|)) for
gamma and 1e-10 of sum |y| / beta^2 for chi: solutions are accepted at a backward error of 1e-12, and the
matrices' condition numbers stay below 1e2.
"""
import numpy as np
import pytest

import ladderdga_b200 as L
from ladderdga_b200 import _lib
from ladderdga_b200 import synthetic as S
from oracle import ldga_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,ns,name", [(2, 24, "warp:1"), (2, 25, "warp:1"), (3, 12, "warp:1"),
                                         (2, 32, "iter8x2dm2ns32:3"), (2, 33, "iter8x2dm2ns32:3"),
                                         (3, 16, "iter8x2dm2ns32:3")])
def test_default_configuration_at_box_30(dim, ns, name, require_gpu, tmp_path):
    L.tune_reset()
    inp = S.make_input(dim=dim, ns=ns, beta=10.0, U=1.0, n_iv=15, n_iw=1, seed=970 + ns)
    h = L.setup_synthetic(inp, precision=L.PREC_MIXED)
    lib = _lib.load()
    assert lib.ldga_bse_config(h.ctx.h).decode() == name
    ref = R.run_chain(inp, lambda_type=None)
    chi0 = L.calc_bubble(h)
    h.ctx.call("ldga_bse_sweeps", None, None)
    for r, s in (("m", 1.0), ("d", -1.0)):
        x, g = L.calc_χγ(r, h, chi0)
        want, chi = ref[f"gamma_{r}"], ref[f"chi_{r}"].data
        scale = np.abs(want * ref["chi0"] * (1.0 + s * inp.U * chi)[:, None, :]).sum(axis=1) / inp.beta**2
        assert float(np.max(np.abs(x.data - chi) / scale)) < 1e-10, r
        assert float(np.max(np.abs(g.data - want) / np.maximum(np.abs(want), 1e-6 * np.abs(want).max()))) < 1e-10, r
    n = _lib.C.c_int64()
    h.ctx.call("ldga_bse_sweeps", None, _lib.C.byref(n))      # warps of the iteration: none in the elimination
    assert (n.value > 0) == name.startswith("iter")
    # a recorded choice of the first entry holds through a file
    f = tmp_path / "tune.txt"
    f.write_text("bse 30 2 warp:1\n")
    try:
        L.tune_load(f)
        L.tune_save(f)
        L.tune_reset()
        L.tune_load(f)
        assert lib.ldga_bse_config(h.ctx.h).decode() == "warp:1"
    finally:
        L.tune_reset()
