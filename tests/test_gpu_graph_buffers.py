"""A captured chain replayed after other calls that need larger buffers of the same handle.

The EoM's partial sums need not grow with numax (2D 64^2, 61 w: 270 rows at 30 nu, 589 at 19), and Sigma_loc and
G_imp may come longer in a later call.  A replay of the graph captured before must see the buffers
that are there now: its results equal the first, uncaptured run's bit for bit (tolerance 0).
"""
import ctypes as C

import numpy as np
import pytest

import ladderdga_b200 as L
from ladderdga_b200 import _lib
from ladderdga_b200 import synthetic as S

pytestmark = pytest.mark.gpu


class Chain:
    """ldga_chain_m of one handle on fixed pinned buffers; the vectors may be longer than needed."""

    def __init__(self, h, extra=0):
        import torch

        def pinned(a):
            v = np.ascontiguousarray(np.asarray(a, dtype=np.complex128).reshape(-1, order="F")).view(np.float64)
            return torch.from_numpy(v.copy()).pin_memory()

        tail = np.zeros(extra, dtype=np.complex128)
        sig, gimp = np.concatenate([h.Σ_loc, tail]), np.concatenate([h.gImp, tail])
        self.h, self.n = h, (len(sig), len(gimp))
        self.src = [pinned(a) for a in (sig, h.Γ_m, h.Γ_d, h.χDMFT_m, gimp)]
        c = h.ctx
        self.out = [torch.zeros(k, dtype=torch.float64).pin_memory()
                    for k in (c.Nq * h.sP.n_iν * 2, c.Nq * c.Nw, c.Nq * c.Nw)]

    def __call__(self, graph):
        p = [C.c_void_p(t.data_ptr()) for t in self.src]
        o = [C.c_void_p(t.data_ptr()) for t in self.out]
        for t in self.out:
            t.zero_()
        sc = (C.c_double * 8)()
        self.h.ctx.call("ldga_chain_m", p[0], self.n[0], p[1], p[2], p[3], p[4], self.n[1], self.h.imp_density,
                        self.h.χloc_m_sum, graph, *o, sc)
        return [t.numpy().copy() for t in self.out] + [np.array(sc[:])]


def same(a, b):
    return all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b))


@pytest.mark.parametrize("dim,ns,n_iv,n_iw", [(2, 64, 30, 30), (3, 12, 17, 13), (2, 8, 4, 3), (2, 9, 5, 2)])
def test_replay_after_other_numbers_of_nu(dim, ns, n_iv, n_iw, require_gpu):
    inp = S.make_input(dim=dim, ns=ns, beta=max(4.0, 0.5 * n_iv), U=1.0, n_iv=n_iv, n_iw=n_iw, seed=810 + ns)
    h = L.setup_synthetic(inp, precision=L.PREC_MIXED)
    run = Chain(h)
    want = run(0)
    assert same(run(1), want)                 # captures
    assert same(run(1), want)                 # replays
    ctx = h.ctx
    for numax in range(1, 2 * n_iv + 1):
        ctx.call("ldga_eom", 0.5, 0.0, numax, 1, h.χloc_m_sum, None)
    assert same(run(1), want)
    lm, ld = C.c_double(), C.c_double()
    st = _lib.load().ldga_lambda_dm(ctx.h, h.χloc_m_sum, 0, 1e-4, 1e-8, 2, C.byref(lm), C.byref(ld), None, None, None,
                                    None, None)
    assert st in (0, 5), st                   # two Newton steps: a root or "not converged"
    assert same(run(1), want)
    for lo, hi in ((0, 1), (1, ctx.Nw), (0, (ctx.Nw + 1) // 2)):
        ctx.call("ldga_set_omega_shard", lo, hi, 1)
        for numax in range(1, n_iv + 1):
            ctx.call("ldga_eom", 0.5, 0.0, numax, 1, h.χloc_m_sum, None)
    ctx.call("ldga_set_omega_shard", 0, ctx.Nw, 1)
    assert same(run(1), want)
    assert same(run(1), want)


def test_replay_after_longer_local_inputs(require_gpu):
    inp = S.make_input(dim=2, ns=8, beta=6.0, U=1.0, n_iv=5, n_iw=4, seed=820)
    h = L.setup_synthetic(inp, precision=L.PREC_MIXED)
    run, longer = Chain(h), Chain(h, extra=5000)
    want = run(0)
    assert same(run(1), want)
    assert same(longer(0), want)              # larger Sigma_loc and G_imp buffers
    assert same(run(1), want)
    sig = np.concatenate([h.Σ_loc, np.zeros(20000, dtype=np.complex128)])
    h.ctx.call("ldga_gloc", _lib.ptr(_lib.as_fc(h.Σ_loc)), len(h.Σ_loc), None)    # shorter again,
    h.ctx.call("ldga_gloc", _lib.ptr(_lib.as_fc(sig)), len(sig), None)           # then longer than any
    assert same(run(1), want)
    assert same(run(1), want)
