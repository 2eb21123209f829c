"""The resident sampler (inverse blocks of a walker in shared memory for the whole make_sample call) against the
direct sampler on the same streams: accept counts, stored configurations, Nfastup and events are equal, and the
stored Pfaffians agree within 1e-6 of the largest, the drift of fast updates that make_sample.f90:120 accepts.

The shapes are the ends of each block size and of the two ways a block's warps are dealt out: up to six projections
(several warps share one projection's rows, a last share shorter than the others) and more (several projections per
warp, a last round that is not full); no RBM units; odd numbers of projections; a rejected and an accepted flip.
"""
import numpy as np
import pytest

from rbm_pp_b200 import capi
from rbm_pp_b200 import formats as fm

pytestmark = pytest.mark.gpu


def _problem(L, n_mp, alphar, seed):
    p = fm.synthetic_problem(L, translations=n_mp > 1, alphar=alphar, nsample=64, seed=seed)
    p.sym.n_mp = n_mp
    p.sym.W_map = np.ascontiguousarray(p.sym.W_map[:, :n_mp])
    p.sym.para_mp = p.sym.para_mp[:n_mp]
    return p


def _run(p, nw, ns, seed, calls):
    g = capi.Context(p, n_walkers=nw, nsample_per_walker=ns)
    g.set_params(p.br, p.Wr, p.slater, 0.01)
    g.seed(seed)
    out = []
    for k in range(calls):
        na = g.make_sample(k == 0)
        x, psi, pf = g.samples()
        out.append((na, x, psi, pf, g.nfastup(), g.events()[0][:, :4]))
    g.close()
    return out


@pytest.mark.parametrize("L,n_mp,alphar,nw,ns", [
    (4, 1, 1, 5, 9), (4, 16, 2, 3, 4), (4, 7, 0, 2, 3), (6, 1, 3, 4, 3), (6, 3, 1, 2, 2), (6, 36, 2, 2, 2),
    (6, 5, 4, 2, 2), (8, 1, 2, 3, 2), (8, 2, 1, 2, 1), (8, 8, 1, 2, 1), (10, 1, 4, 2, 1), (10, 3, 1, 2, 1),
    (12, 1, 2, 2, 1), (12, 2, 1, 1, 1), (14, 1, 2, 2, 1)])
def test_resident_equals_direct(L, n_mp, alphar, nw, ns, monkeypatch):
    p = _problem(L, n_mp, alphar, seed=30 + L)
    got = _run(p, nw, ns, 500 + L, 2)
    monkeypatch.setenv("RBMPP_SAMPLER", "direct")
    want = _run(p, nw, ns, 500 + L, 2)
    for (na, x, psi, pf, nf, ev), (na2, x2, psi2, pf2, nf2, ev2) in zip(got, want):
        assert np.array_equal(na, na2)
        assert np.array_equal(x, x2)
        assert np.array_equal(nf, nf2)
        assert np.array_equal(ev, ev2)
        assert np.abs(pf - pf2).max() <= 1e-6 * np.abs(pf2).max()
        assert np.abs(psi - psi2).max() <= 1e-6 * np.abs(psi2).max()
