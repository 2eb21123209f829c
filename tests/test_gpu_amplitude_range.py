"""Accept tests whose amplitude ratio leaves the double range (make_sample.f90:195-204).

One unit whose weight sits on two sites, with opposite signs, puts 308 decades between configurations with these sites
parallel (theta = 0) and anti-parallel (|theta| = 710.4, cosh = 1.7e308); their f_ij with other sites are lowered, which
puts six more decades between the Pfaffians, and a common factor of f_ij keeps both amplitudes finite.  The first
exchange that makes them anti-parallel has an infinite ratio, which exceeds every drawn number: it is accepted.
"""
import numpy as np
import pytest

import chain_compare as cc
import pyoracle as po
from rbm_pp_b200 import capi
from rbm_pp_b200 import formats as fm

pytestmark = pytest.mark.gpu


def _problem(L, scale, seed):
    p = fm.synthetic_problem(L, translations=False, alphar=1, nsample=64, seed=seed)
    p.slater = p.slater * scale
    p.br = np.zeros(1)
    p.Wr = np.zeros((L * L, 1))
    p.Wr[0], p.Wr[1] = 355.2, -355.2
    low = np.zeros((L * L, L * L), dtype=bool)
    low[:2, 2:] = low[2:, :2] = True
    p.slater[p.orbital_idx[low] - 1] *= 1e-3
    return p


@pytest.mark.parametrize("L,scale,nw", [(4, 1e-20, 8), (6, 1e-9, 8), (10, 1e-4, 6)])
def test_overflowing_ratio_is_accepted(L, scale, nw):
    p = _problem(L, scale, 40 + L)
    o = po.Oracle(p, nranks=nw, nsample_per_rank=1, nthreads=4)
    g = capi.Context(p, n_walkers=nw, nsample_per_walker=1)
    for c in (o, g):
        c.set_params(p.br, p.Wr, p.slater, 0.0)
        c.set_trace(8192)
        c.seed(900 + L)
    o.make_sample(True)
    g.make_sample(True)
    (eo, to), (eg, tg) = o.events(), g.events()
    over = [(to[w, :min(eo[w, 4], 8192), 0] == 0) & np.isinf(to[w, :min(eo[w, 4], 8192), 3]) for w in range(nw)]
    assert sum(int(m.any()) for m in over) >= 2  # walkers that meet such a proposal
    for w in range(nw):
        first = int(np.argmax(over[w])) if over[w].any() else -1
        if first >= 0:
            assert to[w, first, 5] == 1.0
            assert np.array_equal(tg[w, first, [0, 1, 2, 4, 5]], to[w, first, [0, 1, 2, 4, 5]]), w
    for r in cc.compare_walkers(to, eo, tg, eg):
        assert r["kind"] in ("exact", "checkpoint"), r
    g.close()
