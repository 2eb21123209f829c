"""The skew form's kernels over the lattice sizes and numbers of walkers (skew.cu): every even square lattice is an
instance of its own; few walkers have a cluster of blocks each, many one block; small lattices keep a fetch buffer per
warp, large ones read the inverse matrices in place.  Chains are compared with the oracle's decision by decision,
amplitudes, local energies and derivatives of given configurations with its values."""
import numpy as np
import pytest

import chain_compare as cc
from test_gpu_transverse import RTOL, _configs, _pair, _rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,trans,nw,ns", [
    (4, True, 3, 8),
    (4, False, 160, 1),  # more walkers than SMs
    (6, True, 2, 2),     # four blocks per walker
    (6, True, 40, 1),    # two
    (8, True, 1, 1),     # eight
    (8, False, 4, 1),
    (10, False, 2, 1),
])
def test_chains_sizes(L, trans, nw, ns):
    p, o, g = _pair(L, trans, 1, nw, ns, seed=80 + L)
    for c in (o, g):
        c.set_trace(16384)
        c.seed(77)
    na_o, na_g = o.make_sample(True), g.make_sample(True)
    eo, to = o.events()
    eg, tg = g.events()
    recs = cc.compare_walkers(to, eo, tg, eg)
    xo, xg = o.samples()[0], g.samples()[0]
    for r in recs:
        assert r["kind"] not in ("type", "draw", "length"), r
        if r["kind"] == "exact":
            w = r["walker"]
            assert na_o[w] == na_g[w] and np.array_equal(xo[w], xg[w])
        # a walker may part at a checkpoint only where the two drift measures lie on either side of the threshold
        assert r["kind"] != "checkpoint" or r["straddle"], r
    assert any(r["kind"] == "exact" for r in recs)
    g.close()


@pytest.mark.parametrize("L,n", [(8, 6), (10, 3)])
def test_eval_sizes(L, n):
    p, o, g = _pair(L, False, 1, 1, 8, seed=90 + L)
    x = _configs(L * L, n, seed=L)
    ro = o.eval_configs(x, want_h=True, want_O=True)
    rg = g.eval_configs(x, want_h=True, want_O=True)
    assert _rel(rg["psi"], ro["psi"]) < RTOL
    for k in range(n):
        assert abs(rg["hpsi"][k] - ro["hpsi"][k]) <= RTOL * max(abs(ro["hpsi"][k]), abs(ro["psi"][k, 0]))
        assert np.abs(rg["O"][k] - ro["O"][k].real).max() <= RTOL * np.abs(ro["O"][k]).max(), k
    g.close()
