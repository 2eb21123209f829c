"""Estimator and correlation measurement at the block sizes that invert in registers (N/2 = 8, 18, 32, 50) against the
oracle: rounds of projections that are full, partial and a single pair, no RBM units, complex units, the 2-sublattice
map, and unit weights beyond the range in which the pair weights factorise into exponentials.  1e-10 relative, the
tolerance of the other estimator parity tests."""
import numpy as np
import pytest

import pyoracle as po
from rbm_pp_b200 import capi
from rbm_pp_b200 import formats as fm

pytestmark = pytest.mark.gpu
RTOL = 1e-10


def _problem(L, n_mp, alphar, seed, **kw):
    p = fm.synthetic_problem(L, translations=n_mp > 1, alphar=alphar, nsample=64, seed=seed, **kw)
    p.sym.n_mp = n_mp
    p.sym.W_map = np.ascontiguousarray(p.sym.W_map[:, :n_mp])
    p.sym.para_mp = p.sym.para_mp[:n_mp]
    return p


def _configs(N, n, seed):
    rng = np.random.default_rng(seed)
    x = -np.ones((n, N), dtype=np.int32)
    for r in x:
        r[rng.choice(N, N // 2, replace=False)] = 1
    return x


def _rel(a, b):
    return float(np.abs(np.asarray(a) - np.asarray(b)).max() / max(np.abs(np.asarray(b)).max(), 1e-300))


@pytest.mark.parametrize("L,n_mp,alphar,kw", [
    (4, 1, 1, {}), (4, 5, 0, {}), (4, 16, 2, dict(orbital="sublattice2")), (6, 1, 2, {}), (6, 3, 1, dict(spin_parity=-1)),
    (6, 36, 1, {}), (8, 1, 1, dict(orbital="sublattice2")), (8, 6, 2, {}), (10, 1, 4, {}), (10, 5, 1, {})])
def test_estimator(L, n_mp, alphar, kw):
    p = _problem(L, n_mp, alphar, 70 + L, **kw)
    x = _configs(L * L, 9, L)
    o = po.Oracle(p, nranks=1, nsample_per_rank=1, nthreads=8)
    g = capi.Context(p, n_walkers=1, nsample_per_walker=1)
    for c in (o, g):
        c.set_params(p.br, p.Wr, p.slater, 0.0)
    ro, rg = o.eval_configs(x, want_h=True, want_O=True), g.eval_configs(x, want_h=True, want_O=True)
    assert _rel(rg["psi"], ro["psi"]) < RTOL
    assert _rel(rg["hpsi"], ro["hpsi"]) < RTOL
    for k in range(len(x)):
        assert np.abs(rg["O"][k] - ro["O"][k].real).max() <= RTOL * np.abs(ro["O"][k]).max()
    g.close()


@pytest.mark.parametrize("L,n_mp,alphar,w", [(4, 1, 2, None), (4, 7, 1, 200.0), (6, 1, 0, None), (6, 9, 1, None),
                                             (8, 1, 1, 200.0), (8, 3, 2, None), (10, 2, 1, None)])
def test_correlation(L, n_mp, alphar, w):
    p = _problem(L, n_mp, alphar, 90 + L)
    if w is not None:  # equal weights cancel in theta' (Sz = 0) but not in its two parts
        p.Wr = np.full_like(p.Wr, w)
    nw, ns = 2, 2
    o = po.Oracle(p, nranks=nw, nsample_per_rank=ns, nthreads=8)
    g = capi.Context(p, n_walkers=nw, nsample_per_walker=ns)
    x = _configs(L * L, nw * ns, 3 * L)
    for c in (o, g):
        c.set_params(p.br, p.Wr, p.slater, 0.0)
        c.seed(5)
        c.set_samples(x)
    mo, mg = o.measure_correlation(), g.measure_correlation()
    for k in ("Etot", "Etot2", "norm", "wf_av", "chi_sp", "chi_vbs"):
        assert _rel(mg[k], mo[k]) < RTOL, k
    g.close()


@pytest.mark.parametrize("L", [4, 6, 8, 10])
def test_singular_blocks_are_reported(L):
    p = _problem(L, 2, 1, 3)
    g = capi.Context(p, n_walkers=1, nsample_per_walker=1)
    for f in (np.zeros_like(p.slater), np.full_like(p.slater, np.nan)):
        g.set_params(p.br, p.Wr, f, 0.0)
        with pytest.raises(capi.RbmppError) as e:
            g.eval_configs(_configs(L * L, 2, 1))
        assert e.value.code == 8
    g.set_params(p.br, p.Wr, p.slater, 0.0)
    assert np.isfinite(g.eval_configs(_configs(L * L, 2, 1))["psi"].real).all()
    g.close()
