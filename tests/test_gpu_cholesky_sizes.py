"""The SR step's factorisation and solve at parameter counts around multiples of its 128-column blocks (one block, a second
of six columns, a third of fourteen, eleven with a remainder) against numpy's solve of the same conditioned S.  Two
backward-stable solves of one system differ by a small multiple of n eps cond(S)."""
import numpy as np
import pytest

from rbm_pp_b200 import capi
from rbm_pp_b200 import formats as fm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,orbital,alphar,nv", [(4, "sublattice2", 1, 49), (4, "sublattice2", 6, 134),
                                                 (4, "sublattice2", 14, 270), (6, "full", 1, 1333)])
def test_solve(L, orbital, alphar, nv):
    p = fm.synthetic_problem(L, translations=False, alphar=alphar, orbital=orbital, nsample=512, seed=3)
    assert p.Nv == nv
    g = capi.Context(p, n_walkers=64, nsample_per_walker=8)
    g.set_params(p.br, p.Wr, p.slater, 0.0)
    g.seed(11)
    g.make_sample(True)
    m = g.measure(want_S=True)
    out, dx = g.sr_step(1, 0.05, 0.1, 1e-3, precision=capi.SR_FP64)
    n, nr = m["norm"], alphar * (L * L + 1)
    ov, e = m["Ovec"] / n, m["Etot"] / n
    b = m["gvec"] / n - 2.0 * e * ov
    S = m["S"] / n - np.outer(ov, ov)
    dg = np.diag(S).copy()
    live = np.ones(nv, dtype=bool)
    live[nr + np.diag(p.orbital_idx) - 1] = False  # f_ii carry no derivative
    v = np.ones(nv)
    v[nr:] = np.sqrt(dg[:nr].mean() / dg[nr:][live[nr:]].mean())
    S = S * v[:, None] * v[None, :]
    S[np.diag_indices(nv)] += np.diag(S)[live].mean() * 0.1
    x = np.linalg.solve(S, b * v)
    lam = np.sqrt(x @ S @ x) * 5.0 / L
    ref = (x / lam if lam > 1.0 else x) * v
    tol = 4.0 * nv * np.finfo(float).eps * np.linalg.cond(S)
    assert tol < 1e-6
    assert np.abs(dx - ref).max() <= tol * np.abs(ref).max()
    assert abs(out.lambda_ - lam) <= tol * lam
    g.close()
