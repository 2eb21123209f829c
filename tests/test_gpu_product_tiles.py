"""The FP64 upper-triangle products and the factorisation at parameter counts whose products run on 128-wide tiles (from
1,537 rows on; 4,226 takes 96 again for S) and whose panel blocks hold 16 to 72 columns; odd and even counts take the
8- and the 16-byte copies, and the sample counts leave a remainder of the 16 samples of a step.

S against numpy's product of the same derivatives: a sum of K products in any order is within K eps of the sum of
their magnitudes, and the factors carry a few roundings.  The solve by its residual: a Cholesky solve is backward
stable, ||S x - b|| <= c n eps ||S|| ||x||, with c = 4 as in the other tests of the solve."""
import numpy as np
import pytest

from rbm_pp_b200 import capi
from rbm_pp_b200 import formats as fm

pytestmark = pytest.mark.gpu
EPS = np.finfo(float).eps


def _context(L, alphar, nv, walkers, ns):
    p = fm.synthetic_problem(L, translations=False, alphar=alphar, nsample=walkers * ns, seed=3)
    assert p.Nv == nv
    g = capi.Context(p, n_walkers=walkers, nsample_per_walker=ns)
    g.set_params(p.br, p.Wr, p.slater, 0.0)
    g.seed(11)
    g.make_sample(True)
    return p, g


@pytest.mark.parametrize("L,alphar,nv", [(6, 10, 1666), (6, 11, 1703), (8, 1, 4161), (8, 2, 4226)])
def test_product(L, alphar, nv):
    p, g = _context(L, alphar, nv, 53, 7)
    S = g.measure(want_S=True)["S"]
    r = g.eval_configs(g.samples()[0].reshape(-1, L * L), want_h=False, want_O=True)
    O = r["O"] / np.abs(r["psi"][:, 0])[:, None]
    g.close()
    err, mag = np.abs(S - O.T @ O), np.abs(O).T @ np.abs(O)
    assert (err <= 2.0 * (len(O) + 8) * EPS * mag).all()


@pytest.mark.parametrize("L,alphar,nv", [(6, 10, 1666), (6, 11, 1703), (8, 1, 4161), (8, 2, 4226), (10, 4, 10404)])
def test_solve(L, alphar, nv):
    p, g = _context(L, alphar, nv, 64, 8)
    m = g.measure(want_S=True)
    out, dx = g.sr_step(1, 0.05, 0.1, 1e-3, precision=capi.SR_FP64)
    g.close()
    n, nr = m["norm"], alphar * (L * L + 1)
    ov = m["Ovec"] / n
    b = m["gvec"] / n - 2.0 * (m["Etot"] / n) * ov
    S = m["S"] / n
    S -= np.outer(ov, ov)
    dg = np.diag(S).copy()
    live = np.ones(nv, dtype=bool)
    live[nr + np.diag(p.orbital_idx) - 1] = False  # f_ii carry no derivative
    v = np.ones(nv)
    v[nr:] = np.sqrt(dg[:nr].mean() / dg[nr:][live[nr:]].mean())
    S *= v
    S *= v[:, None]
    S[np.diag_indices(nv)] += np.diag(S)[live].mean() * 0.1
    x = dx / v * max(out.lambda_, 1.0)
    tol = 4.0 * nv * EPS
    assert np.linalg.norm(S @ x - b * v) <= tol * np.linalg.norm(S) * np.linalg.norm(x)
    assert abs(out.lambda_ - np.sqrt(x @ S @ x) * 5.0 / L) <= tol * np.linalg.norm(S) * (x @ x) / out.lambda_
