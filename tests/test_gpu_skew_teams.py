"""The transverse sampler's chains do not depend on how many blocks carry a walker: a few walkers run in clusters of blocks,
a hundred and sixty in one block each, and the same walkers (same streams) end with the same decisions, configurations,
amplitudes and Pfaffians to the bit."""
import numpy as np
import pytest

from rbm_pp_b200 import capi
from rbm_pp_b200 import formats as fm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,alphar,nw", [(4, 1, 40), (4, 2, 4), (6, 1, 60), (6, 1, 30), (6, 1, 4), (8, 1, 3)])
def test_clusters_equal_single_blocks(L, alphar, nw):
    out = []
    for walkers in (nw, 160):
        p = fm.synthetic_problem(L, translations=True, alphar=alphar, nsample=160, seed=50 + L)
        g = capi.Context(p, n_walkers=walkers, nsample_per_walker=1,
                         sp_weights=fm.spin_projection_weights(1, transverse=True))
        g.set_params(p.br, p.Wr, p.slater, 0.0)
        g.set_trace(4096)
        g.seed(70 + L)
        for first in (True, False):
            na = g.make_sample(first)
            ev, tr = g.events()
            out.append([a[:nw] for a in (na, *g.samples(), g.nfastup(), ev, tr)])
        g.close()
    for a, b in zip(out[:2], out[2:]):
        for u, v in zip(a, b):
            assert np.array_equal(u, v)
