"""Which sampler a context takes, and the streaming sampler beside the resident one that took over its small shapes.

Blocks of at most 32 rows are summed in the same order by both, so their chains and stored amplitudes are equal to the
bit; the shapes are both ends of each block size with few projections and with many."""
import numpy as np
import pytest

from rbm_pp_b200 import capi
from rbm_pp_b200 import formats as fm

pytestmark = pytest.mark.gpu


def _context(L, trans, alphar, nw=3, ns=3):
    p = fm.synthetic_problem(L, translations=trans, alphar=alphar, nsample=nw * ns, seed=60 + L)
    g = capi.Context(p, n_walkers=nw, nsample_per_walker=ns)
    g.set_params(p.br, p.Wr, p.slater, 0.0)
    g.seed(17)
    return g


@pytest.mark.parametrize("L,trans,alphar,kind", [
    (4, False, 1, "resident"), (6, True, 2, "resident"), (12, False, 2, "resident"), (6, True, 8, "stream"),
    (8, True, 2, "stream"), (10, True, 4, "stream"), (16, False, 2, "direct")])
def test_choice(L, trans, alphar, kind, monkeypatch):
    for want, kinds in (("", (kind,)), ("stream", ("stream", "direct")), ("direct", ("direct",))):
        monkeypatch.setenv("RBMPP_SAMPLER", want)
        g = _context(L, trans, alphar, 1, 1)
        assert g.sampler_kind() in kinds
        if want == "stream":
            assert (g.sampler_kind() == "stream") == (L in (4, 6, 8, 10))
        g.close()


def test_hooks_keep_the_streaming_sampler():
    g = _context(6, True, 2)
    assert g.sampler_kind() == "resident"
    g.debug_hook(2, 4096)
    assert g.sampler_kind() == "stream"
    g.debug_hook(2, 0)
    assert g.sampler_kind() == "stream"
    g.close()


@pytest.mark.parametrize("L,trans,alphar", [(4, False, 1), (4, True, 2), (6, False, 3), (6, True, 2), (8, False, 2)])
def test_resident_equals_streamed(L, trans, alphar, monkeypatch):
    out = []
    for want in ("", "stream"):
        monkeypatch.setenv("RBMPP_SAMPLER", want)
        g = _context(L, trans, alphar)
        out.append([(g.sampler_kind(),)])
        for first in (True, False):
            na = g.make_sample(first)
            out[-1].append((na, *g.samples(), g.nfastup()))
        g.close()
    assert [o[0][0] for o in out] == ["resident", "stream"]
    for a, b in zip(out[0][1:], out[1][1:]):
        for u, v in zip(a, b):
            assert np.array_equal(u, v)


def test_streamed_beyond_resident_equals_direct(monkeypatch):
    """6x6 with 72 projections and eight units per projection: more than an SM's shared memory holds."""
    out = []
    for want in ("", "direct"):
        monkeypatch.setenv("RBMPP_SAMPLER", want)
        g = _context(6, True, 8)
        out.append((g.sampler_kind(), g.make_sample(True), g.make_sample(False), *g.samples()))
        g.close()
    (ka, a1, a2, xa, pa, fa), (kb, b1, b2, xb, pb, fb) = out
    assert (ka, kb) == ("stream", "direct")
    assert np.array_equal(a1, b1) and np.array_equal(a2, b2) and np.array_equal(xa, xb)
    assert np.abs(pa - pb).max() <= 1e-6 * np.abs(pb).max()  # the drift make_sample.f90:120 accepts
    assert np.abs(fa - fb).max() <= 1e-6 * np.abs(fb).max()
