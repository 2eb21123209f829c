"""The scalar FP64 operations of csrc/fp64_ops.cuh against IEEE division and square root (numpy's, correctly rounded as
CUDA's are): random arguments, and every pairing of signs, subnormals, the ends of the ranges in which the Newton forms
apply, significands next to a power of two, 0, infinity and NaN.

Equal: reciprocal and quotient, but for a divisor whose significand is all ones (one unit in the last place: the case
that Markstein's theorem leaves out), and all 2^32 words of the generator.  Within one unit: 1 / sqrt (half a unit
from its last addition, at most half from the rounded product in it) and sqrt (half a unit and a second-order term)."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from rbm_pp_b200 import build

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


def _arguments():
    rng = np.random.default_rng(5)
    n = 1 << 20
    near = rng.uniform(0.1, 10.0, n) * rng.choice([-1.0, 1.0], n)
    wide = rng.uniform(1.0, 2.0, n) * 2.0 ** rng.integers(-1022, 1024, n)
    edge = [0.0, 5e-324, 1e-310, 2.2250738585072014e-308, np.inf, np.nan, np.finfo(float).max]
    for c in (1e-280, 1e-250, 1e-30, 0.5, 1.0, 2.0, 3.0, 1e30, 1e250, 1e280):
        edge += [c, np.nextafter(c, 0.0), np.nextafter(c, np.inf), 1.7 * c, c / 1.7]
    edge = np.array(edge + [-e for e in edge])
    ea, eb = [g.ravel() for g in np.meshgrid(edge, edge)]
    a = np.concatenate([near, wide, np.roll(near, 7), ea])
    b = np.concatenate([np.roll(near, 1), np.roll(wide, 3), wide, eb])
    return a, b


def test_against_ieee(tmp_path):
    so = str(tmp_path / "fp64_ops_check.so")
    subprocess.check_call([build.NVCC, *build.FLAGS, "-I", build.CSRC, "-shared", "-o", so,
                           os.path.join(HERE, "fp64_ops_check.cu")])
    a, b = _arguments()
    n = len(a)
    out, bad = np.zeros((4, n)), ctypes.c_ulonglong(1)
    p = [x.ctypes.data_as(ctypes.c_void_p) for x in (a, b, out)]
    assert ctypes.CDLL(so).fp64_ops_check(n, *p, ctypes.byref(bad)) == 0
    with np.errstate(all="ignore"):
        want = np.array([1.0 / b, a / b])
        ab = np.abs(b).astype(np.longdouble)
        root = np.sqrt(ab)
        inv = 1.0 / root
    same = (out[:2] == want) | (np.isnan(out[:2]) & np.isnan(want))
    ones = np.frexp(np.abs(b))[0] == 1.0 - 2.0 ** -53
    assert same[:, ~ones].all()
    with np.errstate(all="ignore"):
        assert (np.abs(out[:2] - want) <= np.spacing(np.abs(want)))[~same].all()
    for got, ref in ((out[2], inv), (out[3], root)):
        ref64 = ref.astype(np.float64)
        special = ~np.isfinite(ref64) | (ref64 == 0.0)
        assert np.array_equal(got[special], ref64[special], equal_nan=True)
        err = np.abs(got[~special].astype(np.longdouble) - ref[~special])
        assert (err <= np.spacing(ref64[~special])).all()
    assert bad.value == 0
