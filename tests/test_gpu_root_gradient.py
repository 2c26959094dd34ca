"""Rounding of the 3PCF gradient: rows of a thousand members and more whose
sums are known exactly.

One root sees two clusters, each narrower than rmin, every pair across them an
edge: all triangles are the root with a member of either cluster, found in the
root's row alone.  With one bin, cotangent 1 and galaxies only, a member's
gradient is 3 times the root's weight times the other cluster's weights, the
root's 3 times the product of both clusters'.

Bound, in units of 2^-53 of the value: the conversions of a row's integer sum,
its product with the root's weight and the conversion of the total round once
each, 3 units; the terms' own roundings and their quantisation, at least 2^-49
of the largest, are independent, six of their standard deviations under half a
unit (with mu bins, where the scale has room for 1024 terms of the whole
product, under 2.5 units, and no product with the root's weight follows).  A
sum of 500 such terms in FP64 is off by 5 units rms and 15 to 20 at worst."""
from fractions import Fraction

import numpy as np
import pytest

from gramsci_b200 import api

pytestmark = pytest.mark.gpu


def _clusters(m, rng):
    def ball(centre):
        v = rng.normal(size=(m, 3))
        return centre + 0.2 * rng.uniform(size=(m, 1)) * v / np.linalg.norm(v, axis=1)[:, None]

    return np.vstack([np.zeros((1, 3)), ball([2.0, 0.0, 0.0]), ball([1.0, 1.7, 0.0])])


@pytest.mark.parametrize("m", [40, 500, 1500])  # a group's, a warp's and a block's row
@pytest.mark.parametrize("nmu", [1, 2])
@pytest.mark.parametrize("buffer", [False, True])
def test_against_exact_sums(m, nmu, buffer):
    rng = np.random.default_rng(100 * m + nmu)
    xyz = _clusters(m, rng)
    w = rng.uniform(0.5, 1.0, len(xyz))
    with api.Context(0) as ctx:
        ctx.set_catalog(xyz, w, len(w), np.zeros(len(w), np.int32) if buffer else None)
        ctx.set_bins(1.0, 3.0, 1, nmu)
        assert ctx.count_3pcf()["counts"].sum() == 3 * m * m
        got = ctx.adjoint_3pcf(np.ones((1, nmu)))
    f = [Fraction(float(v)) for v in w]
    a, b = sum(f[1:m + 1]), sum(f[m + 1:])
    want = [3 * a * b] + [3 * f[0] * b] * m + [3 * f[0] * a] * m
    off = [abs(float((Fraction(float(g)) - v) / v)) * 2.0 ** 53 for g, v in zip(got, want)]
    assert max(off) <= 4.0, (off[0], max(off))
