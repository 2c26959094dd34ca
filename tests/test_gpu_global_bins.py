"""3PCF histograms too large for shared memory, whole or with the counts (16 by 2
bins: sums in shared memory, counts apart): vertices of a triangle in one
bin share an update, and roots are taken one at a time.  Counts equal the
oracle's; sums within two roundings of each product of three weights and the
rounding of each to 2^-59 of the largest."""
import numpy as np
import pytest

from gramsci_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins", [(0.5, 5.0, 16, 2), (0.5, 5.0, 16, 4), (0.5, 5.0, 17, 2), (0.5, 5.0, 18, 5), (1.0, 4.0, 4, 100)])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("buffers", [False, True])
def test_against_oracle(oracle, bins, weighted, buffers):
    rng = np.random.default_rng(11)
    xyz = np.concatenate([rng.uniform(0, 40, size=(500, 3)), 15 + rng.normal(0, 1.2, size=(120, 3)),
                          30 + rng.normal(0, 2.0, size=(100, 3))])
    xyz = rng.permutation(xyz)
    n, nd = len(xyz), 250
    size = rng.lognormal(0.0, 0.3, n) if weighted else np.ones(n)
    w = np.where(np.arange(n) < nd, size, -size)
    buf = (rng.uniform(size=n) < 0.3).astype(np.int32) if buffers else None
    assert api.ncfg3(bins[2]) * bins[3] * 4 * 24 > 120 * 1024 or not weighted
    ref = oracle.Graph(xyz, *bins).pcf3(w, nd, buffer=buf)
    with api.Context(0) as ctx:
        ctx.set_catalog(xyz, w, nd, buf)
        ctx.set_bins(*bins)
        got, sums = ctx.count_3pcf(), ctx.count_3pcf(counts=False)
    np.testing.assert_array_equal(got["counts"], ref["counts"])
    assert ref["counts"].max() > 1
    tol = 2.0 ** -51 * np.abs(ref["catsum"]) + 2.0 ** -58 * size.max() ** 3 * ref["counts"]
    assert np.all(np.abs(got["catsum"] - ref["catsum"]) <= tol)
    np.testing.assert_array_equal(sums["catsum"], got["catsum"])
