"""Layout of batched regions: every mock's counts and sums from one launch
against a call on the mock alone.  Mock sizes around a warp, with one cell,
many cells, and a mock of one point; identical counts, and sums within the
rounding of their common scale (2^-60 of the largest product for each of the
pairs)."""
import numpy as np
import pytest

from gramsci_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("box", [3.0, 40.0])
@pytest.mark.parametrize("sizes", [(1,), (31, 32, 33), (2, 700, 1, 65)])
def test_mocks_one_by_one(sizes, box):
    rng = np.random.default_rng(sum(sizes))
    n_gal = np.array([max(1, s // 3) if s > 1 else 1 for s in sizes], np.int64)
    n_ran = np.array(sizes, np.int64) - n_gal
    xyz = [rng.uniform(0.0, box, (s, 3)) for s in sizes]
    w = []
    for s, g in zip(sizes, n_gal):
        v = rng.lognormal(0.0, 0.3, s)
        v[g:] *= -1.0
        w.append(v)
    wmax = max(np.abs(v).max() for v in w)
    with api.Context(0) as ctx:
        ctx.set_bins(0.5, 6.0, 5, nmu=4)
        ctx.set_catalog(np.concatenate(xyz), np.concatenate(w), int(n_gal[0]))
        ctx.set_mocks(n_gal, n_ran)
        got = ctx.count_2pcf_regions()
        for m in range(len(sizes)):
            ctx.set_catalog(xyz[m], w[m], int(n_gal[m]))
            one = ctx.count_2pcf()
            np.testing.assert_array_equal(got["counts"][..., m], one["counts"])
            bound = 2.0 ** -60 * wmax ** 2 * 2.0 * (one["counts"].max() + 1) + 4e-16 * np.abs(one["catsum"])
            assert np.all(np.abs(got["catsum"][..., m] - one["catsum"]) <= bound)
