"""Statistics of the 3PCF adjoint: the triangles, edges and pair tests of the
count of the same catalogue, for rows of a warp and beyond (the second
launch), with and without mu bins and buffer points."""
import numpy as np
import pytest

from gramsci_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("members", [60, 1300])
@pytest.mark.parametrize("nmu", [1, 3])
@pytest.mark.parametrize("buffers", [False, True])
def test_as_the_count(members, nmu, buffers):
    rng = np.random.default_rng(members)
    xyz = np.concatenate([rng.uniform(0, 60, size=(500, 3)), 30 + rng.normal(0, 0.8, size=(members, 3))])
    n, nd = len(xyz), 300
    w = rng.lognormal(0.0, 0.3, n)
    buf = (rng.uniform(size=n) < 0.3).astype(np.int32) if buffers else None
    keys = ("tuples", "rooted", "n_edges", "upper_edges", "probes", "candidates")
    with api.Context(0) as ctx:
        ctx.set_catalog(xyz, w, nd, buf)
        ctx.set_bins(0.2, 4.0, 3, nmu)
        ctx.count_3pcf()
        want = ctx.stats()
        ctx.adjoint_3pcf(rng.normal(size=(api.ncfg3(3), nmu)))
        got = ctx.stats()
    assert want["tuples"] > 0
    assert {k: got[k] for k in keys} == {k: want[k] for k in keys}
