"""Graphs filled without host waits (the hash-probe 3PCF): a catalogue whose
candidates do not fit the scratch area is counted again with waits, a catalogue
with another box takes its own grid, default-mode counts in between change
nothing.  Every count against the oracle."""
import numpy as np
import pytest

from gramsci_b200 import api, catalogs

pytestmark = pytest.mark.gpu

BINS = (5.0, 25.0, 8, 5)
N = 3000


def _points(rng, lo, hi):
    corners = np.array([[x, y, z] for x in (0.0, 300.0) for y in (0.0, 300.0) for z in (0.0, 300.0)])
    return np.vstack([corners, rng.uniform(lo, hi, (N - 8, 3))])


@pytest.mark.parametrize("between", [False, True])
@pytest.mark.parametrize("weighted", [False, True])
def test_counts(oracle, between, weighted):
    rng = np.random.default_rng(41)
    sparse, again = _points(rng, 0.0, 300.0), _points(rng, 0.0, 300.0)
    dense, denser = _points(rng, 100.0, 200.0), _points(rng, 110.0, 195.0)
    other = rng.uniform(0.0, 360.0, (N, 3))
    with api.Context(0) as ctx:
        ctx.set_bins(*BINS)
        ctx.set_clique_mode("hash")
        for k, xyz in enumerate((sparse, again, dense, sparse, other, denser, dense)):
            size = rng.lognormal(0, 0.3, N) if weighted else np.ones(N)
            w = catalogs.normalise(size, 1000, N - 1000)
            ref = oracle.Graph(xyz, *BINS).pcf3(w, 1000)
            ctx.set_catalog(xyz, w, 1000)
            if between and k != 2:
                ctx.set_clique_mode("auto")
                ctx.count_3pcf()
                ctx.set_clique_mode("hash")
            for _ in range(2):
                got = ctx.count_3pcf()
                assert np.array_equal(got["counts"], ref["counts"])
                scale = np.abs(ref["catsum"]).max()
                assert np.all(np.abs(got["catsum"] - ref["catsum"]) <= 1e-12 * scale)
            if xyz is dense:
                # more edges than the scratch area of a first build holds
                assert ctx.stats()["upper_edges"] > 64 * N + 1024
