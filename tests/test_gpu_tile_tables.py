"""The tile pair sweep's tables (one update per pair, mirrored at the flush;
a second table for pairs with one buffer end; one update per root where both
do not fit, in shared or in global memory) against the warp-per-cell sweep,
which updates each root's bin as it finds it.  Every sum is an exact
fixed-point integer, so counts and sums are identical.  The lattice puts
separations and cosines on bin edges, where the two mu bins of a pair need
not mirror each other.  Sizes: a run of a few points, chunks of 32 points and
their remainders, and catalogues whose candidates are shared out."""
import numpy as np
import pytest

from gramsci_b200 import api

pytestmark = pytest.mark.gpu


def _points(kind, n):
    rng = np.random.default_rng(n)
    if kind == "lattice":
        xyz = rng.permutation(np.stack(np.meshgrid(*[np.arange(9.0)] * 3), -1).reshape(-1, 3))
        return xyz[:n] - 4.0, rng
    return rng.uniform(20.0, 32.0, size=(n, 3)), rng


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("buffers", [False, True])
@pytest.mark.parametrize("nbins,nmu", [(3, 1), (8, 4), (16, 10), (20, 40), (40, 40)])
@pytest.mark.parametrize("kind,n", [("uniform", 3), ("uniform", 700), ("lattice", 600),
                                    ("uniform", 2500)])
def test_tables(kind, n, nbins, nmu, buffers, weighted, precision):
    xyz, rng = _points(kind, n)
    w = rng.lognormal(0.0, 0.3, n) if weighted else np.ones(n)
    w[n // 3:] *= -1.0
    buf = (rng.uniform(size=n) < 0.4).astype(np.int32) if buffers else None
    if buffers:
        buf[xyz[:, 0] > np.median(xyz[:, 0])] = 1  # whole runs of buffer points
    with api.Context(0) as ctx:
        ctx.set_catalog(xyz, w, n // 3, buf)
        ctx.set_bins(1.0, 4.0, nbins, nmu=nmu)
        ctx.set_precision(precision)
        ctx.set_autotune(0)
        ref = ctx.count_2pcf()
        pairs = ctx.stats()["tuples"]
        cot = rng.normal(size=(2, nbins, nmu))
        grad = ctx.adjoint_2pcf(cot[0], cot[1])
        for variant in (6, 7):
            ctx.set_autotune(variant)
            got = ctx.count_2pcf()
            assert np.array_equal(got["counts"], ref["counts"])
            assert np.array_equal(got["catsum"], ref["catsum"])
            assert ctx.stats()["tuples"] == pairs
            # both gradients round each term once, to 2^-55 of the largest
            # possible sum of a pair's two cotangents (2^-61 for the other)
            g = ctx.adjoint_2pcf(cot[0], cot[1])
            assert np.abs(g - grad).max() <= n * 2.0 ** -50 * np.abs(cot).max() * np.abs(w).max()
