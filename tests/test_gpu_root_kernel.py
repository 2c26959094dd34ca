"""The rooted triangle kernel (gr_root.cu) against the hash-probe kernel on the
neighbour graph: rows from empty to beyond a warp's capacity (the second
launch), groups of roots that split at cells and at the capacity, more bins
than the configuration table takes, a find_normal table that is not symmetric
(25 mu bins), buffer points, -equi, the FP64 path, log bins and separations on
bin edges.

Counts are identical.  Sums: the two multiply three weights in orders that
differ by one rounding of each product (2^-52 relative, products of one
category have one sign) and round each to 2^-59 of the largest.  Gradients are
compared with the oracle's: without mu bins a row's terms, at most 1024 in a
warp's row or a block's, are added in FP64, a relative 2^-43 of the sum of
their sizes, which the gradient of the sizes gives; with mu bins, and on the
hash-probe side, terms are rounded to a fixed fraction of the largest possible
one, and the bound is the other gradient tests' 1e-12 of the largest entry."""
import numpy as np
import pytest

from gramsci_b200 import api

pytestmark = pytest.mark.gpu


def _points(kind, rng):
    if kind == "few":
        return rng.uniform(50.0, 54.0, size=(3, 3))
    if kind == "one":
        return rng.uniform(50.0, 54.0, size=(1, 3))
    if kind == "sparse":
        return rng.uniform(0.0, 60.0, size=(900, 3))
    if kind == "lattice":
        g = np.stack(np.meshgrid(*[np.arange(8.0)] * 3), -1).reshape(-1, 3)
        return rng.permutation(g) - 3.0
    if kind == "clumps":  # rows of 30 to 300
        return np.concatenate([rng.uniform(0, 60, size=(600, 3)),
                               20 + rng.normal(0, 1.0, size=(300, 3)),
                               45 + rng.normal(0, 2.5, size=(150, 3))])
    # rows beyond every capacity
    return np.concatenate([rng.uniform(0, 60, size=(500, 3)), 30 + rng.normal(0, 0.8, size=(1300, 3))])


@pytest.mark.parametrize("kind,bins", [
    ("one", (0.0, 5.0, 3, 1)), ("few", (0.0, 5.0, 3, 4)), ("sparse", (1.0, 6.0, 6, 1)),
    ("sparse", (1.0, 6.0, 8, 5)), ("sparse", (1.0, 12.0, 17, 2)), ("sparse", (1.0, 12.0, 20, 1)),
    ("sparse", (1.0, 9.0, 3, 25)), ("lattice", (1.0, 3.0, 4, 4)), ("lattice", (0.0, 3.0, 3, 1)),
    ("clumps", (0.5, 5.0, 5, 1)), ("clumps", (0.5, 5.0, 5, 5)), ("dense", (0.2, 4.0, 4, 1)),
    ("dense", (0.2, 4.0, 3, 3))])
@pytest.mark.parametrize("weighted,buffers", [(False, False), (True, False), (True, True)])
@pytest.mark.parametrize("precision,logbins", [("f32", False), ("f64", False), ("f32", True)])
def test_against_hash_probes(oracle, kind, bins, weighted, buffers, precision, logbins):
    if logbins and not bins[0] > 0.0:
        pytest.skip("log bins need rmin > 0")
    if kind == "dense" and (precision == "f64" or logbins or weighted != buffers):
        pytest.skip("covered by the clumps (the oracle takes seconds on the long rows)")
    rng = np.random.default_rng(7)
    xyz = _points(kind, rng)
    n = len(xyz)
    nd = (n + 1) // 3
    size = rng.lognormal(0.0, 0.3, n) if weighted else np.ones(n)
    w = np.where(np.arange(n) < nd, size, -size)
    buf = (rng.uniform(size=n) < 0.3).astype(np.int32) if buffers else None
    nc = api.ncfg3(bins[2])
    cot = rng.normal(size=(2, nc, bins[3]))
    got = {}
    with api.Context(0) as ctx:
        ctx.set_bins(*bins[:3], nmu=bins[3], logbins=logbins)
        ctx.set_precision(precision)
        for mode in ("hash", "auto"):
            ctx.set_clique_mode(mode)
            ctx.set_catalog(xyz, w, nd, buf)
            three = ctx.count_3pcf()
            stats = ctx.stats()
            sums = ctx.count_3pcf(counts=False)
            equi = ctx.count_equi()
            grad = ctx.adjoint_3pcf(cot[0], cot[1])
            only2 = ctx.adjoint_3pcf(cot[0])
            got[mode] = (three, stats, sums, equi, grad, only2)
        ctx.set_catalog(xyz, size, nd, buf)
        sizes = ctx.adjoint_3pcf(np.abs(cot[0]) + np.abs(cot[1]))
    (t0, s0, _, e0, g0, h0), (t1, s1, u1, e1, g1, h1) = got["hash"], got["auto"]
    pmax = size.max() ** 3
    for a, b in ((t0, t1), (e0, e1)):
        assert np.array_equal(a["counts"], b["counts"])
        tol = 2.0 ** -52 * np.abs(a["catsum"]) * 2 + 2.0 ** -58 * pmax * a["counts"]
        assert np.all(np.abs(a["catsum"] - b["catsum"]) <= tol)
    assert np.array_equal(u1["catsum"], t1["catsum"]) and np.array_equal(u1["N2"], t1["N2"])
    for k in ("tuples", "rooted", "n_edges"):
        assert s0[k] == s1[k], k
    G = oracle.Graph(xyz, *bins, logbins)
    for c3, a, b in ((cot[1], g0, g1), (None, h0, h1)):
        ref = G.adjoint3(w, nd, cot[0], c3, buffer=buf)
        top = np.abs(ref).max()
        assert np.abs(a - ref).max() <= 1e-12 * top and np.abs(b - ref).max() <= 1e-12 * top
        if bins[3] == 1:
            assert np.all(np.abs(b - ref) <= 2.0 ** -42 * sizes)
