"""-tetra against the oracle from one bin to the most that are taken, with rows
of a few members and of more than the pair bins are kept for, separations on
the bins' edges (a lattice: many regular tetrahedra in one bin) and buffer
points.  Counts are equal to the oracle's; sums, which the oracle adds in FP64
and the kernels exactly, are compared with the hash-probe kernel's: within
three roundings of each product and the rounding of each to 2^-59 of the
largest."""
import numpy as np
import pytest

from gramsci_b200 import api

pytestmark = pytest.mark.gpu


def _points(kind, rng):
    if kind == "lattice":  # face-centred: neighbours at equal distances
        g = np.stack(np.meshgrid(*[np.arange(9.0)] * 3), -1).reshape(-1, 3)
        return rng.permutation(g[g.sum(1) % 2 == 0])
    if kind == "sparse":
        return rng.uniform(0.0, 14.0, size=(900, 3))
    return np.concatenate([rng.uniform(0, 30, size=(250, 3)), 15 + rng.normal(0, 0.7, size=(260, 3))])


@pytest.mark.parametrize("kind", ["lattice", "sparse", "dense"])
@pytest.mark.parametrize("nbins", [1, 4, 60, 127])
@pytest.mark.parametrize("weighted,buffers", [(False, False), (True, False), (True, True)])
def test_against_oracle(oracle, kind, nbins, weighted, buffers):
    rng = np.random.default_rng(5)
    xyz = _points(kind, rng)
    n, nd = len(xyz), len(xyz) // 3
    size = rng.lognormal(0.0, 0.3, n) if weighted else np.ones(n)
    w = np.where(np.arange(n) < nd, size, -size)
    buf = (rng.uniform(size=n) < 0.2).astype(np.int32) if buffers else None
    bins = (1.0, 3.0, nbins)
    ref = oracle.Graph(xyz, *bins).tetra(w, nd, buffer=buf)
    with api.Context(0) as ctx:
        ctx.set_catalog(xyz, w, nd, buf)
        ctx.set_bins(*bins)
        got = ctx.count_tetra()
        stats = ctx.stats()
        ctx.set_clique_mode("hash")
        probes = ctx.count_tetra()
    for c, s, p in (("counts", "catsum", 4), ("dcount", "dsum", 3)):
        np.testing.assert_array_equal(got[c], ref[c])
        tol = 2.0 ** -50 * np.abs(probes[s]) + 2.0 ** -58 * size.max() ** p * ref[c]
        assert np.all(np.abs(got[s] - probes[s]) <= tol)
        assert np.all(np.abs(got[s] - ref[s]) <= 1e-12 * np.abs(ref[s]).max())
    assert stats["rooted"] == ref["counts"].sum() and (nbins > 4 or stats["rooted"] > 0)
