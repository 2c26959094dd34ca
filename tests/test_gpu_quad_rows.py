"""The geometric 4-clique kernel against the hash-probe kernel at the row
lengths where it changes: rows of a block's short and long warps (64 members),
kept and recomputed pair bins (128), its longest row (255; one more goes to the
hash probes), rows split into parts (32, 48, 64, 96, 128), catalogues of long
rows alone.  A clump of m points that are all neighbours has rows of m - 1, m -
2, ... members; labels and catalogue ids differ.  Both kernels form the same
products of the id-ordered weights and round them alike: every array is
identical, gradients included."""
import numpy as np
import pytest

from gramsci_b200 import api

pytestmark = pytest.mark.gpu


def _catalogue(m, background, rng):
    clump = 20.0 + rng.uniform(0.0, 1.1, size=(m, 3))  # all closer than 2
    rest = rng.uniform(0.0, 40.0, size=(background, 3))
    return rng.permutation(np.concatenate([clump, rest]))


@pytest.mark.parametrize("m,background", [(4, 0), (20, 300), (33, 300), (49, 200), (64, 500),
                                          (65, 3000), (66, 3000), (97, 3000), (129, 3000),
                                          (130, 0), (160, 4000), (256, 6000), (257, 6000)])
@pytest.mark.parametrize("weighted,buffers", [(False, False), (True, True)])
@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_rows(m, background, weighted, buffers, precision):
    rng = np.random.default_rng(m)
    xyz = _catalogue(m, background, rng)
    n = len(xyz)
    nd = n // 3
    w = rng.lognormal(0.0, 0.3, n) if weighted else np.ones(n)
    w[nd:] *= -1.0
    buf = (rng.uniform(size=n) < 0.3).astype(np.int32) if buffers else None
    got = {}
    with api.Context(0) as ctx:
        ctx.set_catalog(xyz, w, nd, buf)
        ctx.set_bins(0.05, 2.0, 3)
        ctx.set_precision(precision)
        for mode in ("hash", "geometric"):
            ctx.set_clique_mode(mode)
            four = ctx.count_4pcf()
            stats = ctx.stats()
            sums = ctx.count_4pcf(counts=False)
            tetra = ctx.count_tetra()
            cots = [np.random.default_rng(3).normal(size=four[k].shape)
                    for k in ("N2", "N3", "discN", "discR")]
            got[mode] = (four, sums, tetra, ctx.adjoint_4pcf(*cots), ctx.adjoint_4pcf(cots[0]),
                         stats["tuples"], stats["rooted"])
    a, b = got["hash"], got["geometric"]
    for x, y in zip(a[:3], b[:3]):
        for k in x:
            assert np.array_equal(x[k], y[k]), k
    assert np.array_equal(a[3], b[3]) and np.array_equal(a[4], b[4])
    assert a[5:] == b[5:]
    # (a root has more than three neighbours)
    assert m < 5 or int(b[0]["counts"].sum()) > 0
