"""The longest rows of the geometric 4-clique kernel, 255 and 256 members, and
one more (hash probes), against the hash-probe kernel: the same arrays, with
the root's catalogue id before, among and after its members'."""
import numpy as np
import pytest

from gramsci_b200 import api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("row", [254, 255, 256, 257])
@pytest.mark.parametrize("place", ["first", "middle", "last"])
def test_arrays(row, place):
    rng = np.random.default_rng(row)
    # one root sees every other point, no label is smaller than its own (it lies
    # in the first cell); the others fall into groups that see each other little
    m = row + 1
    xyz = 10.0 + rng.uniform(0.0, 1.1, size=(m, 3))
    xyz[row] = 9.9
    rest = rng.uniform(12.5, 30.0, size=(400, 3))
    if place == "first":
        order = np.concatenate([[row], np.arange(row)])
    elif place == "middle":
        order = np.concatenate([np.arange(row // 2), [row], np.arange(row // 2, row)])
    else:
        order = np.arange(m)
    xyz = np.concatenate([xyz[order], rest])
    n, nd = len(xyz), m // 3
    w = rng.lognormal(0.0, 0.3, n)
    w[nd:] *= -1.0
    got = {}
    with api.Context(0) as ctx:
        ctx.set_catalog(xyz, w, nd)
        ctx.set_bins(0.05, 2.2, 3)
        longest = np.diff(ctx.graph()[0]).max()
        for mode in ("hash", "auto"):
            ctx.set_clique_mode(mode)
            four, tetra = ctx.count_4pcf(), ctx.count_tetra()
            cot = np.random.default_rng(3)
            grad = ctx.adjoint_4pcf(*[cot.normal(size=four[k].shape) for k in ("N2", "N3", "discN", "discR")])
            got[mode] = (four, tetra, {"grad": grad})
    assert longest >= row
    for a, b in zip(got["hash"], got["auto"]):
        for k in a:
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)
