"""Members and buffer flags of the regions against their definition: the
planning kernels keep region boxes and member counts per block up to a number
of regions and in global memory beyond it, hold a box in registers while a
warp's points share a region, and test only the neighbouring subcubes within
reach of a point."""
import numpy as np
import pytest

from gramsci_b200 import api, catalogs

pytestmark = pytest.mark.gpu

RMAX = 12.0


def _catalogue(n, box, seed):
    rng = np.random.default_rng(seed)
    xyz = rng.uniform(0.0, box, size=(n, 3))
    w = catalogs.normalise(rng.lognormal(0.0, 0.3, n), n // 3, n - n // 3)
    return rng, xyz, w, n // 3


def _check(regions, xyz, ids, nreg):
    for r in range(nreg):
        own = np.flatnonzero(ids == r)
        members, buf = regions[r]
        if own.size == 0:
            assert members.size == 0
            continue
        lo, hi = xyz[own].min(0) - RMAX, xyz[own].max(0) + RMAX
        inside = np.flatnonzero(((xyz > lo) & (xyz < hi)).all(1))
        assert np.array_equal(members, inside)
        assert np.array_equal(buf != 0, ids[inside] != r)


@pytest.mark.parametrize("nreg,ordered", [(1, False), (40, True), (511, False), (512, True),
                                          (513, False), (700, True), (4097, True)])
def test_region_ids(nreg, ordered):
    rng, xyz, w, n_data = _catalogue(5003, 100.0, nreg)
    ids = rng.integers(0, nreg, len(xyz)).astype(np.int32)
    if ordered:
        ids.sort()
    with api.Context(0) as ctx:
        ctx.set_catalog(xyz, w, n_data)
        ctx.set_bins(1.0, RMAX, 3, nmu=2)
        whole = ctx.count_2pcf()
        ctx.set_region_ids(ids, nreg)
        for _ in range(3):  # planned, captured, replayed
            got = ctx.count_2pcf_batched()
            assert np.array_equal(got["counts"], whole["counts"])
        _check(ctx.regions(), xyz, ids, nreg)


@pytest.mark.parametrize("split,box", [(1, 30.0), (2, 24.2), (3, 36.5), (4, 100.0), (8, 97.0)])
def test_subcubes(split, box):
    # down to subcubes a fraction of a percent wider than rmax
    _, xyz, w, n_data = _catalogue(4001, box, split)
    with api.Context(0) as ctx:
        ctx.set_catalog(xyz, w, n_data)
        ctx.set_bins(1.0, RMAX, 3)
        whole = ctx.count_2pcf()
        ctx.set_regions(split)
        assert np.array_equal(ctx.count_2pcf_batched()["counts"], whole["counts"])
        per = ctx.count_2pcf_regions()
        assert np.array_equal(per["counts"].sum(-1), whole["counts"])
        lo, span = xyz.min(0), np.ptp(xyz, axis=0)
        s = np.minimum(np.floor((xyz - lo) * (1.0 / span) * split).astype(int), split - 1)
        _check(ctx.regions(), xyz, (s[:, 2] * split + s[:, 1]) * split + s[:, 0], split ** 3)


@pytest.mark.parametrize("sizes", [[(5, 7)], [(0, 40), (300, 0), (1, 1), (33, 1000)]])
def test_mock_points(sizes):
    nd, nr = zip(*sizes)
    n = sum(nd) + sum(nr)
    rng = np.random.default_rng(n)
    xyz = rng.uniform(0.0, 30.0, size=(n, 3))
    w = rng.uniform(0.5, 1.0, n)
    with api.Context(0) as ctx:
        ctx.set_catalog(xyz, w, sum(nd))
        ctx.set_bins(1.0, RMAX, 3)
        ctx.set_mocks(nd, nr)
        per = ctx.count_2pcf_regions()
        at = 0
        for m, (g, r) in enumerate(sizes):
            ctx.set_catalog(xyz[at:at + g + r], w[at:at + g + r], g)
            assert np.array_equal(per["counts"][..., m], ctx.count_2pcf()["counts"])
            at += g + r
