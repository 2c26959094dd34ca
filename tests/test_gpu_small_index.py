"""Catalogue scan and cell index: host and device inputs, and the one-launch
index of small catalogues against the passes that larger ones take.

Sizes sit at the edges of the scan's block (1,536 coordinates), of the share
of points whose layout one block writes (256) and of the small-index rule
(16,384 points).  The points are clustered so that most cells hold points of
several shares.  Counts are whole numbers: they must agree exactly with a
direct FP64 sum over all pairs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

RMIN, RMAX = 1.0, 9.0


def _catalogue(n, seed):
    rng = np.random.default_rng(seed)
    centre = rng.uniform(0.0, 60.0, (max(1, n // 200), 3))
    xyz = centre[rng.integers(0, len(centre), n)] + rng.normal(0.0, 4.0, (n, 3))
    n_data = n // 3
    w = rng.uniform(0.5, 1.5, n)
    w[n_data:] *= -1.0
    buf = (rng.uniform(size=n) < 0.2).astype(np.int32)
    return xyz, w, n_data, buf


def _direct(xyz, n_data, buf):
    """Rooted pair counts by category (root not in the buffer)."""
    x = torch.from_numpy(xyz).cuda()
    ran = (torch.arange(len(xyz), device="cuda") >= n_data)
    root = torch.from_numpy(buf).cuda() == 0
    out = np.zeros(4, np.int64)
    for a in range(0, len(xyz), 2048):
        d = x[a:a + 2048, None, :] - x[None, :, :]
        r2 = d[..., 0] * d[..., 0] + d[..., 1] * d[..., 1] + d[..., 2] * d[..., 2]
        m = (r2 >= RMIN * RMIN) & (r2 < RMAX * RMAX)
        i = torch.arange(a, min(a + 2048, len(xyz)), device="cuda")
        m &= i[:, None] != torch.arange(len(xyz), device="cuda")[None, :]
        m &= root[i][:, None]
        for c in range(4):
            sel = m & (ran[i][:, None] == bool(c >> 1)) & (ran[None, :] == bool(c & 1))
            out[c] += int(sel.sum())
    return out


@pytest.mark.parametrize("n", [1, 2, 255, 256, 257, 511, 512, 513, 1025, 4097, 16384, 16385])
def test_small_index_counts(n):
    from gramsci_b200.api import Context

    xyz, w, n_data, buf = _catalogue(n, n)
    ctx = Context()
    ctx.set_bins(RMIN, RMAX, 1)
    got = []
    for dev in (False, True):
        a = [xyz, w, buf]
        if dev:
            a = [torch.from_numpy(v).cuda() for v in a]
            torch.cuda.synchronize()
        ctx.set_catalog(a[0], a[1], n_data, a[2])
        got.append(ctx.count_2pcf())
    for k in got[0]:
        np.testing.assert_array_equal(got[0][k], got[1][k])
    counts = np.asarray(got[0]["counts"]).reshape(-1)
    want = _direct(xyz, n_data, buf)
    assert counts.sum() == want.sum()
    np.testing.assert_array_equal(np.sort(counts), np.sort(want))


def test_one_cell_and_empty_cells():
    """All points in one cell, and a grid whose cells are mostly empty."""
    from gramsci_b200.api import Context

    rng = np.random.default_rng(5)
    for scale, n in ((2.0, 3000), (3000.0, 3000)):
        xyz = rng.uniform(0.0, scale, (n, 3))
        xyz[1::2] = xyz[::2] + 1.5  # pairs at a known separation
        ctx = Context()
        ctx.set_bins(RMIN, RMAX, 1)
        ctx.set_catalog(xyz, np.ones(n), n)
        got = int(np.asarray(ctx.count_2pcf()["counts"]).sum())
        assert got == _direct(xyz, n, np.zeros(n, np.int32)).sum()


@pytest.mark.parametrize("dev", [False, True])
def test_non_finite_is_refused_where_it_was(dev):
    """A weight by set_catalog, a coordinate by the count."""
    from gramsci_b200.api import Context
    from gramsci_b200._native import GramsciError

    put = (lambda v: torch.from_numpy(v).cuda()) if dev else (lambda v: v)
    xyz, w, n_data, _ = _catalogue(700, 3)
    ctx = Context()
    ctx.set_bins(RMIN, RMAX, 1)
    bad = w.copy()
    bad[699] = np.nan
    with pytest.raises(GramsciError):
        ctx.set_catalog(put(xyz), put(bad), n_data)
    worse = xyz.copy()
    worse[511, 2] = np.inf
    ctx.set_catalog(put(worse), put(w), n_data)
    with pytest.raises(GramsciError):
        ctx.count_2pcf()
    ctx.set_catalog(put(xyz), put(w), n_data)
    assert np.asarray(ctx.count_2pcf()["counts"]).sum() > 0


@pytest.mark.parametrize("n,pinned", [(700, True), (700, False), (5000, True)])
def test_device_entry_takes_what_a_copy_takes(n, pinned):
    """gr_set_catalog_dev: device arrays are read in place, also from the
    middle of an allocation; pinned host memory, which a device-to-device copy
    accepts, is still copied."""
    import ctypes

    from gramsci_b200.api import Context

    xyz, w, n_data, _ = _catalogue(n, 11)
    ctx = Context()
    ctx.set_bins(RMIN, RMAX, 4)
    ctx.set_catalog(xyz, w, n_data)
    want = ctx.count_2pcf()
    if pinned:
        x, v = torch.from_numpy(xyz).pin_memory(), torch.from_numpy(w).pin_memory()
    else:
        room = torch.zeros(4 * n + 7, dtype=torch.float64, device="cuda")
        x, v = room[3:3 + 3 * n], room[5 + 3 * n:5 + 4 * n]
        x.copy_(torch.from_numpy(xyz.ravel()))
        v.copy_(torch.from_numpy(w))
        torch.cuda.synchronize()
    ctx._check(ctx._lib.gr_set_catalog_dev(ctx._h, ctypes.c_void_p(x.data_ptr()),
                                           ctypes.c_void_p(v.data_ptr()), None, n_data, n - n_data))
    ctx.n = n
    got = ctx.count_2pcf()
    for k in want:
        np.testing.assert_array_equal(want[k], got[k])
