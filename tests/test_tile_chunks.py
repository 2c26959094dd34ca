"""The enumeration of the tile pair sweep (gr_tile.cu) restated in numpy: every
chunk of up to 32 consecutive labels of an x-row of cells, taken by the cell
it starts in, against the candidates of its forward ranges (forward_slot in
gr_internal.cuh), shared out over `parts` work items, minus those farther than
rmax from the chunk's box.  Every pair closer than rmax must be met exactly
once, with the larger label as the candidate, and every label read must exist."""
import numpy as np
import pytest


def _grid(xyz, rmax, sub):
    lo, span = xyz.min(0), np.ptp(xyz, axis=0)
    nc = np.maximum(1, np.floor(span / (rmax / sub * 1.000001)).astype(int))
    c = np.minimum(nc - 1, np.floor((xyz - lo) * (nc / np.where(span > 0, span, 1.0))).astype(int))
    key = (c[:, 2] * nc[1] + c[:, 1]) * nc[0] + c[:, 0]
    order = np.argsort(key, kind="stable")
    start = np.concatenate([[0], np.cumsum(np.bincount(key, minlength=nc.prod()))])
    return order, key[order], start, nc


def _slot(k, first, x0, x1, yz, nc, start, sub):
    nx, ny, nz = nc
    cy, cz = yz % ny, yz // ny
    xa, xb = max(0, x0 - sub), min(nx - 1, x1 + sub)
    y, z = cy + k, cz
    if k > sub:
        y = cy - sub + (k - 1 - sub) % (2 * sub + 1)
        z = cz + 1 + (k - 1 - sub) // (2 * sub + 1)
    if not (0 <= y < ny and z < nz):
        return 0, 0
    kb = (z * ny + y) * nx
    b = first if k == 0 else start[kb + xa]
    return b, max(b, start[kb + xb + 1])


def _met(pos, key, start, nc, rmax, sub, parts):
    n, nx = len(pos), nc[0]
    met = np.zeros((n, n), np.int32)
    for cell in range(nc.prod()):
        cb, ce = start[cell], start[cell + 1]
        if cb == ce:
            continue
        cx = cell % nx
        row = cell - cx
        row_beg, row_end = start[row], start[row + nx]
        c0 = row_beg + ((cb - row_beg + 31) & ~31)
        while c0 < ce:
            cend = min(c0 + 32, row_end)
            x1 = key[cend - 1] - row
            assert cx <= x1 < nx
            cand = np.concatenate([np.arange(*_slot(k, c0 + 1, cx, x1, row // nx, nc, start, sub))
                                   for k in range(13 if sub == 2 else 5)]).astype(int)
            assert cand.size == 0 or (cand.min() > c0 and cand.max() < n)
            assert np.all(np.diff(cand) > 0)
            assert np.array_equal(cand[:cend - c0 - 1], np.arange(c0 + 1, cend))
            share = len(cand) if parts == 1 else ((len(cand) + parts - 1) // parts + 31) & ~31
            roots = np.arange(c0, cend)
            lo, hi = pos[roots].min(0), pos[roots].max(0)
            for part in range(parts):
                mine = cand[part * share:(part + 1) * share]
                out = np.maximum(0, np.maximum(lo - pos[mine], pos[mine] - hi))
                mine = mine[(out ** 2).sum(1) <= rmax ** 2]
                for r, p in enumerate(roots):
                    # the first tile leaves out the labels up to the root's
                    skip = r if part == 0 else 0
                    met[p, mine[skip:]] += 1
            c0 += 32
    return met


@pytest.mark.parametrize("parts", [1, 3, 8])
@pytest.mark.parametrize("sub", [1, 2])
@pytest.mark.parametrize("n,box,clump", [(1, 1.0, 0), (40, 9.0, 0), (700, 30.0, 0),
                                         (700, 30.0, 150), (600, 120.0, 0), (300, 4.0, 0)])
def test_every_pair_is_met_once(n, box, clump, sub, parts):
    rng = np.random.default_rng(n + sub)
    xyz = rng.uniform(0, box, size=(n, 3)) * [1.0, 0.7, 0.4]
    if clump:
        xyz[:clump] = xyz[0] + rng.normal(0, 0.5, size=(clump, 3))
    rmax = 5.0
    order, key, start, nc = _grid(xyz, rmax, sub)
    pos = xyz[order]
    met = _met(pos, key, start, nc, rmax, sub, parts)
    d2 = ((pos[:, None] - pos[None]) ** 2).sum(-1)
    near = np.triu(d2 <= rmax ** 2, 1)
    assert met.max(initial=0) <= 1
    assert not np.tril(met).any()
    assert np.all(met[near] == 1)
