"""The workloads whose speed this framework is judged by, each a call that a
user's program makes: a catalogue of galaxies and randoms that lies in GPU
memory is handed to a context and its 2-, 3- or 4-point counts are taken, or
the differentiable counts are run forward and backward.

Sizes are those of the named workloads of gramsci_b200.catalogs (the same
number densities, clustering, radii and bins), whole or cut to a smaller box,
and those that the tests run.  A case is a dict:

  query     2, 3 or 4 points
  call      "count" (one catalogue), "regions" (split^3 subcubes in one
            launch), "mocks" (independent catalogues in one launch, a table
            each) or "grad" (torch.autograd, forward and backward)
  n_gal, n_rand, box, children, sigma, ramp
            galaxies (Neyman-Scott clusters of `children` on average with
            Gaussian offsets, uniform when 0; `ramp`: parent density along
            x), uniform randoms, box edge
  weights   "unit" or "lognormal"
  buffer    whether the points of the outer shell, rmax wide, are buffer
            points (neighbours that are no roots)
  counts    whether the integer counts are asked for (3- and 4-point counts)
  rmin, rmax, nbins, nmu, log
            the bins
"""
import math

import numpy as np
import torch

from gramsci_b200 import api, autograd


def _case(name, query, call, n_gal, n_rand, box, rmin, rmax, nbins, nmu=1, log=False, children=0,
          sigma=0.0, ramp=1.0, weights="unit", buffer=False, counts=True, split=1, mocks=1):
    return dict(name=name, query=query, call=call, n_gal=n_gal, n_rand=n_rand, box=float(box),
                rmin=float(rmin), rmax=float(rmax), nbins=nbins, nmu=nmu, log=log,
                children=children, sigma=float(sigma), ramp=float(ramp), weights=weights,
                buffer=buffer, counts=counts, split=split, mocks=mocks)


def listed():
    return [
        # a small box as a notebook or a unit of a larger job counts it: latency and launches
        _case("2pcf_tiny", 2, "count", 1000, 2500, 368.4, 10, 50, 10),
        # the plain 2PCF workload (c1_2pcf): one box of a parameter scan
        _case("2pcf_box", 2, "count", 20000, 50000, 1000, 10, 50, 10),
        # small scales on logarithmic bins, weighted: projected clustering of one sample
        _case("2pcf_log", 2, "count", 60013, 180001, 843.7, 1, 25, 12, log=True, children=10,
              sigma=4, weights="lognormal"),
        # the weight gradient of a dense survey catalogue (c5_adjoint, 2PCF part)
        _case("2pcf_grad", 2, "grad", 1000000, 2000000, 1000, 10, 40, 10, nmu=4, children=10,
              sigma=5, weights="lognormal"),
        # a large survey in 5^3 subvolumes (c4_batched)
        _case("2pcf_regions", 2, "regions", 4000000, 8000000, 2000, 10, 60, 12, nmu=10,
              children=10, sigma=5, ramp=8, split=5),
        # a covariance from many small mocks in one call, a table for each
        _case("2pcf_mocks", 2, "mocks", 2000, 5000, 464.2, 10, 50, 10, nmu=4, children=10,
              sigma=4, weights="lognormal", mocks=50),
        # a small 3PCF catalogue (c3's share of a box 215 on a side)
        _case("3pcf_tiny", 3, "count", 1000, 3000, 215.4, 5, 25, 8, nmu=5, children=10, sigma=4,
              weights="lognormal"),
        # the 3PCF workload (c2_3pcf) as the command runs it: sums without integer counts
        _case("3pcf_survey", 3, "count", 100000, 300000, 1000, 5, 25, 8, nmu=5, children=10,
              sigma=4, weights="lognormal", counts=False),
        # one subvolume of a decomposed survey: unit weights, a buffer shell, no mu bins
        _case("3pcf_region", 3, "count", 39989, 120011, 736.8, 5, 25, 8, children=10, sigma=4,
              buffer=True),
        # the 3PCF weight gradient at high neighbour numbers (c5_adjoint in a smaller box)
        _case("3pcf_grad", 3, "grad", 200000, 400000, 584.8, 10, 30, 6, children=10, sigma=5,
              weights="lognormal"),
        # the 4PCF workload (c3_4pcf): unit weights
        _case("4pcf_unit", 4, "count", 30000, 90000, 300, 2, 12, 4, children=20, sigma=3),
        # the same catalogue weighted, forward and backward
        _case("4pcf_grad", 4, "grad", 30000, 90000, 300, 2, 12, 4, children=20, sigma=3,
              weights="lognormal"),
    ]


def _between(rng, lo, hi):
    """An integer between lo and hi, uniform in its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["2pcf", "2pcf", "2pcf_grad", "2pcf_regions", "2pcf_mocks", "3pcf", "3pcf",
                       "3pcf_grad", "4pcf", "4pcf_grad"])
    weights = rng.choice(["unit", "lognormal"])
    # number density relative to the listed workload's
    dense = rng.uniform(0.6, 1.2)
    if kind == "2pcf":
        n = _between(rng, 1000, 1000000)
        return _case("", 2, "count", n, int(2.5 * n), 1000 * (n / (20000 * dense)) ** (1 / 3),
                     rng.choice([1, 10]), rng.uniform(30, 60), rng.randint(5, 15),
                     nmu=rng.choice([1, 4, 10]), log=rng.random() < 0.25,
                     children=rng.choice([0, 10]), sigma=4, weights=weights,
                     buffer=rng.random() < 0.2)
    if kind == "2pcf_grad":
        n = _between(rng, 10000, 900000)
        return _case("", 2, "grad", n, 2 * n, 1000 * (n / (1e6 * dense)) ** (1 / 3), 10,
                     rng.uniform(25, 40), rng.randint(5, 12), nmu=rng.choice([1, 4]), children=10,
                     sigma=5, weights="lognormal")
    if kind == "2pcf_regions":
        n = _between(rng, 100000, 3000000)
        return _case("", 2, "regions", n, 2 * n, 2000 * (n / (4e6 * dense)) ** (1 / 3), 10,
                     rng.uniform(40, 60), rng.randint(8, 14), nmu=rng.choice([1, 10]), children=10,
                     sigma=5, ramp=rng.uniform(1, 8), weights=weights, split=rng.randint(2, 5))
    if kind == "2pcf_mocks":
        n = _between(rng, 500, 5000)
        return _case("", 2, "mocks", n, int(2.5 * n), 1000 * (n / (20000 * dense)) ** (1 / 3), 10,
                     rng.uniform(30, 55), rng.randint(5, 15), nmu=rng.choice([1, 4]), children=10,
                     sigma=4, weights=weights, mocks=rng.randint(3, 80))
    if kind == "3pcf":
        n = _between(rng, 1000, 130000)
        return _case("", 3, "count", n, 3 * n, 1000 * (n / (1e5 * dense)) ** (1 / 3),
                     rng.choice([2, 5]), rng.uniform(18, 30), rng.randint(4, 10),
                     nmu=rng.choice([1, 5, 8]), children=10, sigma=4, weights=weights,
                     buffer=rng.random() < 0.3, counts=rng.random() < 0.5)
    if kind == "3pcf_grad":
        n = _between(rng, 3000, 170000)
        return _case("", 3, "grad", n, 2 * n, 1000 * (n / (1e6 * dense)) ** (1 / 3), 10,
                     rng.uniform(15, 28), rng.randint(4, 8), nmu=rng.choice([1, 1, 5]),
                     children=10, sigma=5, weights="lognormal")
    n = _between(rng, 1500, 40000)
    return _case("", 4, "grad" if kind == "4pcf_grad" else "count", n, 3 * n,
                 300 * (n / (30000 * dense)) ** (1 / 3), 2, rng.uniform(8, 12), rng.randint(3, 5),
                 children=20, sigma=3, weights="lognormal" if kind == "4pcf_grad" else weights,
                 counts=rng.random() < 0.5)


def _mock(case, gen):
    """One catalogue: positions (galaxies first), signed normalised weights
    and the number of galaxies."""
    box, dev = case["box"], "cuda"

    def uniform(n):
        return torch.rand((n, 3), generator=gen, device=dev, dtype=torch.float64) * box

    if case["children"]:
        parents = uniform(max(1, case["n_gal"] // case["children"]))
        a = case["ramp"] - 1.0
        if a > 0.0:  # parent density proportional to 1 + a x / box
            u = parents[:, 0] / box
            parents[:, 0] = box * (torch.sqrt(1.0 + a * (a + 2.0) * u) - 1.0) / a
        own = torch.randint(len(parents), (case["n_gal"],), generator=gen, device=dev)
        gal = parents[own]
        gal += case["sigma"] * torch.randn(gal.shape, generator=gen, device=dev,
                                           dtype=torch.float64)
    else:
        gal = uniform(case["n_gal"])
    xyz = torch.cat([gal, uniform(case["n_rand"])])
    w = torch.ones(len(xyz), device=dev, dtype=torch.float64)
    if case["weights"] == "lognormal":
        w = torch.exp(0.3 * torch.randn(len(xyz), generator=gen, device=dev, dtype=torch.float64))
    n_gal = len(gal)
    return xyz, torch.cat([w[:n_gal] / w[:n_gal].sum(), -w[n_gal:] / w[n_gal:].sum()]), n_gal


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    parts = [_mock(case, gen) for _ in range(case["mocks"])]
    xyz = torch.cat([p[0] for p in parts]) if len(parts) > 1 else parts[0][0]
    w = torch.cat([p[1] for p in parts]) if len(parts) > 1 else parts[0][1]
    s = dict(xyz=xyz, w=w, n_data=parts[0][2], buffer=None,
             n_gal=[p[2] for p in parts], n_rand=[len(p[0]) - p[2] for p in parts])
    if case["buffer"]:
        r, box = case["rmax"], case["box"]
        inner = ((xyz > r) & (xyz < box - r)).all(1)
        s["buffer"] = (~inner).to(torch.int32)
    if case["call"] == "grad":
        s["cot"] = [torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
                    for shape in _shapes(case)]
    return s


def _shapes(case):
    """Shapes of the differentiable outputs: N2, N3 (and discN, discR)."""
    nb, nm = case["nbins"], case["nmu"]
    if case["query"] == 2:
        return [(nb, nm)] * 2
    if case["query"] == 3:
        return [(api.ncfg3(nb), nm)] * 2
    nc = api.ncfg4(nb)
    return [(nc, nb, nb)] * 2 + [(nc, nb, nb, 6)] * 2


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    if case["call"] == "grad":
        s["w"].requires_grad_(True)
        return s
    s["ctx"] = api.Context(0)
    s["ctx"].set_bins(case["rmin"], case["rmax"], case["nbins"], case["nmu"], case["log"])
    if case["call"] == "regions":
        s["ctx"].set_regions(case["split"])
    return s


def run(s):
    case = s["case"]
    if case["call"] == "grad":
        bins = (case["rmin"], case["rmax"], case["nbins"])
        if case["query"] < 4:
            bins += (case["nmu"],)
        pcf = {2: autograd.pcf2, 3: autograd.pcf3, 4: autograd.pcf4}[case["query"]]
        out = pcf(s["w"], s["xyz"], s["n_data"], *bins)
        loss = sum((c * o).sum() for c, o in zip(s["cot"], out))
        grad, = torch.autograd.grad(loss, s["w"])
        return dict(sums=[o.detach() for o in out], grad=grad)
    ctx = s["ctx"]
    ctx.set_catalog(s["xyz"], s["w"], s["n_data"], s["buffer"])
    if case["call"] == "regions":
        return ctx.count_2pcf_batched()
    if case["call"] == "mocks":
        ctx.set_mocks(s["n_gal"], s["n_rand"])
        return ctx.count_2pcf_regions()
    if case["query"] == 2:
        return ctx.count_2pcf()
    if case["query"] == 3:
        return ctx.count_3pcf(counts=case["counts"])
    return ctx.count_4pcf(counts=case["counts"])


def _expected(case):
    """Points, and expected pairs and tuples of a catalogue (per mock summed):
    uniform density plus the cluster that a galaxy shares."""
    n_gal, n_rand, r = case["n_gal"], case["n_rand"], case["rmax"]
    n = n_gal + n_rand
    per_volume = n / case["box"] ** 3
    mean = per_volume * 4.0 / 3.0 * math.pi * r ** 3  # uniform neighbours of a point
    own = case["children"] * (1.0 if r > 4.0 * case["sigma"] else (r / (4.0 * case["sigma"])) ** 3)
    pairs = 0.5 * (n * mean + n_gal * own)
    tuples = pairs
    if case["query"] >= 3:
        # two neighbours of a point in a ball are neighbours with chance 15/32
        tri = (n_rand * mean ** 2 + n_gal * (mean + own) ** 2) * (15.0 / 32.0) / 6.0
        tuples = tri
    if case["query"] == 4:
        tuples = (n_rand * mean ** 3 + n_gal * (mean + own) ** 3) * (15.0 / 32.0) ** 3 / 24.0
    return n * case["mocks"], pairs * case["mocks"], tuples * case["mocks"]


def work(case):
    n, pairs, tuples = _expected(case)
    values = sum(int(np.prod(shape)) for shape in _shapes(case)) * case["mocks"]
    byte = 32 * n + (4 * n if case["buffer"] else 0) + 8 * values
    # a separation, its bin and (with mu bins) the line-of-sight cosine of each
    # pair; for each tuple the product of its weights and one sum per root
    flops = pairs * (12 + (16 if case["nmu"] > 1 else 0)) + tuples * 2 * case["query"]
    if case["call"] == "grad":
        byte += 16 * n + 8 * values
        flops += tuples * 3 * case["query"]
    return dict(bytes=int(byte), flops=int(flops))


# ---------------------------------------------------------------- 64 bits --
# The same counts in plain torch: all neighbour pairs by comparing slabs of
# points sorted by x, triangles and 4-cliques by looking up the edges among a
# root's neighbours.

_MOST_TESTS = 4e11   # separations compared
_MOST_TUPLES = 3e9   # tuples looked up


def _edges(xyz, case):
    """Directed edges (i, j, radial bin, mu bin), bins from 0, sorted by (i, j)."""
    rmin, rmax, nb, nm = case["rmin"], case["rmax"], case["nbins"], case["nmu"]
    order = torch.argsort(xyz[:, 0])
    p = xyz[order]
    found = []
    step = 2048
    for a in range(0, len(p), step):
        q = p[a:a + step]
        lo = int(torch.searchsorted(p[:, 0].contiguous(), q[0, 0] - 1.01 * rmax))
        hi = int(torch.searchsorted(p[:, 0].contiguous(), q[-1, 0] + 1.01 * rmax))
        c = p[lo:hi]
        d2 = (q[:, None, 0] - c[None, :, 0]) ** 2
        d2 += (q[:, None, 1] - c[None, :, 1]) ** 2
        d2 += (q[:, None, 2] - c[None, :, 2]) ** 2
        i, j = torch.nonzero(d2 < rmax * rmax * 1.001, as_tuple=True)
        i, j = i + a, j + lo
        keep = i != j
        found.append((order[i[keep]], order[j[keep]]))
    i = torch.cat([f[0] for f in found])
    j = torch.cat([f[1] for f in found])
    d = xyz[j] - xyz[i]
    s2 = d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1] + d[:, 2] * d[:, 2]
    s = torch.sqrt(s2)
    keep = (s > rmin) & (s < rmax)
    i, j, d, s, s2 = i[keep], j[keep], d[keep], s[keep], s2[keep]
    if case["log"]:
        t = (torch.log10(s) - math.log10(rmin)) * (1.0 / ((math.log10(rmax) - math.log10(rmin)) / nb))
    else:
        t = (s - rmin) * (1.0 / ((rmax - rmin) / nb))
    b = torch.floor(t).long().clamp(0, nb - 1)
    mu = torch.zeros_like(b)
    if nm >= 2:
        m = 0.5 * (xyz[i] + xyz[j])
        th = -(m[:, 0] * d[:, 0] + m[:, 1] * d[:, 1] + m[:, 2] * d[:, 2])
        m2 = m[:, 0] * m[:, 0] + m[:, 1] * m[:, 1] + m[:, 2] * m[:, 2]
        th = th / (torch.sqrt(m2) * torch.sqrt(s2))
        mu = torch.floor((th + 1.0) * (0.5 * nm)).long().clamp(0, nm - 1)
    o = torch.argsort(i * len(xyz) + j)
    return i[o], j[o], b[o], mu[o]


def _normal_table(nm):
    """The mu bin of a triangle from those of the root's two edges, in single
    precision as the method defines it."""
    f = np.float32
    m = (((np.arange(1, nm + 1).astype(f) - f(0.5)).astype(np.float64)) / (0.5 * nm) - 1.0).astype(f)
    a, b = m[:, None], m[None, :]
    with np.errstate(invalid="ignore"):
        v = f(1.1547) * np.sqrt(((f(0.75) - a * a) - b * b) + a * b) * f(nm)
    v = np.where(np.isnan(v), f(0), np.floor(v)).astype(np.int64)
    return torch.from_numpy(np.clip(v, 0, nm - 1)).cuda()


def _ranks(nb, k):
    """Lexicographic rank of the non-decreasing k-tuples of bins, -1 for others."""
    table = torch.full((nb,) * k, -1, dtype=torch.long)
    rank = 0
    for t in np.ndindex(*(nb,) * k):
        if all(t[q] <= t[q + 1] for q in range(k - 1)):
            table[t] = rank
            rank += 1
    return table.cuda()


def _grow(start, length, at):
    """For every element e of `at`: the positions start[e] .. start[e] + length[e],
    flattened, with the element each belongs to."""
    own = torch.repeat_interleave(torch.arange(len(at), device=at.device), length)
    first = torch.cumsum(length, 0) - length
    return own, start[own] + torch.arange(len(own), device=at.device) - first[own]


def _chunks(weight, most):
    """Slices of consecutive elements whose weights sum to about `most`."""
    total = torch.cumsum(weight, 0)
    a = 0
    while a < len(weight):
        base = total[a - 1] if a else total.new_zeros(())
        b = max(a + 1, int(torch.searchsorted(total, base + most, right=True)))
        yield a, b
        a = b


class _Sums:
    """Sums of products of weights by bin, and the gradient of their dot
    product with cotangents."""

    def __init__(self, w, cot=None):
        self.w, self.cot = w, cot
        self.grad = torch.zeros_like(w) if cot is not None else None

    def add(self, out, which, k, ids, sign=1.0):
        p = self.w[ids[0]]
        for i in ids[1:]:
            p = p * self.w[i]
        out.index_add_(0, k, sign * p)
        if self.cot is None or which is None:
            return
        c = sign * self.cot[which][k]
        for q, i in enumerate(ids):
            g = c
            for o, j in enumerate(ids):
                if o != q:
                    g = g * self.w[j]
            self.grad.index_add_(0, i, g)


def _flat(t):
    """Flattened with the first index fastest, as the tables are laid out."""
    return t.permute(*reversed(range(t.dim()))).reshape(-1)


def _shaped(t, *shape):
    return t.reshape(shape[::-1]).permute(*reversed(range(len(shape))))


def _one_exact(case, xyz, w, n_data, buffer, cot):
    """N2, N3 (discN, discR), the sums by category and the gradient."""
    nb, nm, query = case["nbins"], case["nmu"], case["query"]
    i, j, b, mu = _edges(xyz, case)
    ran = (torch.arange(len(w), device=w.device) >= n_data).long()
    root = torch.ones_like(ran, dtype=torch.bool) if buffer is None else buffer == 0
    S = _Sums(w, None if cot is None else [_flat(c) for c in cot])

    def zeros(n):
        return torch.zeros(n, dtype=torch.float64, device=w.device)

    if query == 2:
        keep = root[i]
        i, j, k = i[keep], j[keep], (b + nb * mu)[keep]
        n = nb * nm
        N2, N3, cat = zeros(n), zeros(n), zeros(4 * n)
        both = (ran[i] * ran[j]) > 0
        S.add(N2, 0, k, (i, j))
        S.add(N3, 1, k[both], (i[both], j[both]))
        S.add(cat, None, k + n * (2 * ran[i] + ran[j]), (i, j))
        return dict(N2=_shaped(N2, nb, nm), N3=_shaped(N3, nb, nm),
                    catsum=_shaped(cat, nb, nm, 4)), S.grad

    # for each edge (i, a): the later entries c of i's row, kept when (a, c) is an edge
    n_pt = len(w)
    key = i * n_pt + j
    end = torch.cumsum(torch.bincount(i, minlength=n_pt), 0)
    later = end[i] - torch.arange(len(i), device=i.device) - 1
    if query == 4:  # roots with at most three neighbours count nothing
        root = root & (torch.bincount(i, minlength=n_pt) > 3)
    later = torch.where(root[i], later, torch.zeros_like(later))
    if float(later.sum()) > _MOST_TUPLES:
        return None
    normal = _normal_table(nm)
    cfg_of = _ranks(nb, 3 if query == 3 else 4)
    nc = api.ncfg3(nb) if query == 3 else api.ncfg4(nb)
    n = nc * nm if query == 3 else nc * nb * nb
    N2, N3 = zeros(n), zeros(n)
    cat = zeros((4 if query == 3 else 5) * n)
    dN, dR, dcat = (zeros(6 * n), zeros(6 * n), zeros(24 * n)) if query == 4 else (None,) * 3
    disc = ((3, 0, 1), (3, 0, 2), (1, 0, 3), (0, 1, 2), (0, 3, 2), (0, 3, 1))
    for lo, hi in _chunks(later, 2e7):
        own, e2 = _grow(torch.arange(lo, hi, device=i.device) + 1, later[lo:hi],
                        torch.arange(lo, hi, device=i.device))
        e1 = own + lo
        at = torch.searchsorted(key, j[e1] * n_pt + j[e2]).clamp(max=len(key) - 1)
        hit = key[at] == j[e1] * n_pt + j[e2]
        e1, e2, e3 = e1[hit], e2[hit], at[hit]
        if query == 3:
            s = torch.sort(torch.stack([b[e1], b[e2], b[e3]]), 0)[0]
            k = cfg_of[s[0], s[1], s[2]]
            if nm >= 2:
                k = k + nc * normal[mu[e1], mu[e2]]
            ids = (i[e1], j[e1], j[e2])
            nr = ran[ids[0]] + ran[ids[1]] + ran[ids[2]]
            S.add(N2, 0, k, ids)
            S.add(N3, 1, k[nr == 3], tuple(v[nr == 3] for v in ids), -1.0)
            S.add(cat, None, k + n * nr, ids)
            continue
        for a, z in _chunks(later[e2], 2e7):
            own, e4 = _grow(e2[a:z] + 1, later[e2[a:z]], e2[a:z])
            f1, f2, f3 = e1[a:z][own], e2[a:z][own], e3[a:z][own]
            want = j[f2] * n_pt + j[e4]
            at5 = torch.searchsorted(key, want).clamp(max=len(key) - 1)
            want6 = j[f1] * n_pt + j[e4]
            at6 = torch.searchsorted(key, want6).clamp(max=len(key) - 1)
            hit = (key[at5] == want) & (key[at6] == want6)
            f1, f2, f3, e4, at5, at6 = (v[hit] for v in (f1, f2, f3, e4, at5, at6))
            k = cfg_of[b[f1], b[f3], b[at5], b[e4]]
            good = k >= 0
            f1, f2, e4, at6, k = (v[good] for v in (f1, f2, e4, at6, k))
            k = k + nc * (b[f2] + nb * b[at6])
            ids = (i[f1], j[f1], j[f2], j[e4])
            r = [ran[v] for v in ids]
            nr = r[0] + r[1] + r[2] + r[3]
            S.add(N2, 0, k, ids)
            S.add(N3, 1, k[nr == 4], tuple(v[nr == 4] for v in ids))
            S.add(cat, None, k + n * nr, ids)
            for t, (g, u, v) in enumerate(disc):
                on = r[g] > 0
                kt, pu, pv = k[on] + n * t, ids[u][on], ids[v][on]
                npr = ran[pu] + ran[pv]
                S.add(dN, 2, kt, (pu, pv))
                S.add(dcat, None, kt + 6 * n * npr, (pu, pv))
                S.add(dR, 3, kt[npr == 2], (pu[npr == 2], pv[npr == 2]))
                S.add(dcat, None, kt[npr == 2] + 18 * n, (pu[npr == 2], pv[npr == 2]))
    if query == 3:
        return dict(N2=_shaped(N2, nc, nm), N3=_shaped(N3, nc, nm),
                    catsum=_shaped(cat, nc, nm, 4)), S.grad
    return dict(N2=_shaped(N2, nc, nb, nb), N3=_shaped(N3, nc, nb, nb),
                discN=_shaped(dN, nc, nb, nb, 6), discR=_shaped(dR, nc, nb, nb, 6),
                catsum=_shaped(cat, nc, nb, nb, 5), dsum=_shaped(dcat, nc, nb, nb, 6, 4)), S.grad


def exact(case, seed):
    n, pairs, tuples = _expected(case)
    slab = min(1.0, 2.5 * case["rmax"] / case["box"])
    lookups = tuples * {2: 1, 3: 8, 4: 60}[case["query"]]
    if n * n / case["mocks"] * slab > _MOST_TESTS or pairs > 4e8 or lookups > _MOST_TUPLES:
        return None
    s = _inputs(case, seed)
    if case["call"] == "mocks":
        parts, at = [], 0
        for g, r in zip(s["n_gal"], s["n_rand"]):
            parts.append(_one_exact(case, s["xyz"][at:at + g + r], s["w"][at:at + g + r], g, None,
                                    None)[0])
            at += g + r
        out = {k: torch.stack([p[k] for p in parts], -1) for k in parts[0]}
        out["counts"] = None
        return out
    found = _one_exact(case, s["xyz"], s["w"], s["n_data"], s["buffer"], s.get("cot"))
    if found is None:
        return None
    out, grad = found
    if case["call"] == "grad":
        names = ("N2", "N3", "discN", "discR") if case["query"] == 4 else ("N2", "N3")
        return dict(sums=[out[k] for k in names], grad=grad)
    if case["query"] < 4 and case["counts"]:
        out["counts"] = None
    if case["query"] == 4 and case["counts"]:
        out["counts"] = out["dcount"] = None
    return out
