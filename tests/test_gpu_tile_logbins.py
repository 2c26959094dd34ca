"""Tile pair sweep on logarithmic bins: FP32 binning with the guard band
against the FP64 form.  Every sum is an exact fixed-point integer and the
guard sends every undecided pair to FP64, so all arrays are identical.  The
lattice puts separations on bin edges (bins of a factor 2 or sqrt 2 from 1);
the far catalogue's coordinates are too large for the FP32 form at its
smallest separations, or leave a wide guard."""
import numpy as np
import pytest

from gramsci_b200 import api

pytestmark = pytest.mark.gpu


def _points(kind, n):
    rng = np.random.default_rng(n)
    if kind == "lattice":
        xyz = np.stack(np.meshgrid(*[np.arange(11.0)] * 3), -1).reshape(-1, 3)
        return rng.permutation(xyz)[:n] - 5.0, rng
    xyz = rng.uniform(-9.0, 9.0, size=(n, 3))
    if kind == "far":
        xyz += 3000.0
    if kind == "farther":
        xyz += 1.0e6
    return xyz, rng


@pytest.mark.parametrize("variant", [6, 7])
@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("rmin,rmax,nbins,nmu", [(1.0, 4.0, 4, 1), (1.0, 4.0, 2, 6), (0.05, 5.0, 30, 10),
                                                 (1e-4, 3.0, 7, 1)])
@pytest.mark.parametrize("kind,n", [("lattice", 1331), ("uniform", 2000), ("far", 2000),
                                    ("farther", 1500), ("uniform", 40)])
def test_logbins(kind, n, rmin, rmax, nbins, nmu, weighted, variant):
    xyz, rng = _points(kind, n)
    w = rng.lognormal(0.0, 0.3, n) if weighted else np.ones(n)
    w[n // 3:] *= -1.0
    buf = (rng.uniform(size=n) < 0.1).astype(np.int32)
    out = []
    cot = np.random.default_rng(1).normal(size=(2, nbins, nmu))
    with api.Context(0) as ctx:
        ctx.set_bins(rmin, rmax, nbins, nmu=nmu, logbins=True)
        ctx.set_autotune(variant)
        for mode in ("f32", "f64"):
            ctx.set_precision(mode)
            ctx.set_catalog(xyz, w, n // 3, buf)
            out.append(ctx.count_2pcf())
            out[-1]["grad"] = ctx.adjoint_2pcf(cot[0], cot[1])
            ctx.count_2pcf()
            if mode == "f32" and kind == "uniform" and rmin == 1.0 and n > 1000:
                # the FP32 form ran: a few pairs only went to FP64
                assert 0 <= ctx.stats()["fp64_rechecks"] < 0.02 * ctx.stats()["tuples"]
    for k in out[0]:
        np.testing.assert_array_equal(out[0][k], out[1][k])
    assert out[0]["counts"].sum() > 0
