"""Kept indices: the 2PCF and its adjoint reuse the index of a 3PCF (or of a
graph) of the same catalogue and bins and leave it to the next one, with the
numbers of a new context; another catalogue, other bins or another precision
end that."""
import numpy as np
import pytest

from gramsci_b200 import api

pytestmark = pytest.mark.gpu


def _catalogue(n, box, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(0.0, box, (n, 3)), rng.normal(size=n), n // 3


def _results(ctx):
    two, three = ctx.count_2pcf(), ctx.count_3pcf()
    cot = np.linspace(-1.0, 1.0, two["N2"].size).reshape(two["N2"].shape)
    return [two["counts"], two["catsum"], three["counts"], three["catsum"], ctx.adjoint_2pcf(cot)]


@pytest.mark.parametrize("n,box", [(2000, 40.0), (3000, 12.0), (40000, 100.0)])
@pytest.mark.parametrize("graph", [False, True])
def test_reuse(n, box, graph):
    a, b = _catalogue(n, box, 1), _catalogue(n, box, 2)
    bins, bins2 = (1.0, 4.0, 3, 2), (0.5, 3.0, 4, 1)
    with api.Context(0) as ctx:
        ctx.set_keep_graph(True)
        for cat, bn, prec in ((a, bins, "f32"), (b, bins, "f32"), (b, bins2, "f32"), (b, bins2, "f64"),
                              (a, bins2, "f64")):
            ctx.set_catalog(*cat)
            ctx.set_bins(*bn)
            ctx.set_precision(prec)
            if graph:
                ctx.graph()
            else:
                ctx.count_3pcf()
            ctx.count_2pcf()
            first = ctx.stats()["kernel_launches"]
            ctx.count_3pcf()
            ctx.adjoint_2pcf(np.ones((bn[2], bn[3])))
            second = ctx.stats()["kernel_launches"]
            assert (first, second) == (3, 2)  # clearing, sweep, results; sweep, gradient
            got = _results(ctx)
            with api.Context(0) as fresh:
                fresh.set_catalog(*cat)
                fresh.set_bins(*bn)
                fresh.set_precision(prec)
                want = _results(fresh)
            for g, w in zip(got, want):
                if g.dtype.kind == "i":
                    np.testing.assert_array_equal(g, w)
                else:
                    assert np.abs(g - w).max() <= 1e-12 * np.abs(w).max()
