"""After a catalogue is refused (a weight that is not finite) nothing of the
one before it is counted, exported or described any more, whatever the two
sizes, and the next catalogue is counted as on a new context."""
import ctypes

import numpy as np
import pytest

from gramsci_b200 import _native, api

pytestmark = pytest.mark.gpu


def _catalogue(n, seed):
    rng = np.random.default_rng(seed)
    return rng.uniform(0.0, 12.0, (n, 3)), rng.normal(size=n), n // 3


@pytest.mark.parametrize("n", [1, 200, 900])
def test_nothing_survives(n):
    with api.Context(0) as ctx:
        lib, h = ctx._lib, ctx._h
        ctx.set_bins(1.0, 3.0, 3, 1)
        ctx.set_catalog(*_catalogue(400, 1))
        ctx.set_regions(2)
        ctx.count_2pcf_batched()
        ctx.graph()
        xyz, w, n_data = _catalogue(n, 2)
        w[n // 2] = np.nan
        with pytest.raises(_native.GramsciError):
            ctx.set_catalog(xyz, w, n_data)
        edges, regions, members = ctypes.c_int64(-1), ctypes.c_int32(-1), ctypes.c_int64(-1)
        assert lib.gr_graph_nedges(h, ctypes.byref(edges)) == _native.GR_E_ARG
        assert lib.gr_graph_export(h, None, None, None, None) == _native.GR_E_ARG
        assert lib.gr_regions_info(h, ctypes.byref(regions), ctypes.byref(members)) == _native.GR_E_ARG
        assert lib.gr_regions_export(h, None, None, None) == _native.GR_E_ARG
        assert (edges.value, regions.value, members.value) == (-1, -1, -1)
        for call in (ctx.count_2pcf, ctx.count_3pcf, ctx.count_2pcf_batched, ctx.graph):
            with pytest.raises(_native.GramsciError):
                call()
        again = _catalogue(500, 3)
        ctx.set_catalog(*again)
        got, graph = ctx.count_3pcf(), ctx.graph()
        with api.Context(0) as fresh:
            fresh.set_bins(1.0, 3.0, 3, 1)
            fresh.set_catalog(*again)
            want, graph2 = fresh.count_3pcf(), fresh.graph()
        np.testing.assert_array_equal(got["counts"], want["counts"])
        for a, b in zip(graph, graph2):
            np.testing.assert_array_equal(a, b)
