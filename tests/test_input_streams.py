"""Catalogues that torch's stream is still computing when they are handed to
the library, which reads them on its own stream: its work is ordered after
them, the conversions that the call queues itself included."""
import numpy as np
import pytest
import torch

from gramsci_b200 import api

from test_device_arrays import catalogue, context


def test_the_library_waits_first(monkeypatch):
    asked = []
    monkeypatch.setattr(api, "_torch_stream", lambda index: asked.append(index) or 7)
    ctx = context()
    ctx.set_catalog(*catalogue(4, 4, 4))
    assert asked == [0] and ctx._lib.log == ["gr_wait_stream", "gr_set_catalog_dev"]


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("side", [False, True])
def test_inputs_still_being_computed(dtype, side):
    """Positions and weights that are the last of a queue of work, on torch's
    default stream or another one."""
    rng = np.random.default_rng(1)
    n = 200000
    xyz0 = rng.integers(0, 4096, (n, 3)) / 32.0  # exact in both types
    w0 = rng.integers(1, 64, n) / 64.0
    with api.Context(0) as ctx:
        ctx.set_bins(1.0, 4.0, 3, 1)
        ctx.set_catalog(xyz0, w0, n // 2)
        want = ctx.count_2pcf()
        stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
        a = torch.ones((4096, 4096), device="cuda")
        src = torch.tensor(xyz0, dtype=dtype, device="cuda"), torch.tensor(w0, dtype=dtype, device="cuda")
        torch.cuda.synchronize()
        for _ in range(3):
            with torch.cuda.stream(stream):
                xyz, w = torch.full_like(src[0], -1.0), torch.full_like(src[1], -1.0)
                for _ in range(20):
                    a = a @ a * (1.0 / 4096)
                xyz += (src[0] + 1.0) * a[0, 0]
                w += (src[1] + 1.0) * a[0, 0]
                ctx.set_catalog(xyz, w, n // 2)
                got = ctx.count_2pcf()
            np.testing.assert_array_equal(got["counts"], want["counts"])
            np.testing.assert_array_equal(got["catsum"], want["catsum"])
