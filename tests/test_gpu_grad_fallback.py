"""Gradients into memory that the kernels do not write directly: device memory
off the alignment of a double (declined like memory that spans several
mappings or lies on another device), pinned and pageable host memory.  The
same numbers as the adjoint's own host array."""
import ctypes

import numpy as np
import pytest
import torch

from gramsci_b200 import _native, api

pytestmark = pytest.mark.gpu

N = 300


def _gradient(ctx, order, cots, pointer):
    lib = ctx._lib
    fn = {2: lib.gr_adjoint_2pcf, 3: lib.gr_adjoint_3pcf, 4: lib.gr_adjoint_4pcf}[order]
    arrays = [np.ascontiguousarray(c.T.ravel()) for c in cots]
    args = [ctypes.c_void_p(a.ctypes.data) for a in arrays] + [None] * (2 if order == 4 else 0)
    _native.check(lib, ctx._h, fn(ctx._h, *args, ctypes.c_void_p(pointer)))


@pytest.mark.parametrize("order", [2, 3, 4])
def test_declined_memory(order):
    rng = np.random.default_rng(order)
    xyz, w = rng.uniform(0.0, 9.0, (N, 3)), rng.normal(size=N)
    with api.Context(0) as ctx:
        ctx.set_catalog(xyz, w, 100)
        ctx.set_bins(1.0, 3.5, 2, 1)
        out = {2: ctx.count_2pcf, 3: ctx.count_3pcf, 4: ctx.count_4pcf}[order]()
        cots = [rng.normal(size=out[k].shape) for k in ("N2", "N3")]
        fn = {2: ctx.adjoint_2pcf, 3: ctx.adjoint_3pcf, 4: ctx.adjoint_4pcf}[order]
        want = fn(*cots)
        assert np.abs(want).max() > 0.0
        for off, where in ((0, "cuda"), (4, "cuda"), (8, "cuda"), (0, "pinned"), (0, "host")):
            if where == "cuda":
                room = torch.full((8 * N + 32,), 7, dtype=torch.uint8, device="cuda")
                torch.cuda.synchronize()
            else:
                room = torch.full((8 * N + 32,), 7, dtype=torch.uint8, pin_memory=where == "pinned")
            _gradient(ctx, order, cots, room.data_ptr() + off)
            raw = room.cpu().numpy()
            got = np.frombuffer(raw[off:off + 8 * N].tobytes())
            np.testing.assert_array_equal(got, want)
            assert (raw[:off] == 7).all() and (raw[off + 8 * N:] == 7).all()
