"""Gradients written to device memory by the library against the same
gradients read back to the host: identical arrays, through the C entry and
through torch.autograd, for weights of either precision and on either side,
and with work still pending on torch's stream."""
import numpy as np
import pytest
import torch

from gramsci_b200 import api, autograd

pytestmark = pytest.mark.gpu

BINS = {2: (1.0, 6.0, 5, 4), 3: (1.0, 4.0, 3, 2), 4: (1.0, 3.5, 2, 1)}


def _points(n):
    rng = np.random.default_rng(n)
    w = rng.lognormal(0.0, 0.3, n)
    w[n // 3:] *= -1.0
    return rng.uniform(0.0, 12.0, (n, 3)), w, n // 3


@pytest.mark.parametrize("order", [2, 3, 4])
@pytest.mark.parametrize("n", [1, 31, 700])
def test_gradient_in_place(order, n):
    xyz, w, n_data = _points(n)
    with api.Context(0) as ctx:
        ctx.set_catalog(xyz, w, n_data)
        ctx.set_bins(*BINS[order])
        out = {2: ctx.count_2pcf, 3: ctx.count_3pcf, 4: ctx.count_4pcf}[order]()
        rng = np.random.default_rng(3)
        cot = [rng.normal(size=out[k].shape) for k in ("N2", "N3")]
        fn = {2: ctx.adjoint_2pcf, 3: ctx.adjoint_3pcf, 4: ctx.adjoint_4pcf}[order]
        host = fn(*cot)
        # a view that starts in the middle of an allocation, guarded by its ends
        room = torch.full((n + 2,), -7.0, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        fn(*cot, _out=room[1:n + 1])
        got = room.cpu().numpy()
    np.testing.assert_array_equal(got[1:-1], host)
    assert got[0] == -7.0 and got[-1] == -7.0


@pytest.mark.parametrize("order", [2, 3, 4])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_autograd_devices_agree(order, dtype):
    xyz, w, n_data = _points(500)
    fn = {2: autograd.pcf2, 3: autograd.pcf3, 4: autograd.pcf4}[order]
    bins = BINS[order] if order < 4 else BINS[4][:3]
    grads = []
    for dev in ("cpu", "cuda"):
        for _ in range(3):
            x = torch.tensor(xyz, device=dev)
            v = torch.tensor(w, dtype=dtype, device=dev, requires_grad=True)
            N2, N3 = fn(v, x, n_data, *bins)[:2]
            ((N2 * N2).sum() + N3.sum()).backward()
            assert v.grad.dtype == dtype and v.grad.device.type == dev
            # freed and reused while later work is queued
            torch.empty(500, dtype=torch.float64, device="cuda").normal_()
            grads.append(v.grad.cpu().numpy())
    for g in grads[1:]:
        np.testing.assert_array_equal(g, grads[0])
