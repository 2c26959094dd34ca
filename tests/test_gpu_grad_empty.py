"""Differentiable counts of a catalogue without points, on either side: sums of
zero and an empty gradient (an empty CUDA tensor has no address)."""
import pytest
import torch

from gramsci_b200 import autograd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [2, 3, 4])
@pytest.mark.parametrize("device", ["cpu", "cuda"])
def test_empty(order, device):
    xyz = torch.zeros((0, 3), dtype=torch.float64, device=device)
    w = torch.zeros(0, dtype=torch.float64, device=device, requires_grad=True)
    out = {2: autograd.pcf2, 3: autograd.pcf3, 4: autograd.pcf4}[order](w, xyz, 0, 1.0, 4.0, 2)
    assert not any(o.any() for o in out)
    sum(o.sum() for o in out).backward()
    assert w.grad.shape == (0,) and w.grad.device.type == device
