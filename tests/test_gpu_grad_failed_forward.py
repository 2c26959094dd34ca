"""A forward call that fails after its catalogue went to the shared context
(bins that the library refuses, weights that are not finite) leaves the
gradients of earlier calls as they are."""
import pytest
import torch

from gramsci_b200 import autograd

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [2, 3, 4])
@pytest.mark.parametrize("failure", ["bins", "weights"])
@pytest.mark.parametrize("device", ["cpu", "cuda"])
def test_earlier_gradient(order, failure, device):
    gen = torch.Generator().manual_seed(order)
    fn = {2: autograd.pcf2, 3: autograd.pcf3, 4: autograd.pcf4}[order]

    def inputs():
        xyz = torch.rand((150, 3), generator=gen, dtype=torch.float64) * 9.0
        w = torch.rand(150, generator=gen, dtype=torch.float64) + 0.5
        return xyz.to(device), w.to(device).requires_grad_(True)

    (xyz, w), (other, w2) = inputs(), inputs()
    out = fn(w, xyz, 60, 1.0, 3.5, 2)
    want, = torch.autograd.grad(sum((o * o).sum() for o in out), w)
    assert want.abs().max() > 0
    out = fn(w, xyz, 60, 1.0, 3.5, 2)
    with pytest.raises(Exception):
        if failure == "bins":
            fn(w2, other, 60, 1.0, 3.5, 0)
        else:
            fn(w2 * float("nan"), other, 60, 1.0, 3.5, 2)
    got, = torch.autograd.grad(sum((o * o).sum() for o in out), w)
    assert torch.equal(got, want)
