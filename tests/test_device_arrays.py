"""Device arrays handed to the library by their addresses, without a GPU: a
library that records its calls and CPU tensors that claim to lie on a device.
Arrays with fewer entries than the call touches never reach it."""
import pytest
import torch

from gramsci_b200 import api


class DeviceTensor(torch.Tensor):
    """A CPU tensor that answers as one on the first CUDA device."""

    is_cuda = True
    device = torch.device("cuda", 0)

    def get_device(self):
        return 0


def on_device(t):
    return t.as_subclass(DeviceTensor)


class Library:
    def __init__(self, log=None):
        self.log = [] if log is None else log

    def __getattr__(self, name):
        def call(*args):
            self.log.append(name)
            return 0

        return call


def context(log=None):
    ctx = object.__new__(api.Context)
    ctx._lib, ctx._h = Library(log), None
    ctx.device, ctx.n, ctx.nbins, ctx.nmu, ctx._nsplit = 0, None, 3, 2, 0
    return ctx


def catalogue(n, nw=None, nbuf=None, columns=3):
    xyz = on_device(torch.zeros((n, columns), dtype=torch.float64))
    w = on_device(torch.ones(n if nw is None else nw, dtype=torch.float64))
    buf = None if nbuf is None else on_device(torch.zeros(nbuf, dtype=torch.int32))
    return xyz, w, 1, buf


@pytest.mark.parametrize("args", [(4, 3), (4, 0), (4, 4, 3), (4, 4, None, 2)],
                         ids=["w", "no-w", "buffer", "xyz"])
def test_short_inputs_are_refused(args):
    ctx = context()
    with pytest.raises(ValueError):
        ctx.set_catalog(*catalogue(*args))
    assert ctx._lib.log == []


@pytest.mark.parametrize("args", [(4,), (4, 6), (4, 4, 4), (0,)], ids=["plain", "long-w", "buffer", "empty"])
def test_inputs_that_fit_are_taken(monkeypatch, args):
    monkeypatch.setattr(api, "_torch_stream", lambda index: 0)
    ctx = context()
    ctx.set_catalog(*catalogue(*args))
    assert ctx.n == args[0] and ctx._lib.log[-1] == "gr_set_catalog_dev"


@pytest.mark.parametrize("order", [2, 3, 4])
@pytest.mark.parametrize("out", [
    torch.zeros(4, dtype=torch.float64), torch.zeros(6, dtype=torch.float64),
    torch.zeros(5, dtype=torch.float32), torch.zeros(10, dtype=torch.float64)[::2],
], ids=["short", "long", "float32", "strided"])
def test_gradient_that_does_not_fit_is_refused(order, out):
    ctx = context()
    ctx.n = 5
    fn = {2: ctx.adjoint_2pcf, 3: ctx.adjoint_3pcf, 4: ctx.adjoint_4pcf}[order]
    cot = torch.zeros({2: (3, 2), 3: (api.ncfg3(3), 2), 4: (api.ncfg4(3), 3, 3)}[order])
    with pytest.raises(ValueError):
        fn(cot, _out=on_device(out))
    with pytest.raises(ValueError):
        fn(cot, _out=torch.zeros(5, dtype=torch.float64))  # not on the device
    assert ctx._lib.log == []
    fn(cot, _out=on_device(torch.zeros(5, dtype=torch.float64)))
    assert len(ctx._lib.log) == 1


@pytest.mark.gpu
@pytest.mark.parametrize("order", [2, 3, 4])
@pytest.mark.parametrize("extra", [-3, 7])
def test_weights_of_another_length(order, extra):
    """No gradient for weights that are not one per point: too few are refused
    forward, too many backward, by torch."""
    from gramsci_b200 import autograd

    xyz = torch.rand((40, 3), dtype=torch.float64, device="cuda") * 12.0
    w = torch.ones(40 + extra, dtype=torch.float64, device="cuda", requires_grad=True)
    fn = {2: autograd.pcf2, 3: autograd.pcf3, 4: autograd.pcf4}[order]
    with pytest.raises(ValueError if extra < 0 else RuntimeError):
        fn(w, xyz, 20, 1.0, 4.0, 2)[0].sum().backward()
    assert w.grad is None
