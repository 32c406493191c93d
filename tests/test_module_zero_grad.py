"""``BoxConv2d.zero_grad``: what ``torch.nn.Module.zero_grad`` does, for plain parameters, further ones, frozen and missing ones, and the
cases that it leaves to that method."""
import pytest
import torch

import box_convolution as bc


class Renamed(bc.BoxConv2d):
    def named_parameters(self, *args, **kwargs):
        return iter([("x_min", self.x_min)])


def _module(cls=bc.BoxConv2d):
    m = cls(2, 3, 8, 8)
    m.register_parameter("gain", torch.nn.Parameter(torch.ones(2)))
    m.register_parameter("missing", None)
    for p in m._parameters.values():
        if p is not None:
            p.grad = torch.ones_like(p)
    m.gain.requires_grad_(False)
    return m


@pytest.mark.parametrize("cls", [bc.BoxConv2d, Renamed])
@pytest.mark.parametrize("args", [(), (True,), (False,)])
def test_as_the_base_class(cls, args):
    m, want = _module(cls), _module(cls)
    m.zero_grad(*args)
    torch.nn.Module.zero_grad(want, *args)
    for (n, p), q in zip(m._parameters.items(), want._parameters.values()):
        if p is not None:
            assert (p.grad is None) == (q.grad is None), n
            assert p.grad is None or torch.equal(p.grad, q.grad), n


@pytest.mark.parametrize("name,value", [("parameters", lambda m: iter([m.x_min])), ("named_parameters", lambda m: iter([("x_min", m.x_min)]))])
def test_methods_set_on_the_object(name, value):
    m, want = _module(), _module()
    for each in (m, want):
        setattr(each, name, lambda *args, each=each, **kwargs: value(each))
    m.zero_grad()
    torch.nn.Module.zero_grad(want)
    assert want.x_min.grad is None and want.x_max.grad is not None
    assert m.x_min.grad is None and m.x_max.grad is not None


def test_submodules_and_parametrizations():
    m = _module()
    m.inner = torch.nn.Linear(2, 2)
    m.inner.weight.grad = torch.ones(2, 2)
    m.zero_grad()
    assert m.inner.weight.grad is None and m.x_min.grad is None
    m = _module()
    torch.nn.utils.parametrize.register_parametrization(m, "x_min", torch.nn.Identity())
    original = m.parametrizations.x_min.original
    original.grad = torch.ones_like(original)
    m.zero_grad()
    assert original.grad is None and m.x_max.grad is None
