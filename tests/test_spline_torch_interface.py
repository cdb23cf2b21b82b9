"""The check for plain tensors asks torch's private interface; a torch without
one of its functions must give the op-by-op recurrences, not an error."""
import pytest
import torch

from conftest import GOLDEN
from yspec_b200 import model_chain
from yspec_b200.model_chain import KnotModel


class _Without:
    """torch._C without one function."""

    def __init__(self, path):
        self.path = path

    def __getattr__(self, name):
        head, _, rest = self.path.partition(".")
        if name == head and not rest:
            raise AttributeError(name)
        inner = getattr(_REAL, name)
        return _Functorch(inner, rest) if name == head else inner


class _Functorch:
    def __init__(self, real, gone):
        self.real, self.gone = real, gone

    def __getattr__(self, name):
        if name == self.gone:
            raise AttributeError(name)
        return getattr(self.real, name)


_REAL = torch._C


@pytest.mark.parametrize("path", ["_len_torch_function_stack", "_len_torch_dispatch_stack", "_functorch",
                                  "_functorch.is_functorch_wrapped_tensor"])
def test_missing_function(monkeypatch, path):
    km = KnotModel(GOLDEN / "model200.deck")
    Y = torch.randn((km.nknot, 2), dtype=torch.float64, generator=torch.Generator().manual_seed(3))
    want = torch.cat([sp(Y[lo:hi + 1]) for sp, (lo, hi) in zip(km.spl, km.layers)])
    monkeypatch.setattr(torch, "_C", _Without(path))
    plain = model_chain._plain(Y)
    monkeypatch.undo()
    assert plain is False
    monkeypatch.setattr(model_chain, "_plain", lambda t: False)
    assert torch.equal(km._spline_rec(Y), want)
