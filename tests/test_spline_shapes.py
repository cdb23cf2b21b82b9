"""Arrays the library's spline does not take keep the op-by-op recurrences:
it reads nknot rows of the array's columns, so an array with other rows or
dimensions must not reach it."""
import pytest
import torch

from conftest import GOLDEN
from yspec_b200.model_chain import KnotModel


def _recurrences(km, Y):
    return torch.cat([sp(Y[lo:hi + 1]) for sp, (lo, hi) in zip(km.spl, km.layers)])


@pytest.mark.parametrize("tail", [(), (1,), (2, 3), (1, 4, 2)])
def test_dimensions(tail):
    km = KnotModel(GOLDEN / "model200.deck")
    Y = torch.randn((km.nknot,) + tail, dtype=torch.float64, generator=torch.Generator().manual_seed(1))
    assert torch.equal(km._spline_rec(Y), _recurrences(km, Y))


def test_rows():
    km = KnotModel(GOLDEN / "model200.deck")
    Y = torch.randn((km.nknot + 5, 2), dtype=torch.float64, generator=torch.Generator().manual_seed(2))
    assert torch.equal(km._spline_rec(Y), _recurrences(km, Y))          # the rows beyond the knots are left out
    with pytest.raises((IndexError, RuntimeError)):
        km._spline_rec(Y[: km.nknot - 3])
