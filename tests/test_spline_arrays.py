"""The library's spline of many arrays at once (ysh_spline_arrays) against the
op-by-op recurrences it stands in for, and the callers that must keep the
latter: the same numbers for real arrays, rounding (a few units in the last
place of the largest value per recurrence step) for complex ones, and vmap,
forward mode and tracing through the chain."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import GOLDEN
from yspec_b200 import native as N
from yspec_b200.model_chain import KnotModel, _plain

DECKS = ["model200.deck", "model200_fic.deck", "model200_ocean.deck", "model400.deck"]


def _recurrences(km, Y):
    return torch.cat([sp(Y[lo:hi + 1]) for sp, (lo, hi) in zip(km.spl, km.layers)])


@pytest.mark.parametrize("deck", DECKS)
@pytest.mark.parametrize("m", [1, 2, 25])
def test_equals_recurrences(deck, m):
    km = KnotModel(GOLDEN / deck)
    g = torch.Generator().manual_seed(m)
    Y = torch.randn((km.nknot, m), dtype=torch.float64, generator=g)
    assert _plain(Y)
    assert torch.equal(km._spline_rec(Y), _recurrences(km, Y))
    assert torch.equal(km._spline_rec(Y.T.contiguous().T), _recurrences(km, Y))        # other strides
    Z = torch.complex(Y, torch.randn((km.nknot, m), dtype=torch.float64, generator=g))
    a, b = km._spline_rec(Z), _recurrences(km, Z)
    assert (a - b).abs().max() <= 1e-13 * b.abs().max()
    # a lazily conjugated view keeps the recurrences
    assert torch.equal(km._spline_rec(Z.conj()), _recurrences(km, Z.conj()))


def test_transforms_keep_the_operations():
    km = KnotModel(GOLDEN / "model200.deck")
    p = km.params()
    d = torch.ones_like(p[0])
    _, jv = torch.func.jvp(lambda r: km.arrays(r, p[1], p[2])["grav_cs"], (p[0],), (d,))
    want = torch.from_numpy(km.tangent((d, 0 * d, 0 * d)).cs[10])
    assert (jv - want).abs().max() <= 1e-12 * want.abs().max()
    s = torch.tensor([1.0, 1.25], dtype=torch.float64)
    v = torch.func.vmap(lambda q: km.arrays(p[0] * q, p[1], p[2])["rho_cs"])(s)
    one = km.arrays(p[0] * s[1], p[1], p[2])["rho_cs"]
    assert (v[1] - one).abs().max() <= 1e-13 * one.abs().max()
    z = (p[0] + 0j).requires_grad_()
    assert km.arrays(z, p[1] + 0j, p[2] + 0j)["rho_cs"].requires_grad


def test_arguments():
    f = N.lib().ysh_spline_arrays
    x = np.array([0.0, 1.0, 1.0, 2.0, 4.0])
    y = np.array([1.0, 2.0, 2.0, 5.0, 3.0])
    out = np.full(5, np.nan)
    assert f(5, N.dptr(x), 1, N.dptr(y), N.dptr(out)) == 0
    assert np.all(out[:2] == 0.0) and out[2] == out[4] == 0.0     # a layer of two knots, one of three
    assert out[3] == 6.0 * ((3.0 - 5.0) / 2.0 - (5.0 - 2.0) / 1.0) / (2.0 * (2.0 + 1.0))
    one = np.full(1, np.nan)
    assert f(1, N.dptr(x[:1].copy()), 1, N.dptr(y[:1].copy()), N.dptr(one)) == 0 and one[0] == 0.0
    assert f(5, N.dptr(x), 0, None, None) == 0
    assert f(0, N.dptr(x), 1, N.dptr(y), N.dptr(out)) == 1
    assert f(5, None, 1, N.dptr(y), N.dptr(out)) == 1
    assert f(5, N.dptr(x), -1, N.dptr(y), N.dptr(out)) == 1
