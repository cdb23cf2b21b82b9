"""Reverse sweeps by groups of degrees (k_group_adjoint.cu) at their edges.

For a random trace adjoint g and a random model direction d the reverse
sweep's <dL/dm, d> must equal <g, d traces / dd> of the tangent-linear solver
(one walk per thread).  Both differentiate the same discrete solve, so they
differ by rounding alone: a relative error of some 1e-13 per term of the
inner product (a few thousand operations of 1e-16), so 1e-11 of the sum of
the terms' magnitudes bounds it.  The cases: runs of degrees of one lane, one
warp and one block more or less, l = 0 and toroidal limits, every gravity
setting, starts in the inner core, the outer core and the mantle.
"""
import numpy as np
import pytest

from yspec_b200 import Engine, Event, Params, workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-11

BANDS = [(0, 0), (1, 1), (2, 2), (0, 31), (1, 32), (2, 34), (1, 128), (1, 129), (97, 258)]
CASES = [dict(lmin=a, lmax=b, grav=2 - i % 3) for i, (a, b) in enumerate(BANDS)]
CASES += [dict(lmin=0, lmax=40, grav=g, model_file=d, depth_r=3.0, out=2, cor=1)
          for g in (0, 1, 2) for d in ("model200_ocean.deck", "model200_fic.deck")]
CASES += [dict(lmin=0, lmax=20, grav=2, fmax=20.0, f21=18.0, f22=19.0),
          dict(lmin=0, lmax=20, grav=0, depth_s=20.0, depth_r=300.0)]


@pytest.fixture(scope="module")
def engine():
    return Engine(0)


@pytest.mark.parametrize("i", range(len(CASES)))
def test_gradient_against_tangent(engine, workdir, i):
    import torch

    from yspec_b200.adjoint import tangent_traces
    from yspec_b200.model_chain import KnotModel

    kw = dict(ats=1, fmax=8.0, f21=6.0, f22=7.0, nrec=2)
    kw.update(CASES[i])
    if "model_file" in kw:
        kw["model_file"] = str(W.GOLDEN / kw["model_file"])
    p = W.config("c1", seed=5, **kw)[0]
    km = KnotModel(p.model_file)
    ev = Event(km.host, Params(p.write(workdir / f"ga_{i}.in")))
    engine.upload(km.array_model())
    rng = np.random.default_rng(11)
    g = rng.standard_normal((ev.nr, 4, ev.nout()))
    g[:, 0, :] = 0.0
    gval, gcs = engine.gradient(ev, g)
    d = tuple(torch.from_numpy(rng.standard_normal(km.nknot)) * x * 1e-2 for x in km.params())
    dm = km.tangent(d)
    terms = np.concatenate([np.concatenate([gval[q] * dm.val[q], gcs[q] * dm.cs[q]]) for q in range(13)])
    rhs = float(np.sum(g[:, 1:4, :] * tangent_traces(engine, ev, km, d)))
    assert np.abs(terms).sum() > 0.0
    assert abs(terms.sum() - rhs) <= TOL * np.abs(terms).sum(), (CASES[i], terms.sum(), rhs, np.abs(terms).sum())
