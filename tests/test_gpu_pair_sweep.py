"""Reverse sweeps of single pairs (k_solve_adjoint.cu): the gradient of a model
one of whose core boundaries is not a double knot, which neither the solves nor
the sweeps take by groups of degrees.  The knot below the boundary is moved down
by one unit in the last place or by 1e-6 of its radius, which the model upload
accepts.  The reverse sweep's <dL/dm, d> must equal <g, d traces / dd> of the
tangent-linear solver on the same model; tolerance and its derivation as in
test_gpu_group_adjoint.py."""
import numpy as np
import pytest

from yspec_b200 import Engine, Event, Params, workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-11

CASES = [dict(grav=2), dict(grav=1, out=1), dict(grav=0, out=2, cor=1),
         dict(grav=2, model_file="model200_ocean.deck", depth_r=3.0, out=2, cor=1),
         dict(grav=2, model_file="model200_fic.deck", depth_r=3.0),
         dict(grav=2, lmin=1, lmax=1), dict(grav=0, lmin=0, lmax=0), dict(grav=1, lmin=2, depth_s=20.0, depth_r=300.0)]


@pytest.fixture(scope="module")
def engine():
    return Engine(0)


@pytest.mark.parametrize("boundary", ["inner core", "outer core"])
@pytest.mark.parametrize("i", range(len(CASES)))
def test_gradient_against_tangent(engine, workdir, i, boundary):
    import torch

    from yspec_b200.adjoint import tangent_traces
    from yspec_b200.model_chain import KnotModel

    kw = dict(ats=1, lmax=40, fmax=8.0, f21=6.0, f22=7.0, nrec=2)
    kw.update(CASES[i])
    if "model_file" in kw:
        kw["model_file"] = str(W.GOLDEN / kw["model_file"])
    p = W.config("c1", seed=5, **kw)[0]
    km = KnotModel(p.model_file)
    at = (km.view0.nic if boundary == "inner core" else km.view0.noc) - 1
    assert km.r[at] == km.r[at + 1]
    km.r = km.r.clone()
    km.r[at] = np.nextafter(float(km.r[at]), 0.0) if i % 2 == 0 else float(km.r[at]) * (1.0 - 1e-6)
    ev = Event(km.host, Params(p.write(workdir / f"ps_{i}.in")))
    engine.upload(km.array_model())
    engine.run(ev)
    assert engine.last_forms() == [-1] * 5                # the pair lists
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
