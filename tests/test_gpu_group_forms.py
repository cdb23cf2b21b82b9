"""Both forms of the group kernels (k_solve_group.cu), and which of them ran:
the rule picks one per kind from the sizes of the lists, so every case states
the forms it is there for.

The wide forms, longest items first, against the pair lists, and events of a
batch that differ in the moment tensor alone, whose coefficients one wide solve
writes, against the events by themselves.  All of them take the same steps, so
they differ by rounding: some 2,000 steps of six stages, ten roundings of
1.1e-16 each, are 1.3e-11 if they all add up.  1e-11 of a row's or a trace's norm
is asked for; digits lost in a coefficient of every step would show."""
import numpy as np
import pytest

from yspec_b200 import Engine, Event, Model, Params, workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-11
WIDE, NARROW, NONE = 0, 1, -1


@pytest.fixture(scope="module")
def engine():
    return Engine(0)


def _case(workdir, name, **kw):
    a = dict(seed=5, ats=1, nrec=1, tout=120.0, dt=10.0)
    a.update(kw)
    p = W.config("c1", **a)[0]
    return Model(p.model_file), p.write(workdir / f"{name}.in")


LARGE = dict(lmax=500, fmax=45.0, f21=30.0, f22=40.0, depth_s=300.0)
SMALL = dict(lmax=70, fmax=4.0, f21=2.5, f22=3.5, dt=20.0)


@pytest.mark.parametrize("grav", [0, 1, 2])
@pytest.mark.parametrize("form,size", [(WIDE, LARGE), (NARROW, SMALL)])
def test_against_pair_lists(engine, workdir, grav, form, size):
    model, pf = _case(workdir, f"w{grav}{form}", grav=grav, **size)
    engine.upload(model)
    out = {}
    for sched in (2, 1):
        engine.set_schedule(sched)
        out[sched] = engine.coef(Event(model, Params(pf)))
        forms = engine.last_forms()
        if sched == 2:
            assert forms[grav] == form and forms[3] == form, forms
            assert [forms[k] for k in range(3) if k != grav] == [NONE, NONE]
        else:
            assert forms == [NONE] * 5
    engine.set_schedule(-1)
    for q in range(15):
        a, b = out[2][:, q].ravel(), out[1][:, q].ravel()
        assert np.linalg.norm(a - b) <= TOL * np.linalg.norm(b), q


@pytest.mark.parametrize("grav", [0, 1, 2])
def test_shared_wide_solves(engine, workdir, grav):
    model, pf = _case(workdir, f"s{grav}", grav=grav, out=2, cor=1, **LARGE)
    engine.upload(model)
    rng = np.random.default_rng(grav)
    evs = [Event(model, Params(pf)) for _ in range(3)]
    for e in evs[1:]:
        for q in range(6):
            e.raw.ev.mm[q] = float(rng.standard_normal() * 1e-3)
    outs = engine.batch_run(evs)
    forms = engine.last_forms()
    assert forms[grav] == WIDE and forms[3] == WIDE, forms
    for e, o in zip(evs, outs):
        want = engine.run(e)
        for k in range(e.nr):
            for c in (1, 2, 3):
                d = np.linalg.norm(o[k, c] - want[k, c])
                assert d <= TOL * np.linalg.norm(want[k, c]), (k, c, d)
