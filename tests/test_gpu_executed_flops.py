"""Operations counted for a rate: by groups of degrees the l-independent part of
a coefficient matrix, 163 - 13 of the 666 flops of a self-gravitating
right-hand side, is formed once per item of 128 or 32 degrees.  The pair lists
form it for every pair."""
import pytest

from yspec_b200 import Engine, Event, Model, Params, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grav", [0, 1, 2])
def test_shared_points_count_once(workdir, grav):
    p = W.config("c1", seed=5, ats=1, grav=grav, lmin=1, lmax=60, fmax=6.0, f21=4.0, f22=5.0, nrec=1)[0]
    model = Model(p.model_file)
    ev = Event(model, Params(p.write(workdir / "x.in")))
    eng = Engine(0)
    eng.upload(model)
    eng.set_schedule(1)
    eng.coef(ev)
    lists = eng.work()[1]
    assert eng.executed_flops() == lists > 0.0
    eng.set_schedule(2)
    eng.coef(ev)
    assert eng.work()[1] == lists                         # the same steps
    # steps of six right-hand sides and 88 flops per component: the largest share the points can save
    # is 145 of 300 (b-vectors without self-gravitation 145 of 290), the smallest 43 of 88 less a 32nd
    low, high = (0.80, 0.86) if grav == 2 else (0.55, 0.75)
    assert low * lists < eng.executed_flops() < high * lists
