"""Device memory a gradient call holds: the step logs of the resident lanes,
14 complex components and a factor per step for self-gravitating spheroidal
sweeps, 5 without, 2 for the toroidal ones.  The number of steps is bounded as
ysg_event_gradient bounds it; 0.3 GB are left for everything else (bases,
traces, orders, modules loaded on first use)."""
import math

import numpy as np
import pytest

from yspec_b200 import Engine, Event, Model, Params, workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grav", [0, 2])
def test_logs_follow_the_system(workdir, grav):
    import torch

    def event(model, name, **kw):
        p = W.config("c1", seed=5, ats=1, grav=grav, lmin=2, dt=10.0, nrec=1, depth_s=100.0, **kw)[0]
        model = model or Model(p.model_file)
        return model, Event(model, Params(p.write(workdir / f"{name}.in")))

    model, ev = event(None, "m", lmax=500, fmax=20.0, f21=15.0, f22=18.0, tout=120.0)
    e = ev.raw.ev
    eng = Engine(0)
    eng.upload(model)
    _, short = event(model, "s", lmax=10, fmax=4.0, f21=2.0, f22=3.0)
    eng.gradient(short, np.ones((short.nr, 4, short.nout())))
    eng.run(ev)                                           # events, coefficients, tables
    v = model.view()
    r, al = model.array("r"), model.array("alpha")
    w = e.wmin + (e.nw - 1) * e.dw
    steps = [0.0, 0.0, 0.0]
    for i in range(1, r.size):
        h = r[i] - r[i - 1]
        if h > 0.0:
            steps[0 if i < v.nic else 1 if i < v.noc else 2] += 2.0 + math.floor(h * 4.0 * w / max(al[i - 1], al[i]))
    lane = (max(steps) + sum(steps) + 4.0)                # logged steps per lane
    lanes = 256 * torch.cuda.get_device_properties(0).multi_processor_count     # resident, eight warps per SM
    bound = lanes * lane * (16 * (14 if grav == 2 else 5) + 8) + 2 * lanes * lane * (16 * 2 + 8) + 0.3e9
    g = np.random.default_rng(1).standard_normal((ev.nr, 4, ev.nout()))
    before = torch.cuda.mem_get_info(0)[0]
    eng.gradient(ev, g)
    held = before - torch.cuda.mem_get_info(0)[0]
    assert held <= bound, (held / 1e9, bound / 1e9)
