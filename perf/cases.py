"""The work a user has this framework do, as timed cases.

Every case goes through a public entry point: `Engine.run` (one event),
`Engine.prepare` / `execute` / `fetch` (one event with caller-owned pinned
output), `Engine.batch_run` (many events), `Engine.potential`,
`Engine.gradient`, `adjoint.ModelSynthetics` (an inversion step),
`adjoint.tangent_traces_many` (forward-mode derivatives) and
`ysg_traces_noalloc` (the time stage on device spectra, as a sharded run
calls it).  Shapes are those of `yspec_b200.workloads`, of the reference's
example input and of the tests; sources, moment tensors and receivers are
drawn from the seed.  Engines are kept per earth model and solver use, as a
program that runs many events keeps them.
"""
from __future__ import annotations

import ctypes as C
import math
import tempfile
from pathlib import Path

import numpy as np
import torch

from yspec_b200 import Engine, Event, Model, Params, adjoint, model_chain, native as N, workloads as W

GOLDEN = Path(W.GOLDEN)
DECKS = {
    "prem200": "model200.deck",              # 200 knots, solid inner core
    "prem400": "model400.deck",              # 400 knots
    "ocean": "model200_ocean.deck",          # with an ocean
    "fic": "model200_fic.deck",              # fluid inner core
    "example": "examples/prem.200",          # the reference's PREM: 220 knots, ocean, transversely isotropic
}

_BASE = dict(kind="event", deck="prem200", ats=1, grav=2, out=0, cor=0, lmin=0, lmax=150, fmin=0.1, fmax=10.0,
             tout=60.0, dt=10.0, depth=100.0, depth_r=0.0, nrec=10)


def _case(name=None, **kw):
    c = dict(_BASE)
    c.update(kw)
    if name is not None:
        c["name"] = name
    return c


def listed():
    return [
        # a quick look: long periods, a few stations, no gravity, velocity
        _case("quick_nograv", grav=0, ats=0, out=1, lmax=40, fmax=6.0, dt=20.0, nrec=3),
        # the small configuration: one event at long periods, displacement
        _case("small", ats=0),
        # a deep receiver below the source, Cowling approximation, a band of degrees
        _case("cowling_below", grav=1, lmin=3, lmax=297, fmax=20.0, dt=5.0, depth=20.0, depth_r=150.0, nrec=53),
        # the reference's example input: velocity on its PREM with an ocean
        _case("example", deck="example", out=1, cor=1, lmax=600, fmin=0.2, fmax=40.0, dt=1.0, depth=29.5, depth_r=3.0,
              nrec=60),
        # one event at scale: acceleration with the potential / tilt correction
        _case("scale", kind="phases", out=2, cor=1, lmax=750, fmax=50.0, tout=120.0, dt=1.0, depth=445.0, nrec=100),
        # one event of the largest configuration with a dense network
        _case("dense", kind="phases", deck="prem400", lmax=1500, fmax=100.0, tout=120.0, dt=0.5, depth=360.0,
              nrec=1500),
        # a catalogue of uneven events as one batch
        _case("catalogue", kind="batch", events=40, fmax=50.0, lmax=750),
        # potential perturbations on a deck with a fluid inner core
        _case("potential", kind="potential", deck="fic", out=1, lmax=120, fmax=12.0, dt=8.0, depth=300.0,
              depth_r=3.0, nrec=25),
        # the gradient of a misfit on an ocean deck at long periods
        _case("gradient_small", kind="gradient", deck="ocean", out=1, lmax=120, fmax=8.0, nrec=12, depth=60.0,
              depth_r=3.0),
        # one step of an inversion for the knot parameters and the moment tensor
        _case("inversion", kind="inversion", lmax=300, fmax=20.0, dt=5.0, depth=150.0, nrec=50),
        # forward-mode derivatives along several directions
        _case("tangents", kind="tangents", lmax=90, fmax=8.0, nrec=10, directions=6),
        # time series of device-resident spectra (the last stage of a sharded event)
        _case("time_series", kind="series", out=1, fmax=50.0, tout=120.0, dt=1.0, nrec=400),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["event", "event", "event", "phases", "batch", "potential", "gradient", "inversion", "tangents",
                       "series"])
    deck = rng.choice(["prem200", "prem200", "ocean", "fic", "example", "prem400"])
    top = {"event": 50.0, "phases": 60.0, "batch": 40.0, "potential": 30.0, "gradient": 14.0, "inversion": 14.0,
           "tangents": 7.0, "series": 60.0}[kind]
    fmax = round(_log(rng, 4.0, top), 2)
    lmax = max(12, int(fmax * rng.uniform(8.0, 15.0)))
    nrec = int(_log(rng, 1.0, {"series": 400, "gradient": 60, "inversion": 60, "tangents": 30}.get(kind, 600)))
    c = _case(kind=kind, deck=deck, fmax=fmax, lmax=lmax, nrec=max(1, nrec), lmin=rng.choice([0, 0, 0, 1, 2, 5]),
              dt=max(0.5, math.floor(1.0 / (2.2 * fmax * 1e-3) / 0.5) * 0.5), ats=rng.choice([0, 1, 1]),
              grav=rng.choice([0, 1, 2, 2, 2, 2]), out=rng.choice([0, 1, 2]), cor=rng.choice([0, 1]),
              tout=rng.choice([30.0, 60.0, 120.0]), depth=round(rng.uniform(1.0, 690.0), 1),
              depth_r=rng.choice([0.0, 0.0, 0.0, 50.0, 400.0]))
    if deck in ("ocean", "fic", "example"):
        # these decks end in 3 km of ocean: stations on its floor or deeper
        c["depth_r"] = max(3.0, c["depth_r"])
        c["depth"] = max(3.5, c["depth"])
    if kind in ("gradient", "inversion"):
        c["depth"] = round(rng.uniform(10.0, 400.0), 1)
    if kind == "batch":
        c["events"] = rng.randint(2, 24)
        c["nrec"] = min(c["nrec"], 100)
    if kind == "tangents":
        c["directions"] = rng.randint(1, 6)
    if kind == "potential":
        c["grav"] = 2
    return c


def _params(case, rng, fmax=None, lmax=None, nrec=None, depth=None, dt=None):
    """One event's parameter set; source, moment tensor and receivers from rng."""
    fmax = case["fmax"] if fmax is None else fmax
    (la, lo), = W.sphere_points(rng, 1)
    mm = W.moment_tensor(rng)
    return W.Params(model_file=str(GOLDEN / DECKS[case["deck"]]), ats=case["ats"], grav=case["grav"],
                    out=case["out"], cor=case["cor"], lmin=case["lmin"], lmax=case["lmax"] if lmax is None else lmax,
                    fmin=case["fmin"], fmax=fmax, tout=case["tout"], dt=case["dt"] if dt is None else dt,
                    f11=0.1, f12=0.2, f21=0.9 * fmax, f22=0.98 * fmax,
                    depth_s=case["depth"] if depth is None else depth, lat_s=la, lon_s=lo, mm=mm,
                    depth_r=case["depth_r"], receivers=W.sphere_points(rng, case["nrec"] if nrec is None else nrec))


def _event(model, p, tmp, i=0):
    return Event(model, Params(p.write(Path(tmp) / f"e{i}.in")))


_engines = {}


def _engine(deck, use="primal"):
    """(engine, model) of a deck, kept: a program keeps its engine for all its
    events.  The inversion and tangent uses upload other models, so each has
    its own."""
    key = (deck, use)
    if key not in _engines:
        model = Model(str(GOLDEN / DECKS[deck]))
        eng = Engine(0)
        eng.upload(model)
        _engines[key] = (eng, model)
    return _engines[key]


def _sizes(case, seed_rng):
    """(fmax, lmax, nrec, depth, dt) of the events of a batch."""
    out = []
    for _ in range(case["events"]):
        f = float(seed_rng.uniform(10.0 * case["fmax"] / 50.0, case["fmax"]))
        lmax = max(12, int(round(case["lmax"] * f / case["fmax"])))
        nr = max(1, int(round(math.exp(seed_rng.uniform(0.0, math.log(100.0 * max(case["nrec"], 1)))))))
        out.append((f, lmax, min(nr, 1000), float(seed_rng.uniform(0, 700)),
                    math.floor(1.0 / (2.2 * f * 1e-3) / 0.5) * 0.5))
    return out


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = {"kind": kind}
    with tempfile.TemporaryDirectory() as tmp:
        if kind == "series":
            _, model = _engine(case["deck"])
            ev = _event(model, _params(case, rng), tmp)
            g = torch.Generator(device="cuda").manual_seed(int(seed))
            # spectra fall off towards the band's ends, as responses do
            w = torch.hann_window(ev.nw + 2, periodic=False, dtype=torch.float64, device="cuda")[1:-1]
            s["spec"] = torch.randn((3, ev.nr, ev.nw, 2), dtype=torch.float64, device="cuda", generator=g) * \
                w[None, None, :, None]
            s["az"] = torch.from_numpy(np.ctypeslib.as_array(ev.raw.azep, (ev.nr,)).copy()).cuda()
            s["out"] = torch.zeros((ev.nr, 4, ev.nout()), dtype=torch.float64, device="cuda")
            s["ev"] = ev
            return s
        if kind == "batch":
            eng, model = _engine(case["deck"])
            # the catalogue's sizes are the case's, its sources and stations the seed's
            sizes = _sizes(case, np.random.default_rng(12345))
            s["evs"] = [_event(model, _params(case, rng, f, l, nr, d, dt), tmp, i)
                        for i, (f, l, nr, d, dt) in enumerate(sizes)]
            s["outs"] = [np.zeros((e.nr, 4, e.nout())) for e in s["evs"]]
            s["eng"] = eng
            return s
        use = kind if kind in ("inversion", "tangents", "gradient") else "primal"
        eng, model = _engine(case["deck"], use)
        ev = _event(model, _params(case, rng), tmp)
        s.update(eng=eng, ev=ev)
        if kind == "phases":
            s["out"] = torch.zeros((ev.nr, 4, ev.nout()), dtype=torch.float64, pin_memory=True)
        elif kind == "gradient":
            gout = rng.standard_normal((ev.nr, 4, ev.nout()))
            gout[:, 0, :] = 0.0
            s["gout"] = gout
        elif kind in ("inversion", "tangents"):
            s["km"] = km = model_chain.KnotModel(str(GOLDEN / DECKS[case["deck"]]))
            base = km.params()
            if kind == "inversion":
                # the current model of the inversion: a few per mille off the deck
                s["p"] = tuple(t * (1.0 + 2e-3 * torch.from_numpy(rng.standard_normal(t.shape[0]))) for t in base)
                s["mm"] = torch.tensor([float(x) for x in W.moment_tensor(rng)], dtype=torch.float64)
                s["syn"] = adjoint.ModelSynthetics(eng, ev, km)
                s["obs"] = torch.from_numpy(rng.standard_normal((ev.nr, 3, ev.nout())))
            else:
                s["dirs"] = [tuple(t * 1e-2 * torch.from_numpy(rng.standard_normal(t.shape[0])) for t in base)
                             for _ in range(case["directions"])]
    return s


def run(state):
    kind = state["kind"]
    if kind == "event":
        return state["eng"].run(state["ev"])
    if kind == "phases":
        eng = state["eng"]
        eng.prepare(state["ev"])
        eng.execute()
        eng.fetch(out_ptr=state["out"].data_ptr())
        return state["out"]
    if kind == "batch":
        return state["eng"].batch_run(state["evs"], outs=state["outs"])
    if kind == "potential":
        return state["eng"].potential(state["ev"])
    if kind == "gradient":
        return state["eng"].gradient(state["ev"], state["gout"])
    if kind == "inversion":
        rho, vp, vs = (t.clone().requires_grad_() for t in state["p"])
        mm = state["mm"].clone().requires_grad_()
        traces = state["syn"](rho, vp, vs, mm)
        loss = 0.5 * ((traces - state["obs"]) ** 2).sum()
        loss.backward()
        return traces.detach(), rho.grad, vp.grad, vs.grad, mm.grad
    if kind == "tangents":
        return adjoint.tangent_traces_many(state["eng"], state["ev"], state["km"], state["dirs"])
    ev, spec = state["ev"], state["spec"]
    n = C.c_int()
    N.check(N.lib().ysg_traces_noalloc(C.byref(ev.raw.tm), spec[0].data_ptr(), spec[1].data_ptr(), spec[2].data_ptr(),
                                       state["az"].data_ptr(), state["out"].data_ptr(), C.byref(n),
                                       C.c_void_p(torch.cuda.current_stream().cuda_stream)), "traces")
    return state["out"]


def _band(case, fmax, tout, dt):
    """(frequencies, transform length) of an event's frequency grid."""
    with tempfile.TemporaryDirectory() as tmp:
        _, model = _engine(case["deck"])
        p = _params(case, np.random.default_rng(0), fmax=fmax, nrec=1, dt=dt)
        p.tout = tout
        ev = _event(model, p, tmp)
        return ev.nw, ev.raw.tm.nt, ev.nout()


def _steps(case, fmax, lmax, nw, depth):
    """Cash-Karp steps of all (omega, l) pairs, (toroidal, fluid, solid chain,
    source-to-receiver), from a thinned (omega, l) grid: per knot interval
    1 + 4 omega h / alpha, from the depth where a wave of degree l has decayed
    by e^-11 below its turning point."""
    d = model_chain.read_deck(GOLDEN / DECKS[case["deck"]])
    r, vp, vs = d["r"], d["vpv"], d["vsv"]
    h = np.diff(r)
    a = np.maximum(vp[1:], vp[:-1])
    v = np.where(vs[:-1] > 0, vs[:-1], vp[:-1])
    rs = r[-1] - 1e3 * max(depth, case["depth_r"])
    nl = lmax - case["lmin"] + 1
    ls = np.unique(np.linspace(max(1, case["lmin"]), lmax, 33).astype(int))
    fs = np.linspace(case["fmin"], fmax, 17)[1:] * 1e-3
    rm = 0.5 * (r[1:] + r[:-1])
    tot = np.zeros(4)
    for f in fs:
        w = 2 * math.pi * f
        n = np.where(h > 0, 1.0 + np.floor(4 * w * h / a), 0.0)
        for l in ls:
            q = l * (l + 1.0) / np.maximum(rm, 1.0) ** 2 - (w / v) ** 2
            decay = np.sqrt(np.maximum(q, 0.0)) * h
            turn = int(np.argmax(q <= 0)) if (q <= 0).any() else len(h)
            i = min(turn, int(np.searchsorted(r, rs)) - 1)
            s = 0.0
            while i > 0 and s < 11.0:
                i -= 1
                s += decay[i]
            use = (np.arange(len(h)) >= i) & (h > 0)
            solid = vs[:-1] > 0
            top = rm > rs
            mant = solid & (rm > 3.5e6)
            tot += [(n * (use & mant)).sum(), (n * (use & ~solid)).sum(), (n * (use & solid)).sum(), (n * top).sum()]
    return tot / (len(fs) * len(ls)) * nl * nw


def _forward(case, fmax, lmax, nrec, depth, dt, solves=1):
    nw, nt, nout = _band(case, fmax, case["tout"], dt)
    tor, fluid, solid, top = _steps(case, fmax, lmax, nw, depth)
    # Cash-Karp steps: six right-hand sides and the stage combinations
    if case["grav"] == 2:
        rows = 3 if (case["out"] == 2 and case["cor"]) else 2
        fl = tor * 350 + fluid * 1200 + (solid + rows * top) * 4200
    else:
        fl = tor * 350 + fluid * 400 + solid * 1300 + 2 * top * 1000
    L = lmax - case["lmin"] + 1
    fl = fl * solves + 4.0 * nw * nrec * 22 * max(L, 1) + 3 * nrec * 5.0 * nt * math.log2(nt)
    return {"bytes": nrec * 24.0 + nout * 4 * nrec * 8.0, "flops": fl, "nw": nw, "nt": nt, "nout": nout}


def work(case):
    kind = case["kind"]
    if kind == "series":
        nw, nt, nout = _band(case, case["fmax"], case["tout"], case["dt"])
        return {"bytes": case["nrec"] * (3 * 16.0 * nw + 8 + 32.0 * nout),
                "flops": case["nrec"] * 3 * 5.0 * nt * math.log2(nt)}
    if kind == "batch":
        b = f = 0.0
        for fmax, l, nr, d, dt in _sizes(case, np.random.default_rng(12345)):
            x = _forward(case, fmax, l, nr, d, dt)
            b, f = b + x["bytes"], f + x["flops"]
        return {"bytes": b, "flops": f}
    x = _forward(case, case["fmax"], case["lmax"], case["nrec"], case["depth"], case["dt"])
    if kind == "tangents":
        # value and derivative of every operation (three products in place of one)
        return {"bytes": x["bytes"] * case["directions"], "flops": 3.0 * x["flops"] * case["directions"]}
    if kind == "gradient":
        # a forward sweep and its reverse (two products for each forward one)
        return {"bytes": x["bytes"], "flops": 3.0 * x["flops"]}
    if kind == "inversion":
        return {"bytes": 2.0 * x["bytes"], "flops": 4.0 * x["flops"]}
    return {"bytes": x["bytes"], "flops": x["flops"]}


def exact(case, seed):
    """The time stage has a plain 64-bit statement: the radix-2 network with
    the reference's single-precision pi (module_fourier.f90:7-145), the taper,
    e^{eps t}, the scales and the rotation.  The solves are a discrete
    Cash-Karp solution of hundreds of steps per (omega, l) pair: in numpy they
    take minutes, so those cases have none."""
    if case["kind"] != "series":
        return None
    s = prepare(case, seed)
    tm = s["ev"].raw.tm
    pi = float(np.float32(3.14159265358979323846))
    n, i1, i2 = tm.nt, tm.i1, tm.i2
    spec = torch.view_as_complex(s["spec"].cpu()).numpy()           # (3, nr, nw)
    w = np.arange(n // 2 + 1) * tm.df
    filt = np.select([w < tm.f11, w < tm.f12, w < tm.f21, w < tm.f22],
                     [0.0, 0.5 * (1 - np.cos(pi * (w - tm.f11) / (tm.f12 - tm.f11))), 1.0,
                      0.5 * (1 - np.cos(pi * (tm.f22 - w) / (tm.f22 - tm.f21)))], 0.0)
    p = n.bit_length() - 1
    idx = np.arange(n)
    rev = np.zeros(n, dtype=np.int64)
    for b in range(p):
        rev |= ((idx >> b) & 1) << (p - 1 - b)
    nr, nout = spec.shape[1], s["out"].shape[2]
    t = np.arange(nout) * tm.dt
    out = np.empty((nr, 4, nout))
    out[:, 0, :] = t * tm.t_norm
    for k0 in range(0, nr, 64):
        k1 = min(nr, k0 + 64)
        row = np.zeros((3, k1 - k0, n), dtype=np.complex128)
        row[:, :, i1 - 1:i2] = spec[:, k0:k1] * filt[i1 - 1:i2]
        row[:, :, n // 2 + 1:] = np.conj(row[:, :, 1:n // 2][:, :, ::-1])
        x = row[:, :, rev].reshape(3 * (k1 - k0), n)
        m = 1
        while m < n:
            tw = np.exp(1j * (np.arange(m) * (pi / m)))
            y = x.reshape(x.shape[0], n // (2 * m), 2, m)
            odd = y[:, :, 1] * tw
            x = np.stack([y[:, :, 0] + odd, y[:, :, 0] - odd], axis=2).reshape(x.shape[0], n)
            m *= 2
        v = x.real.reshape(3, k1 - k0, n)[:, :, :nout] / (tm.dt * n) * np.exp(tm.ep * t) * tm.amp_norm
        az = s["az"].cpu().numpy()[k0:k1, None]
        out[k0:k1, 1] = v[0]
        out[k0:k1, 2] = -v[1] * np.cos(az) + v[2] * np.sin(az)
        out[k0:k1, 3] = v[1] * np.sin(az) + v[2] * np.cos(az)
    return out
