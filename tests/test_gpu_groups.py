"""Solves by groups of degrees (k_solve_group.cu) against the pair lists.

The group kernels share a frequency's radial walk between the lanes of a
block; the pair lists (schedule 1) run one walk per thread.  Both form the
same quantity by the same steps, so each coefficient row must agree within
1e-9 of its norm (the parity bar of the solve stage).  The cases sit where
the groups can go wrong: runs of degrees of one lane, one warp and one block
more or less, lists that do and do not fill the GPU (both forms of a
kernel), lanes that start in the inner core, the outer core and the mantle,
the receiver above, at and below the source, oceans and fluid inner cores,
every gravity setting, and frequency shards.
"""
import numpy as np
import pytest

from yspec_b200 import Engine, Event, Model, Params, workloads as W

pytestmark = pytest.mark.gpu

TOL = 1e-9


@pytest.fixture(scope="module")
def engine():
    return Engine(0)


def _coef(engine, pf, model, sched, shard=None):
    ev = Event(model, Params(pf))
    if shard:
        ev.raw.ev.jofs, ev.raw.ev.jstride = shard
        ev.raw.ev.nw = len(range(shard[0], ev.raw.ev.nw, shard[1]))
    engine.set_schedule(sched)
    try:
        c = engine.coef(ev)
        return c, engine.work()
    finally:
        engine.set_schedule(-1)


def _compare(engine, pf, model, shard=None):
    a, wa = _coef(engine, pf, model, 2, shard)
    b, wb = _coef(engine, pf, model, 1, shard)
    assert wa == wb                                   # pairs and counted steps
    for q in range(15):
        na, nb = a[:, q].ravel(), b[:, q].ravel()
        d = np.linalg.norm(na - nb)
        assert d <= TOL * np.linalg.norm(nb), (q, d, np.linalg.norm(nb))
        # pair by pair, against the row's largest value
        if np.abs(nb).max() > 0:
            assert np.abs(na - nb).max() <= 100 * TOL * np.abs(nb).max(), q


BANDS = [(0, 0), (1, 1), (2, 2), (0, 31), (1, 32), (1, 33), (2, 33), (3, 34), (5, 130), (1, 128), (1, 129), (97, 258)]


@pytest.mark.parametrize("lmin,lmax", BANDS)
def test_runs_of_degrees(engine, workdir, lmin, lmax):
    p = W.config("c1", seed=3, ats=1, lmin=lmin, lmax=lmax, fmax=8.0, f21=6.0, f22=7.0, nrec=1)[0]
    pf = p.write(workdir / f"g_{lmin}_{lmax}.in")
    model = Model(p.model_file)
    engine.upload(model)
    _compare(engine, pf, model)


DECKS = ["model200.deck", "model200_ocean.deck", "model200_fic.deck"]


@pytest.mark.parametrize("grav", [0, 1, 2])
@pytest.mark.parametrize("deck", DECKS)
@pytest.mark.parametrize("depths", [(100.0, 3.0), (20.0, 250.0), (150.0, 150.0), (2880.0, 3.0)])
def test_decks_and_depths(engine, workdir, deck, grav, depths):
    p = W.config("c1", seed=4, ats=1, grav=grav, out=2, cor=1, lmax=70, fmax=7.0, f21=5.0, f22=6.0, nrec=1,
                 model_file=str(W.GOLDEN / deck), depth_s=depths[0], depth_r=depths[1])[0]
    pf = p.write(workdir / f"d_{deck}_{grav}_{depths[0]}.in")
    model = Model(p.model_file)
    engine.upload(model)
    _compare(engine, pf, model)


@pytest.mark.parametrize("grav", [0, 1, 2])
def test_lists_that_fill_the_gpu(engine, workdir, grav):
    """More items than resident blocks: the wide form, longest first."""
    p = W.config("c1", seed=5, ats=1, grav=grav, lmax=300, fmax=30.0, tout=120.0, dt=10.0, f21=20.0, f22=25.0,
                 nrec=1, depth_s=300.0)[0]
    pf = p.write(workdir / f"w_{grav}.in")
    model = Model(p.model_file)
    engine.upload(model)
    _compare(engine, pf, model)


def test_frequency_shard(engine, workdir):
    p = W.config("c1", seed=6, lmax=60, fmax=8.0, f21=6.0, f22=7.0, nrec=1)[0]
    pf = p.write(workdir / "s.in")
    model = Model(p.model_file)
    engine.upload(model)
    _compare(engine, pf, model, shard=(1, 3))


def test_core_source_takes_the_pair_lists(engine, workdir):
    """Source in the outer core: schedule 2 runs the pair lists, as before."""
    p = W.config("c1", seed=7, lmax=20, fmax=5.0, f21=3.5, f22=4.5, dt=20.0, nrec=1, depth_s=3500.0)[0]
    pf = p.write(workdir / "core.in")
    model = Model(p.model_file)
    engine.upload(model)
    a, _ = _coef(engine, pf, model, 2)
    b, _ = _coef(engine, pf, model, 1)
    np.testing.assert_allclose(a, b, rtol=1e-12, atol=0, equal_nan=True)
