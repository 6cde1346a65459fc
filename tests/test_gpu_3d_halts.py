"""3D runs that stop in the middle of a call.

A 3D step swaps the run's two plane copies; steps that are queued behind a halt (end
time, a tmovie dump) do nothing.  However many are, the state is that of the steps
taken: the same bits as a run advanced one step per call, through single steps,
graphs and batches, and what is asked of the run after it goes on from there."""
import pytest

import penguin_2_0_b200 as pg

GRID = dict(imax=20, jmax=130, kmax=8, nprin=1)
CALLS = [(4, 0), (7, 0), (8, 0), (8, 2), (9, 4), (20, 4)]


def _setup(steps, stop):
    p = pg.params(1, endtime=1e6, tmovie=1e6, **GRID)
    ic = pg.build_ic(p)
    with pg.Run(p, 0) as r:
        r.load(ic)
        dt = pg.get_dt(p.endtime, r, pg.init_planet(p)[1])
    p.update(**{stop: (steps - 0.5) * dt})
    return p, ic


def _alone(p, ic, steps, more=0):
    with pg.Run(p, 0) as r:
        r.load(ic)
        r.clock_reset(0)
        for _ in range(steps + more):
            assert r.advance(1) == 1
        return bytes(r.save()), r.history().tolist()


@pytest.mark.gpu
@pytest.mark.parametrize("stop", ["endtime", "tmovie"])
@pytest.mark.parametrize("steps", [2, 3])
def test_state_where_a_call_stopped(gpu, steps, stop):
    p, ic = _setup(steps, stop)
    want = _alone(p, ic, steps)
    for n, chunk in CALLS:
        with pg.Run(p, 0) as r:
            r.load(ic)
            r.clock_reset(0)
            assert r.advance(n, graph_chunk=chunk) == steps
            assert (bytes(r.save()), r.history().tolist()) == want, (n, chunk)


@pytest.mark.gpu
def test_steps_after_a_stop(gpu):
    p, ic = _setup(3, "tmovie")
    want, _ = _alone(p, ic, 3, more=2)
    for n, chunk in CALLS:
        with pg.Run(p, 0) as r:
            r.load(ic)
            r.clock_reset(0)
            assert r.advance(n, graph_chunk=chunk) == 3
            assert r.advance(2, graph_chunk=chunk) == 2
            assert bytes(r.save()) == want, (n, chunk)


@pytest.mark.gpu
@pytest.mark.parametrize("steps", [2, 3])
@pytest.mark.parametrize("end", ["remove", "sync", "status", "close"])
def test_members_of_a_batch(gpu, steps, end):
    p, ic = _setup(steps, "endtime")
    want, _ = _alone(p, ic, steps)
    runs = [pg.Run(p, 0).load(ic), pg.Run(pg.params(1, endtime=1e6, tmovie=1e6, **GRID), 0).load(ic)]
    b = pg.Batch(0)
    for r in runs:
        r.clock_reset(0)
        b.add(r)
    b.advance(7, chunk=2)
    if end == "remove":
        for r in runs:
            b.remove(r)
    else:
        getattr(b, end)()
    assert bytes(runs[0].save()) == want
    assert runs[1].clock()[0].ncycle == 7
    b.close()
    for r in runs:
        r.close()


@pytest.mark.gpu
def test_a_member_destroyed_in_its_batch(gpu):
    p, ic = _setup(3, "endtime")
    q = pg.params(0, imax=40, jmax=130, endtime=1e6, tmovie=1e6)
    gone, stays = pg.Run(p, 0).load(ic), pg.Run(q, 0).load(pg.build_ic(q))
    with pg.Batch(0) as b:
        for r in (gone, stays):
            r.clock_reset(0)
            b.add(r)
        b.advance(4, chunk=2)
        gone.close()
        b.advance(4, chunk=2)
        b.sync()
        assert [s["ncycle"] for s in b.status()][:1] == [8]
        b.remove(stays)
    assert stays.advance(1) == 1
    stays.close()
