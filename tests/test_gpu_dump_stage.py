"""Dumps in and out of a run: the device block they pass through is shared by
a device's runs (pg_run.cu, DumpStage), and a captured graph outlives a load."""
import threading

import numpy as np
import pytest

import penguin_2_0_b200 as pg

pytestmark = pytest.mark.gpu


def _p(nr, nphi, **kw):
    return pg.params(0, imax=nr, jmax=nphi, endtime=1e6, tmovie=1e6, **kw)


def _fields(buf, p):
    rb = 72 * p.jmax + 96
    a = np.frombuffer(bytes(buf), np.uint8).reshape(p.imax, rb)
    return a[:, : 32 * p.jmax].copy().view(np.float64)


# small, larger (the block grows), smaller again, above what is kept (512 MiB)
@pytest.mark.parametrize("sizes", [[(64, 130), (200, 600), (64, 130)], [(1700, 4700), (64, 130)]])
def test_a_dump_comes_back_as_it_went_in(sizes):
    for nr, nphi in sizes:
        p = _p(nr, nphi)
        ic = pg.build_ic(p)
        r = pg.Run(p, 0).load(ic)
        assert np.array_equal(_fields(r.save(), p), _fields(ic, p))
        r.close()


def test_threads_with_runs_of_their_own():
    errs = []

    def work(k):
        try:
            p = _p(96 + 8 * k, 260 + k * 16, seed=k)
            ic = pg.build_ic(p)
            want = _fields(ic, p)
            for _ in range(4):
                r = pg.Run(p, 0)
                for _ in range(4):
                    r.load(ic)
                    if not np.array_equal(_fields(r.save(), p), want):
                        errs.append(k)
                r.close()
        except Exception as e:   # noqa: BLE001
            errs.append(repr(e))

    ts = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join(120)
    assert not errs


@pytest.mark.parametrize("world", [0, 1])
def test_a_graph_serves_the_next_dump_too(world):
    kw = dict(imax=72, jmax=150, endtime=1e6, tmovie=1e6)
    if world:
        kw["kmax"] = 12
    p, q = pg.params(world, seed=3, **kw), pg.params(world, seed=4, **kw)
    r = pg.Run(p, 0).load(pg.build_ic(p))
    r.clock_reset(0)
    r.advance(9, graph_chunk=4)
    r.load(pg.build_ic(q))
    r.clock_reset(0)
    r.advance(9, graph_chunk=4)
    f = pg.Run(p, 0).load(pg.build_ic(q))
    f.clock_reset(0)
    f.advance(9, graph_chunk=4)
    assert bytes(r.save()) == bytes(f.save())
    r.close()
    f.close()
