"""Calls that need device memory when little or none is free, while the block that
dumps pass through lies idle: it is given back and the call succeeds."""
import ctypes as C
from contextlib import contextmanager

import pytest

import penguin_2_0_b200 as pg


def _p(nr, nphi, **kw):
    return pg.params(0, imax=nr, jmax=nphi, endtime=1e6, tmovie=1e6, **kw)


@contextmanager
def _memory_taken(leave):
    """All but `leave` bytes of the device's memory taken (0: to the last 512)."""
    import torch
    cu = C.CDLL("libcuda.so.1")
    got = []

    def take(n):
        d = C.c_uint64(0)
        if cu.cuMemAlloc_v2(C.byref(d), C.c_size_t(n)):
            return False
        got.append(d)
        return True

    try:
        if leave:
            assert take(torch.cuda.mem_get_info(0)[0] - leave)
        else:
            for n in (1 << 32, 1 << 28, 1 << 24, 1 << 21, 1 << 16, 1 << 12, 512):
                while take(n):
                    pass
        yield
    finally:
        for d in got:
            cu.cuMemFree_v2(d)


@pytest.fixture
def idle_block(gpu):
    """A run whose save left a block of 475 MB."""
    p = _p(1500, 4400)
    with pg.Run(p, 0) as r:
        r.load(pg.build_ic(p))
        r.save()
        yield r


@pytest.mark.gpu
def test_a_dump_larger_than_what_is_free(idle_block):
    p = _p(1700, 4700)                       # 575 MB: more than the block may grow to
    with pg.Run(p, 0) as r:
        r.load(pg.build_ic(p))
        want = r.save()
        idle_block.save()
        with _memory_taken(200 << 20):
            assert r.save() == want
            r.load(want)
        assert r.save() == want


@pytest.mark.gpu
@pytest.mark.parametrize("what", ["batch", "graph", "harmonic", "load", "create"])
def test_calls_with_no_memory_free(idle_block, what):
    p = _p(64, 130)
    ic = pg.build_ic(p)

    def call(r, b):
        if what == "batch":
            b.add(r)
            b.advance(4, chunk=2)
            b.sync()
            b.remove(r)
        elif what == "graph":
            r.advance(5, graph_chunk=2)
        elif what == "harmonic":
            r.harmonic(2.0)
            r.post_torque(1e-3)
        elif what == "load":
            r.load(ic)
            r.clock_reset(0)
            r.advance(2)
        else:
            pg.Run(p, 0).close()

    out = []
    for full in (False, True):               # the first loads every kernel
        with pg.Run(p, 0) as r, pg.Batch(0) as b:
            r.load(ic)
            r.clock_reset(0)
            r.advance(1)
            idle_block.save()
            if full:
                with _memory_taken(0):
                    call(r, b)
            else:
                call(r, b)
            out.append(bytes(r.save()))
    assert out[0] == out[1]
