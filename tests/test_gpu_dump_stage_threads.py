"""Loads and saves of several threads' runs at the same time: each thread ends, has
done all its rounds and got its own dump back.  The dumps differ in size, so one
thread at a time has the kept block and the others memory of their own."""
import threading

import numpy as np
import pytest

import penguin_2_0_b200 as pg

THREADS, ROUNDS = 4, 6


def _fields(buf, p):
    rec = np.frombuffer(bytes(buf), np.uint8).reshape(p.imax, -1)
    return rec[:, :32 * p.jmax].copy()


@pytest.mark.gpu
def test_every_thread_ends_with_its_own_dump(gpu):
    done, errors = [0] * THREADS, []

    def work(k):
        try:
            p = pg.params(0, imax=90 + 31 * k, jmax=250 + 40 * k, seed=k, endtime=1e6, tmovie=1e6)
            ic = pg.build_ic(p)
            want = _fields(ic, p)
            for _ in range(ROUNDS):
                with pg.Run(p, 0) as r:
                    r.load(ic)
                    assert np.array_equal(_fields(r.save(), p), want)
                done[k] += 1
        except Exception as e:   # noqa: BLE001
            errors.append(repr(e))

    ts = [threading.Thread(target=work, args=(k,), daemon=True) for k in range(THREADS)]
    for t in ts:
        t.start()
    for t in ts:
        t.join(60)
    assert not any(t.is_alive() for t in ts)
    assert not errors
    assert done == [ROUNDS] * THREADS
