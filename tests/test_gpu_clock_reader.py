"""A thread that looks at a run's clock while another steps the run.

Each look is a copy in stream order, so the clock of one moment: its step count
and its time belong together."""
import threading

import pytest

import penguin_2_0_b200 as pg

STEPS = 500


def _run():
    p = pg.params(0, imax=24, jmax=122, endtime=1e6, tmovie=1e6)
    r = pg.Run(p, 0).load(pg.build_ic(p))
    r.clock_reset(0)
    return r


@pytest.mark.gpu
def test_clock_read_from_another_thread(gpu):
    want = {}
    with _run() as r:
        for _ in range(STEPS):
            r.advance(1)
            c, _ = r.clock()
            want[c.ncycle] = c.simtime
    last = max(want)
    r = _run()
    seen, errors, stop = [], [], threading.Event()

    def look():
        try:
            while not stop.is_set():
                c, _ = r.clock()
                if 0 < c.ncycle <= last:
                    seen.append((c.ncycle, c.simtime))
        except Exception as e:   # noqa: BLE001
            errors.append(repr(e))

    ts = [threading.Thread(target=look, daemon=True) for _ in range(2)]
    for t in ts:
        t.start()
    for _ in range(STEPS):
        r.advance(1)
    stop.set()
    for t in ts:
        t.join(60)
    assert not any(t.is_alive() for t in ts)
    assert not errors
    bad = [s for s in seen if want[s[0]] != s[1]]
    assert seen and not bad, (len(bad), len(seen), bad[:3])
    r.close()
