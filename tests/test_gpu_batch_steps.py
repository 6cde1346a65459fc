"""The steps that a run reports after a batch has stepped it.

pg_advance returns the difference of two step counts; the one before comes from
the host where the run itself made the last step.  Members of a batch are stepped
by replayed graphs that the run does not see, whatever is asked of it between."""
import pytest

import penguin_2_0_b200 as pg

CASES = [
    dict(which=0, imax=72, jmax=150),
    dict(which=0, imax=72, jmax=150, precision=1),
    dict(which=0, imax=72, jmax=150, EOS=1, gam=1.4),
    dict(which=0, imax=72, jmax=150, plnt_flag=2),
    dict(which=1, imax=20, jmax=130, kmax=8),
]


@pytest.mark.gpu
@pytest.mark.parametrize("ask", ["history", "clock"])
def test_advance_after_a_batch_counts_its_own_steps(gpu, ask):
    runs = []
    for c in CASES:
        c = dict(c)
        p = pg.params(c.pop("which"), nprin=4, endtime=1e6, tmovie=1e6, **c)
        r = pg.Run(p, 0).load(pg.build_ic(p))
        r.clock_reset(0)
        assert r.advance(2) == 2
        runs.append(r)
    with pg.Batch(0) as b:
        for r in runs:
            b.add(r)
        for _ in range(3):                     # captured, then replayed
            b.advance(8, chunk=4)
            if ask == "history":               # it clears the rows it returns
                b.sync()
            for r in runs:
                getattr(r, ask)()
        b.advance(8, chunk=4)
        b.tune(1)
        st = b.status()
        for r in runs:
            b.remove(r)
    for r, s in zip(runs, st):
        assert r.advance(3) == 3
        assert r.advance(6, graph_chunk=2) == 6
        assert r.clock()[0].ncycle == s["ncycle"] + 9
        r.close()
