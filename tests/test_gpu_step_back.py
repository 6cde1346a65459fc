"""A run that starts after its end time takes one step back to it (main.cu:355 clips
the step to endtime - simtime, whatever its sign).  The device's loop damps by that
step as the host's does: relative 1e-12 (a step of 2D and 3D disks with damping
zones on both sides)."""
import numpy as np
import pytest

import penguin_2_0_b200 as pg
from tests._lockstep import rel_linf


@pytest.mark.gpu
@pytest.mark.parametrize("case", [dict(which=0, imax=64, jmax=150), dict(which=0, imax=64, jmax=232, EOS=1, gam=1.4),
                                  dict(which=0, imax=64, jmax=150, precision=1), dict(which=1, imax=20, jmax=130, kmax=8)],
                         ids=range(4))
def test_last_step_of_a_run_past_its_end(gpu, case):
    c = dict(case)
    p = pg.params(c.pop("which"), nprin=1, kill_rin=0.7, kill_rout=1.5, endtime=0.16, tmovie=0.18, **c)
    ic = pg.build_ic(p)
    with pg.Run(p, 0) as run:
        run.load(ic)
        run.clock_reset(1)
        assert run.advance(4) == 1
        got = pg.dump_fields(run.save(), p)
        clock, _ = run.clock()
        assert abs(clock.simtime - 0.16) < 1e-12 and clock.dt_used < 0.0
        run.load(ic)
        run.kernel_loop(1, startat=1)
        want = pg.dump_fields(run.save(), p)
    tol = 4e-7 if p.precision else 1e-12
    speed = max(np.max(np.abs(want[k])) for k in "uvw")
    assert rel_linf(got["r"], want["r"]) <= tol
    assert max(np.max(np.abs(got[k] - want[k])) / speed for k in "uvw") <= tol
