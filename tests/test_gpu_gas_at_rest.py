"""Gas at rest next to moving gas, against the CPU oracle: a polar sweep first, then
the others.  The polar sweep's viscosity moves the lowest layers a little and leaves
the others' radial velocity at zero; flatten (flatten.cu:21) asks whether a shock's
velocities rise, and equal ones do not.  Strong density noise makes every other cell
a shock by its pressures.  Bound: relative 1e-12 per sweep; a change of the input's
last bit moves the oracle's results by at most 1e-13 here."""
import ctypes as C

import numpy as np
import pytest

import penguin_2_0_b200 as pg
from oracle.pyoracle import Oracle, lib as olib
from tests._lockstep import rel_linf


@pytest.mark.gpu
@pytest.mark.parametrize("case", [dict(imax=18, jmax=125, kmax=32, sc_h=0.07, noise_amp=0.6),
                                  dict(imax=117, jmax=122, kmax=9, ntop=3, sc_h=0.1, noise_amp=0.5)], ids=[0, 1])
def test_polar_sweep_first(gpu, case):
    p = pg.params(1, nprin=1, endtime=1e6, tmovie=1e6, **case)
    ic = pg.build_ic(p)
    planet, fr = pg.init_planet(p)
    body = planet.to_c()
    o = Oracle(p, ic)
    dt = 0.4 * o.get_dt(p.endtime, fr)
    with pg.Run(p, 0) as run:
        run.load(ic)
        for axis in (2, 0, 2, 0):
            (olib().orc_sweepx, olib().orc_sweepy, olib().orc_sweepz)[axis](o._h, dt, C.byref(body), fr)
            pg.sweep_axis(run, axis, dt, planet, fr)
            f, g = (pg.dump_fields(x.save(), p) for x in (o, run))
            speed = max(np.max(np.abs(f[k])) for k in "uvw")
            assert rel_linf(g["r"], f["r"]) <= 1e-12, axis
            assert max(np.max(np.abs(g[k] - f[k])) / speed for k in "uvw") <= 1e-12, axis
