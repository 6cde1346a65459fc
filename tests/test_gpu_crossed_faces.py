"""A sweep over faces that cross in one step, against the CPU oracle.

A block of cells a million times thinner than the disk around it: the gas runs
into it faster than a cell per step, so Lagrangian widths turn negative there.
remap.cu picks a flux's donor by the way the face moved and then divides by the
donor's width, whatever its sign.  Bound: relative 1e-12 as for the other
comparisons with the oracle, whose own result moves by at most 8e-14 when the
input's last bits do."""
import ctypes as C

import numpy as np
import pytest

import penguin_2_0_b200 as pg
from oracle.pyoracle import Oracle, lib as olib
from tests._lockstep import rel_linf


@pytest.mark.gpu
@pytest.mark.parametrize("factor", [1e-5, 1e-6, 1e-8])
def test_radial_sweep_over_crossed_faces(gpu, factor):
    p = pg.params(0, nprin=1, imax=30, jmax=123)
    rec = np.frombuffer(bytes(pg.build_ic(p)), np.uint8).reshape(p.imax * p.kmax, -1).copy()
    f = rec[:, :40 * p.jmax].copy().view(np.float64).reshape(-1, 5, p.jmax)
    f[10:16, 0:2, 20:40] *= factor
    rec[:, :40 * p.jmax] = f.reshape(len(rec), -1).view(np.uint8)
    ic = bytearray(rec.tobytes())
    planet, fr = pg.init_planet(p)
    body = planet.to_c()
    o = Oracle(p, ic)
    dt = o.get_dt(p.endtime, fr)
    olib().orc_sweepx(o._h, dt, C.byref(body), fr)
    want = pg.dump_fields(o.save(), p)
    with pg.Run(p, 0) as run:
        run.load(ic)
        pg.sweep_axis(run, 0, dt, planet, fr)
        got = pg.dump_fields(run.save(), p)
    speed = max(np.max(np.abs(want[k])) for k in "uvw")
    assert rel_linf(got["r"], want["r"]) <= 1e-12
    assert max(np.max(np.abs(got[k] - want[k])) / speed for k in "uvw") <= 1e-12
