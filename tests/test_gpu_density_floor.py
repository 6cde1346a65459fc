"""Cells whose Lagrangian density falls to the bound 1e-15, against the CPU oracle.

evolve.cu sets such a cell's density to the bound, and remap.cu takes its mass
from that density and the moved volume.  It happens where both faces of a nearly
empty cell cross in one step (density noise of 90 %) and where the disk itself is
thinner than the bound (ten scale heights above the midplane).  Bound: relative
1e-12 per step, as for the other comparisons with the oracle; a change of the
input in its last bit moves the oracle's own results by at most 4e-14 here."""
import ctypes as C
import math

import numpy as np
import pytest

import penguin_2_0_b200 as pg
from oracle.pyoracle import Oracle, lib as olib
from tests._lockstep import OracleLoop, rel_linf

TOL = 1e-12

STEPS = [
    dict(which=0, imax=60, jmax=160, noise_amp=0.9),
    dict(which=0, imax=60, jmax=160, noise_amp=0.9, flat_flag=0),
    dict(which=1, imax=16, jmax=123, kmax=24, zmin=math.pi / 2 - 0.5),
]
SWEEPS = [
    (0, dict(which=0, imax=130, jmax=131, noise_amp=0.9)),
    (0, dict(which=0, imax=60, jmax=160, noise_amp=0.9, EOS=1, gam=1.4)),
    (2, dict(which=1, imax=20, jmax=130, kmax=16, noise_amp=0.9)),
]


def _params(case):
    c = dict(case)
    return pg.params(c.pop("which"), nprin=1, **c)


def _errors(g, f):
    speed = max(np.max(np.abs(f[k])) for k in "uvw")
    return [rel_linf(g["r"], f["r"])] + [np.max(np.abs(g[k] - f[k])) / speed for k in "uvw"]


@pytest.mark.gpu
@pytest.mark.parametrize("case", STEPS, ids=lambda c: "x".join(str(v) for v in c.values()))
def test_steps_with_cells_at_the_bound(gpu, case):
    p = _params(case)
    ic = pg.build_ic(p)
    ref = OracleLoop(p, ic)
    got = []
    with pg.Run(p, 0) as run:
        run.load(ic)
        run.kernel_loop(3, record=lambda s, t, dt, pl, fr: got.append((dt, pg.dump_fields(run.save(), p))))
    for s, (gdt, g) in enumerate(got):
        dt, _, _ = ref.step()
        f = ref.fields()
        np.testing.assert_array_equal(g["rot_j"], f["rot_j"])
        assert max(_errors(g, f)) <= TOL, (s, _errors(g, f))
        assert abs(gdt - dt) <= TOL * dt


@pytest.mark.gpu
@pytest.mark.parametrize("axis,case", SWEEPS, ids=lambda c: str(c) if isinstance(c, int) else "x".join(str(v) for v in c.values()))
def test_sweep_with_cells_at_the_bound(gpu, axis, case):
    p = _params(case)
    ic = pg.build_ic(p)
    planet, fr = pg.init_planet(p)
    body = planet.to_c()
    o = Oracle(p, ic)
    dt = o.get_dt(p.endtime, fr)
    (olib().orc_sweepx, olib().orc_sweepy, olib().orc_sweepz)[axis](o._h, dt, C.byref(body), fr)
    f = pg.dump_fields(o.save(), p)
    with pg.Run(p, 0) as run:
        run.load(ic)
        pg.sweep_axis(run, axis, dt, planet, fr)
        g = pg.dump_fields(run.save(), p)
    assert max(_errors(g, f)) <= TOL, _errors(g, f)
