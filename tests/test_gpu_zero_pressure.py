"""Dumps that hold no pressure in some cells.

A load looks at the density only, so the first radial sweep meets whatever
pressure a dump holds: its sound speed is the square root of that, and the
Riemann problem's bound on p takes over.  Two steps against the CPU oracle at the
bound of the other comparisons, relative 1e-12; a change of the input's last bit
moves the oracle's own results by at most 3e-14 here.  1e-310 is a number below
the normal ones."""
import struct

import numpy as np
import pytest

import penguin_2_0_b200 as pg
from tests._lockstep import OracleLoop, rel_linf

TOL = 1e-12
CASES = [
    (dict(which=0, imax=30, jmax=123), 0.0),
    (dict(which=0, imax=30, jmax=123), 1e-310),
    (dict(which=0, imax=130, jmax=131, EOS=1, gam=1.4), 0.0),
    (dict(which=1, imax=13, jmax=125, kmax=8), 0.0),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case,value", CASES, ids=range(len(CASES)))
def test_cells_without_pressure_step(gpu, case, value):
    c = dict(case)
    p = pg.params(c.pop("which"), nprin=1, **c)
    ic = bytearray(pg.build_ic(p))
    for ring, j in ((4, 7), (12, 60), (12, 61)):
        struct.pack_into("<d", ic, ring * (72 * p.jmax + 96) + 8 * (p.jmax + j), value)
    ref = OracleLoop(p, ic)
    got = []
    with pg.Run(p, 0) as run:
        run.load(ic)
        run.kernel_loop(2, record=lambda s, t, dt, pl, fr: got.append((dt, pg.dump_fields(run.save(), p))))
        run.load(ic)
        run.clock_reset(0)
        assert run.advance(2) == 2
    for gdt, g in got:
        dt, _, _ = ref.step()
        f = ref.fields()
        np.testing.assert_array_equal(g["rot_j"], f["rot_j"])
        speed = max(np.max(np.abs(f[k])) for k in "uvw")
        assert rel_linf(g["r"], f["r"]) <= TOL
        assert max(np.max(np.abs(g[k] - f[k])) / speed for k in "uvw") <= TOL
        assert abs(gdt - dt) <= TOL * dt
