"""The warp-per-chunk sweeps at the sizes where their layout changes, against
the CPU oracle.

A pencil's last chunk of lim = n % 116 + 12 cells takes ceil(lim / C) lanes,
and as many pencils as fit share a warp (C = 4 cells per lane, or 3 in the
polar sweep where that leaves fewer slots empty); tiles of 4 warps end in
columns or rings that do not exist.  The grids below have chunks of 13 cells
(eight pencils per warp), of one cell less and more than a whole number of
lanes, of exactly 32 lanes, the idle chunk of a multiple of 116, and column
counts with every remainder modulo a tile's width.  Bound: relative 1e-12 per
step, as for the other comparisons with the oracle."""
import numpy as np
import pytest

import penguin_2_0_b200 as pg
from tests._lockstep import OracleLoop, rel_linf

TOL = 1e-12

CASES = [
    dict(which=0, imax=117, jmax=122),            # radial 1 + 12 cells: 4 lanes; azimuthal 6 + 12: 5 lanes
    dict(which=0, imax=121, jmax=127),            # 5 + 12, 11 + 12
    dict(which=0, imax=168, jmax=168),            # 52 + 12 cells: 16 lanes, two pencils
    dict(which=0, imax=169, jmax=169),            # 53 + 12: 17 lanes, one pencil
    dict(which=0, imax=231, jmax=347),            # 115 + 12: the largest last chunk
    dict(which=0, imax=116, jmax=232),            # both last chunks idle
    dict(which=0, imax=30, jmax=123, EOS=1, gam=1.4),
    dict(which=0, imax=30, jmax=131, plnt_flag=0),
    dict(which=1, imax=20, jmax=122, kmax=6),     # polar 6 + 12 cells
    dict(which=1, imax=13, jmax=125, kmax=31),    # 31 + 12: 3 cells per lane, 15 lanes
    dict(which=1, imax=13, jmax=126, kmax=33),    # 33 + 12: 15 whole lanes
    dict(which=1, imax=13, jmax=127, kmax=34),    # 34 + 12: 16 lanes
    dict(which=1, imax=11, jmax=122, kmax=60),
    dict(which=1, imax=7, jmax=123, kmax=120),    # two polar chunks, the last of 4 + 12 cells
    dict(which=1, imax=117, jmax=122, kmax=9, ntop=3),
]


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(str(v) for v in c.values()))
def test_step_matches_oracle_at_layout_edges(gpu, case):
    c = dict(case)
    p = pg.params(c.pop("which"), nprin=1, **c)
    ic = pg.build_ic(p)
    ref = OracleLoop(p, ic)
    got = {}
    with pg.Run(p, 0) as run:
        run.load(ic)
        run.kernel_loop(2, record=lambda s, t, dt, pl, fr: got.__setitem__(s, (dt, pg.dump_fields(run.save(), p))))
    for s in range(2):
        dt, _, _ = ref.step()
        f, (gdt, g) = ref.fields(), got[s]
        np.testing.assert_array_equal(g["rot_j"], f["rot_j"])
        speed = max(np.max(np.abs(f[k])) for k in "uvw")
        e = [rel_linf(g["r"], f["r"])] + [np.max(np.abs(g[k] - f[k])) / speed for k in "uvw"]
        assert max(e) <= TOL, (case, s, e)
        assert abs(gdt - dt) <= TOL * dt
