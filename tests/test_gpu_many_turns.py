"""Rings that turn more than once in a step: index_shift and rotate_rings with
long steps.  A ring's offset is the sum of its shifts modulo the columns, and
dumps and sums that index by it see every column once.  Offsets are integers:
equal; the mass is a sum of 20x130 terms in another order: relative 1e-12."""
import ctypes as C

import numpy as np
import pytest

import penguin_2_0_b200 as pg
from penguin_2_0_b200 import _lib


@pytest.mark.gpu
def test_long_shifts(gpu):
    p = pg.params(0, imax=20, jmax=130)
    planet, fr = pg.init_planet(p)
    want, most = np.zeros(p.imax, np.int64), 0
    with pg.Run(p, 0) as run:
        run.load(pg.build_ic(p))
        for dt in (1.0, 7.0, 50.0, 1e3, 1.0):
            assert _lib.lib().pg_index_shift(run._h, C.c_double(dt), C.c_double(fr)) == 0
            pg.rotate_rings(run)
            buf = run.save()
            rj = np.frombuffer(bytes(buf), np.uint8).reshape(p.imax, -1)[:, 72 * p.jmax + 88:].copy().view(np.int32)
            want = (want + rj[:, 1]) % p.jmax
            most = max(most, np.max(np.abs(rj[:, 1])))
            assert np.array_equal(rj[:, 0], want)
            f = pg.dump_fields(buf, p)
            mass = np.sum(f["r"] * f["xvol"][:, None]) * (2 * np.pi / p.jmax)
            assert abs(pg.GPU_output_reduction(run, planet, 0.0, 0) - mass) <= 1e-12 * mass
    assert most > 100 * p.jmax
