"""The ring sums against the reference's summation order restated in numpy.

Mass: per ring, 1024-cell blocks of the stored (rotated) order through a
halving tree, blocks added in turn; per polar stack a half-point tree over the
layers; rings through a 1024-wide tree.  Every addition has the same operands,
so the sums are equal bit for bit.  The torque's terms are formed differently
(to rounding), so it is held to 1e-12 of the sum of absolute terms.  Sizes:
ring lengths below, at and above one and two blocks, fewer rings than CTAs and
more, one and several layers."""
import numpy as np
import pytest

import penguin_2_0_b200 as pg

CASES = [dict(which=0, imax=3, jmax=122), dict(which=0, imax=40, jmax=1024), dict(which=0, imax=7, jmax=1025),
         dict(which=0, imax=601, jmax=130), dict(which=0, imax=1030, jmax=140), dict(which=0, imax=5, jmax=2100, precision=1),
         dict(which=1, imax=9, jmax=123, kmax=6), dict(which=1, imax=20, jmax=200, kmax=33)]


def _tree(v):
    v = np.concatenate([v, np.zeros(1024 - v.size)])
    h = 512
    while h:
        v = v[:h] + v[h:2 * h]
        h //= 2
    return v[0]


def _blocks(v):
    t = 0.0
    for b in range(0, v.size, 1024):
        t += _tree(v[b:b + 1024])
    return t


@pytest.mark.gpu
@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(str(v) for v in c.values()))
def test_ring_sums_follow_the_reference_order(gpu, case):
    c = dict(case)
    p = pg.params(c.pop("which"), **c)
    with pg.Run(p, 0) as run:
        run.load(pg.build_ic(p))
        run.kernel_loop(2)                       # rotated rings
        planet, _ = pg.init_planet(p)
        mass, torque = (pg.GPU_output_reduction(run, planet, 0.0, m) for m in (0, 9))
        f = pg.dump_fields(run.save(), p)
    nk, nr = p.kmax, p.imax
    col = np.frombuffer(bytes(pg.build_ic(p)), np.float64)[5 * p.jmax + 4:9 * p.jmax + 4].reshape(4, p.jmax)
    yvol, yc = col[2], col[3]
    store = (np.arange(p.jmax)[None, :] + f["rot_j"][:, None]) % p.jmax      # physical column of a storage slot
    zvol = f["zvol"][:, None] if p.ndim == 3 else 1.0
    v = f["r"] * f["xvol"][:, None] * yvol[store] * zvol
    part = np.array([_blocks(v[i]) for i in range(nk * nr)]).reshape(nk, nr)
    if p.ndim == 3:
        acc, n = list(part), 1
        while n < nk:
            n *= 2
        while n > 1:
            n //= 2
            for q in range(n):
                if q + n < nk:
                    acc[q] = acc[q] + acc[q + n]
        part = acc[0][None]
    assert mass == _blocks(part[0])
    if p.ndim == 3:
        assert torque == 0.0
        return
    x, phi = f["xc"][:, None], yc[store] - planet.y
    R3 = np.sqrt(x * x + planet.x ** 2 - 2 * planet.x * x * np.cos(phi) + planet.rs ** 2) ** 3
    g = planet.m * planet.x * np.sin(phi) / R3 - planet.m * np.sin(phi) / planet.x ** 2
    t = g * x * (f["r"] - x ** -p.p_alpha) * f["xvol"][:, None] * yvol[store]
    assert abs(torque - t.sum()) <= 1e-12 * np.abs(t).sum()
