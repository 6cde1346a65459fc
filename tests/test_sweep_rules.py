"""Rules by which the sweeps take a short form (pg_warp.cuh), compared with the
general one over the range that each rule accepts: the series of sincos_near and
riemann_near against numpy in long double, and flatten's look at the high words."""
import numpy as np
import pytest

LD = np.longdouble
EPS = 2.0 ** -53


def _horner(z, c):
    q = LD(c[0])
    for k in c[1:]:
        q = q * z + LD(k)
    return q


def test_small_angles():
    x = np.linspace(0.0, 0.05, 4001).astype(LD)[1:]
    z = x * x
    s = x + x * z * _horner(z, [1 / LD(362880), -1 / LD(5040), 1 / LD(120), -1 / LD(6)])
    c = 1 + z * _horner(z, [1 / LD(40320), -1 / LD(720), 1 / LD(24), -1 / LD(2)])
    assert np.max(np.abs(s / np.sin(x) - 1)) < EPS / 8
    assert np.max(np.abs(c - np.cos(x))) < EPS / 8


def test_riemann_series():
    z = np.linspace(-0.125, 0.125, 4001).astype(LD)
    z = z[z != 0]
    q = _horner(z * z, [1 / LD(k) for k in (17, 15, 13, 11, 9, 7, 5, 3)])
    log = 2 * (z + z ** 3 * q)                     # of (1 + z) / (1 - z)
    assert np.max(np.abs(log / (np.log1p(z) - np.log1p(-z)) - 1)) < EPS / 8
    t = np.linspace(-0.125, 0.125, 4001).astype(LD)
    f, k = LD(1), []
    for n in range(1, 11):
        f = f * n
        k.append(1 / f)
    e = _horner(t, k[::-1] + [LD(1)])
    assert np.max(np.abs(e / np.exp(t) - 1)) < EPS / 8


def _hi(x):
    return (x.view(np.int64) >> 32).astype(np.int64)


@pytest.mark.parametrize("seed", range(4))
def test_no_shock_without_a_difference_of_high_words(seed):
    """Cells that flatten treats as shocked, |p+ - p-| > 0.33 min, never fall
    below the bound on the high words that lets a warp skip the rest."""
    r = np.random.default_rng(seed)
    a = np.concatenate([2.0 ** r.uniform(-60, 60, 200000), np.ldexp(np.nextafter(1.0, [0, 2]), 3), [1e-15, 1.0, 2.0]])
    for k in (1.33, 1.3300000001, np.nextafter(1.33, 2), 1.5, 2.0, 10.0):
        b = a * k
        shock = np.abs(b - a) > 0.33 * np.minimum(a, b)
        far = np.abs(_hi(a) - _hi(b)) > 335544
        assert not np.any(shock & ~far)
    b = a * (1.33 + r.uniform(0.0, 1e-6, a.size))
    shock = np.abs(b - a) > 0.33 * np.minimum(a, b)
    assert not np.any(shock & ~(np.abs(_hi(a) - _hi(b)) > 335544))


def _quot16(a, d):
    return (a * (65536 // d + 1)) >> 16


def test_quotients_by_multiplication():
    a = np.arange(0, 128, dtype=np.int64)
    for d in range(1, 129):
        assert np.array_equal(_quot16(a, d), a // d)
    r = np.random.default_rng(0)
    for d in [1, 2, 3, 7, 116, 255, 1021, 4096, 99991]:
        m = (1 << 40) // d + 1
        a = np.unique(np.concatenate([r.integers(0, min(1 << 23, (1 << 40) // d), 20000), np.arange(0, 5) * d,
                                      np.arange(1, 5) * d - 1]))
        q = np.array([(int(x) * m) >> 40 for x in a])
        q = np.where(q * d > a, q - 1, q)
        assert np.array_equal(q, a // d)
