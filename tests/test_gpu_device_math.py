"""The short forms of pg_warp.cuh as the GPU computes them, against 80-bit floating
point (or integers) over the ranges that the sweeps give them, and at their edges.

The header is compiled into a small library here, with the flags of the sweeps.
Bounds in units of u = 2^-53, from the forms themselves:
  rcp          the last fma rounds (1 u); the step leaves e^3 <= 2^-60
  rsq          the same, and x y rounds inside e, half of which arrives
  root         rsq and one more product
  quot         the last fma rounds; what it adds is off by 2^-50 of itself
  sin, cos, sinc of a small angle: the last fma rounds, the polynomial's own
               roundings arrive times x^2/6 <= 4e-4; beyond 0.05 CUDA's sincos (2 u)
  riemann_near p*: the roundings of t times 1/8, of two fma's and of the product;
               u*: those of z times w/16, and of the sum of the velocities
"""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from penguin_2_0_b200 import build as B

LD = np.longdouble
U = LD(2.0) ** -53

SOURCE = r"""
#include "pg_warp.cuh"
using namespace pgd;
__global__ void k(int what, int n, const double *a, const double *b, const double *c, const double *d, const double *e,
                  double *o, double *p, double *q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (what == 0) o[i] = rcp(a[i]);
  if (what == 1) o[i] = rsq(a[i]);
  if (what == 2) o[i] = root(a[i]);
  if (what == 3) o[i] = quot(a[i], b[i], 1.0 / b[i]);
  if (what == 4) {
    sincos_near(a[i], o[i], p[i]);
    q[i] = sinc_near(a[i], true);
  }
  if (what == 5) q[i] = riemann_near(a[i], b[i], 1.0, c[i], d[i], e[i], o[i], p[i]);
  if (what == 6) o[i] = quot16((int)a[i], 65536 / (int)b[i] + 1);
  if (what == 8) o[i] = above_bound(a[i]);
  if (what == 7) o[i] = quot40((int)a[i], (int)b[i], (1ull << 40) / (unsigned long long)b[i] + 1);
}
extern "C" int run(int what, int n, const double *const *in, double *const *out) {
  double *d[8] = {};
  int bad = 0;
  for (int i = 0; i < 8; i++) bad |= cudaMalloc(&d[i], n * sizeof(double)) != cudaSuccess;
  for (int i = 0; i < 5; i++) bad |= cudaMemcpy(d[i], in[i], n * sizeof(double), cudaMemcpyHostToDevice) != cudaSuccess;
  if (!bad) k<<<(n + 127) / 128, 128>>>(what, n, d[0], d[1], d[2], d[3], d[4], d[5], d[6], d[7]);
  for (int i = 0; i < 3; i++) bad |= cudaMemcpy(out[i], d[5 + i], n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess;
  for (int i = 0; i < 8; i++) cudaFree(d[i]);
  return bad;
}
"""


@pytest.fixture(scope="module")
def device(gpu, tmp_path_factory):
    d = tmp_path_factory.mktemp("math")
    src, so = d / "m.cu", d / "m.so"
    src.write_text(SOURCE)
    flags = B.SOURCE_FLAGS["pg_sweep.cu"]
    subprocess.check_call(["nvcc", *B.ARCH, *B.NVFLAGS, *flags, "-I", B.CSRC, "-shared", str(src), "-o", str(so)])
    lib = C.CDLL(str(so))

    def call(what, *arrays):
        n = len(arrays[0])
        ins = [np.ascontiguousarray(x, np.float64) for x in arrays] + [np.ones(n)] * (5 - len(arrays))
        outs = [np.zeros(n) for _ in range(3)]
        ptr = lambda v: (C.c_void_p * len(v))(*[x.ctypes.data for x in v])
        assert lib.run(what, n, ptr(ins), ptr(outs)) == 0
        return outs

    return call


def _off(got, want):
    """Largest relative error in u."""
    return float(np.max(np.abs(got.astype(LD) / want - 1)) / U)


def _spread(rng, n, lo, hi):
    m = np.concatenate([rng.uniform(1, 2, n), 1 + np.arange(64) * 2.0 ** -52, 2 - np.arange(1, 65) * 2.0 ** -52])
    return m * 2.0 ** rng.integers(lo, hi, m.size)


@pytest.mark.gpu
def test_reciprocals_and_roots(device):
    r = np.random.default_rng(1)
    x = _spread(r, 400000, -1000, 1000)
    x = np.concatenate([x, -x])
    assert _off(device(0, x)[0], 1 / x.astype(LD)) <= 1.02
    x = _spread(r, 400000, -1000, 1000)
    assert _off(device(1, x)[0], 1 / np.sqrt(x.astype(LD))) <= 1.55
    x = np.concatenate([x, [np.finfo(float).tiny, np.finfo(float).max / 4]])
    assert _off(device(2, x)[0], np.sqrt(x.astype(LD))) <= 2.56
    small = np.array([0.0, 5e-324, 1e-310, np.nextafter(np.finfo(float).tiny, 0), np.inf])
    assert np.array_equal(device(2, small)[0], np.sqrt(small))
    assert np.all(np.isnan(device(2, np.array([-1.0, np.nan, -1e-310]))[0]))


@pytest.mark.gpu
def test_quotients(device):
    r = np.random.default_rng(2)
    a, b = _spread(r, 400000, -40, 40), _spread(r, 400000, -40, 40)
    r.shuffle(a)
    assert _off(device(3, a, b)[0], a.astype(LD) / b.astype(LD)) <= 1.001


@pytest.mark.gpu
def test_small_angles(device):
    r = np.random.default_rng(3)
    x = np.concatenate([r.uniform(0, 0.05, 200000), 0.05 * 2.0 ** -r.uniform(0, 40, 100000)])
    edge = 0.05 * (1 + np.linspace(-2e-6, 2e-6, 4001))
    far = r.uniform(0.0501, 3.2, 100000)
    for v, bound in ((x, 1.02), (edge, 2.0), (far, 2.0)):
        v = np.concatenate([v, -v])
        s, c, q = device(4, v)
        w = v.astype(LD)
        assert _off(c, np.cos(w)) <= (bound if bound < 2 else 2.0 / float(np.min(np.abs(np.cos(v)))))
        assert _off(s, np.sin(w)) <= (bound if bound < 2 else 2.0 / float(np.min(np.abs(np.sin(v)))))
        assert _off(q, np.sin(w) / w) <= (bound if bound < 2 else 1.0 + 2.0 / float(np.min(np.abs(np.sin(v)))))
    s, c, q = device(4, np.array([0.0, -0.0]))
    assert np.all(s == 0) and np.all(c == 1) and np.all(q == 1)


@pytest.mark.gpu
def test_riemann_series(device):
    r = np.random.default_rng(4)
    n = 400000
    w = 2.0 ** r.uniform(-12, 2, n)
    z = np.concatenate([r.uniform(-0.2, 0.2, n // 2), 0.2 * 2.0 ** -r.uniform(0, 50, n // 2)])
    t = np.concatenate([r.uniform(-0.2, 0.2, n // 2), -0.2 * 2.0 ** -r.uniform(0, 50, n // 2)])
    r.shuffle(t)
    a = 2.0 ** r.uniform(-40, 10, n)
    b = a * (1 + z) / (1 - z)
    ul = r.uniform(-1, 1, n) * w
    ur = ul - t * w
    um, pm, ok = device(5, a, b, w, ul, ur)
    A, Bb, W, L, R = (v.astype(LD) for v in (a, b, w, ul, ur))
    T, Z = (L - R) / W, (Bb - A) / (Bb + A)
    inside = (np.abs(Z) <= 0.125 - 1e-12) & (np.abs(T) <= 0.125 - 1e-12)
    outside = (np.abs(Z) >= 0.125 + 1e-12) | (np.abs(T) >= 0.125 + 1e-12)
    assert np.all(ok[inside] == 1) and np.all(ok[outside] == 0) and inside.sum() > n // 4 and outside.sum() > n // 4
    assert _off(pm[inside], np.exp(T)[inside]) <= 2.6
    want = (L + R) / 2 - W / 4 * (np.log1p(Z) - np.log1p(-Z))
    err = np.abs(um.astype(LD) - want) / (U * (W / 4 + np.abs(L) + np.abs(R)))
    assert float(np.max(err[inside])) <= 1.0


@pytest.mark.gpu
def test_quotients_by_multiplication(device):
    a, d = (v.ravel() for v in np.meshgrid(np.arange(128), np.arange(1, 129)))
    assert np.array_equal(device(6, a, d)[0], a // d)
    r = np.random.default_rng(5)
    d = np.concatenate([2.0 ** r.uniform(0, 20, 200000), [1, 2, 3, 116, 1 << 20]]).astype(np.int64)
    q = (2.0 ** r.uniform(0, np.minimum(24, 31 - np.log2(d + 1.0)))).astype(np.int64)
    for off in (-1, 0, 1):                      # around a multiple, where a quotient by multiplication goes wrong
        a = np.maximum(q * d + off, 0)
        a = np.minimum(a, 2 ** 31 - 2)
        assert np.array_equal(device(7, a, d)[0], a // d)


@pytest.mark.gpu
def test_density_bound_by_its_high_word(device):
    r = np.random.default_rng(6)
    b = 1e-15
    x = np.concatenate([_spread(r, 200000, -1000, 1000), b * (1 + r.uniform(-4e-6, 4e-6, 200000)), [b, np.nextafter(b, 0), np.nextafter(b, 1)]])
    x = np.concatenate([x, -x])
    got = device(8, x)[0]
    assert np.all(x[got == 1] > b)                       # never where the bound replaces a density
    assert np.all(x[got == 0] <= b * (1 + 2e-6))         # and not far above it does it ask for the exact look
    assert np.all(device(8, np.array([0.0, -0.0, 5e-324, np.inf, -np.inf, np.nan, -np.nan]))[0] == 0)
