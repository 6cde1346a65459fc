"""What the hydro step is used for, as cases that can be timed and compared.

A case names a disk (2D r-phi or 3D r-phi-theta; FP64 or FP32 planes;
isothermal or isentropic; planet on a fixed or a moving orbit) and the public
call that a program makes on it:

  reduce   one GPU_output_reduction each of the disk mass and the planet's torque
  host     Run.kernel_loop: the reference's call sequence, one call per phase
  advance  Run.advance: the device-resident loop, launch by launch or in graphs
  batch    Batch.advance: several disks of uneven sizes stepped together
  job      load a dump, advance, read the history, save the dump (pinned host memory)

Disks start as a run looks part way through: the seeded initial disk with
spiral density waves, and the velocities that go with them, on top.  exact()
restates the step (PPM Lagrange-remap sweeps, FARGO shift, planet, viscosity,
wave damping, CFL step) in torch float64, formula by formula, without the
package's code; only the input dump comes from the package.
"""
import math

import numpy as np
import torch

import penguin_2_0_b200 as pg
from penguin_2_0_b200 import _lib

PI, TWOPI = math.pi, 2.0 * math.pi
MOST_CELL_STEPS = 15_000_000


# ---- the cases --------------------------------------------------------------------
def _case(name, kind, nr, nphi, nk=1, precision=0, eos=0, planet=1, q=1e-3, steps=1, chunk=0, members=1):
    c = dict(kind=kind, nr=nr, nphi=nphi, nk=nk, precision=precision, eos=eos, planet=planet, q=q, steps=steps,
             chunk=chunk, members=members)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the diagnostics of a small disk, as a driver prints them: launch and read-back latency
        _case("reduce_128x384", "reduce", 128, 384),
        # a small disk of odd sizes stepped launch by launch (parameter studies, unit runs)
        _case("step_136x203", "advance", 136, 203, q=1e-4, steps=8),
        # the reference's driver moved over call by call, moving planet (its default), ragged sizes
        _case("host_251x767_moving", "host", 251, 767, planet=2, q=1e-4, steps=2),
        # the plain 2D disk in its device loop
        _case("plain_256x768", "advance", 256, 768, steps=32, chunk=16),
        # an isentropic disk
        _case("isentropic_384x1152", "advance", 384, 1152, eos=1, q=1e-4, steps=8, chunk=8),
        # the 2D disk with FP32 planes
        _case("planes32_1024x3072", "advance", 1024, 3072, precision=1, steps=4, chunk=4),
        # a large 2D disk
        _case("large_1536x4608", "advance", 1536, 4608, steps=2, chunk=2),
        # a small 3D disk as the serving stream draws them
        _case("small3d_80x240x24", "advance", 80, 240, nk=24, q=1e-4, steps=16, chunk=16),
        # the 3D disk with FP32 planes, ragged
        _case("planes32_3d_100x301x16", "advance", 100, 301, nk=16, precision=1, q=1e-5, steps=8, chunk=8),
        # the large 3D spherical disk
        _case("disk3d_128x1024x32", "advance", 128, 1024, nk=32, q=3e-4, steps=2, chunk=2),
        # an ensemble of uneven disks, FP64 and FP32 members
        _case("ensemble_16", "batch", 512, 1536, steps=4, chunk=4, members=16),
        # a whole job from a dump in host memory to a dump in host memory
        _case("job_256x768", "job", 256, 768, q=3e-4, steps=32, chunk=16),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _nphi(n, lo=126):
    """The nearest azimuthal count that the reference's chunking takes."""
    n = max(n, lo)
    while n % 116 in (1, 2, 3, 4, 5):
        n += 1
    return n


def draw(rng):
    kind = rng.choice(["reduce", "host", "advance", "advance", "advance3d", "advance3d", "batch", "job"])
    q = 10.0 ** rng.uniform(-5.0, -3.0)
    if kind == "batch":
        nr = _log_int(rng, 128, 512)
        return _case(None, "batch", nr, 3 * nr, steps=rng.randint(2, 4), chunk=2, members=rng.randint(3, 16))
    if kind == "advance3d":
        nr, nk = _log_int(rng, 48, 128), rng.randint(12, 48)
        nphi = _nphi(_log_int(rng, 130, 1024))
        steps = 2 * max(1, min(8, int(1.0e6 / (nr * nphi * nk))))
        return _case(None, "advance", nr, nphi, nk=nk, precision=rng.choice([0, 0, 1]), q=q, steps=steps,
                     chunk=rng.choice([0, 2]))
    nr = _log_int(rng, 64, 400 if kind in ("host", "job") else 1024)
    nphi = _nphi(int(nr * rng.uniform(1.5, 4.0)))
    steps = max(1, min(32, int(6.0e6 / (nr * nphi)), MOST_CELL_STEPS // (nr * nphi)))
    if kind == "reduce":
        return _case(None, "reduce", nr, nphi, precision=rng.choice([0, 1]), q=q)
    if kind == "host":
        return _case(None, "host", nr, nphi, planet=rng.choice([0, 1, 2]), q=q, steps=min(steps, 4))
    eos = rng.choice([0, 0, 0, 1])
    return _case(None, kind, nr, nphi, precision=0 if eos else rng.choice([0, 1]), eos=eos,
                 planet=rng.choice([1, 1, 2]), q=q, steps=steps, chunk=rng.choice([0, 4]))


# ---- inputs -----------------------------------------------------------------------
def _params(case, seed):
    """The pg_params of a case's disk; one per member of a batch."""
    far = dict(endtime=1.0e6, tmovie=1.0e6, seed=int(seed) & 0xFFFFFFFF)
    if case["kind"] == "batch":
        r = np.random.default_rng(int(seed) + 1)
        out = []
        for k in range(case["members"]):
            # the sizes and the precision policy of the ensemble: FP32 planes for weak planets
            nr = [case["nr"], case["nr"] // 2, case["nr"] // 4 + 64, case["nr"] // 3 + 21][k % 4]
            h, q = 0.04 + 0.03 * (k % 5) / 4.0, 10.0 ** (-5.0 + 2.0 * (k % 7) / 6.0)
            out.append(pg.params(0, imax=nr, jmax=_nphi(3 * nr), M_p=q, sc_h=h, ss_alpha=10.0 ** r.uniform(-4, -2),
                                 p_alpha=0.5 + 0.25 * (k % 5), precision=1 if q / h ** 3 <= 0.5 else 0,
                                 **dict(far, seed=far["seed"] + k)))
        return out
    if case["nk"] > 1:
        return [pg.params(1, imax=case["nr"], jmax=case["nphi"], kmax=case["nk"], M_p=case["q"],
                          plnt_flag=case["planet"], precision=case["precision"], **far)]
    more = dict(EOS=1, gam=1.4) if case["eos"] else {}
    return [pg.params(0, imax=case["nr"], jmax=case["nphi"], M_p=case["q"], plnt_flag=case["planet"],
                      precision=case["precision"], **more, **far)]


def _fields(buf, p):
    """The dump's r, p, u, v, w as one writable [rings, 5, jmax] view."""
    rb = 72 * p.jmax + 96
    return np.ndarray((p.imax * p.kmax, 5, p.jmax), np.float64, buf, strides=(rb, 8 * p.jmax, 8))


def _dump(p, seed):
    """The seeded disk with spiral waves (some 10 % in density, 0.1 of the sound speed) on top."""
    buf = pg.build_ic(p)
    f = _fields(buf, p)
    r = np.random.default_rng([int(seed), p.imax, p.jmax])
    rad = np.ndarray((p.imax * p.kmax,), np.float64, buf, offset=40 * p.jmax + 24, strides=(72 * p.jmax + 96,))
    phi = np.ndarray((p.jmax,), np.float64, buf, offset=40 * p.jmax + 32 + 24 * p.jmax)
    wave = np.zeros((2, p.imax * p.kmax, p.jmax))
    for m in (1, 2, 3, 5):
        k, a, b = r.uniform(-25.0, 25.0), r.uniform(0.02, 0.04), r.uniform(0.0, TWOPI)
        lead = k * np.log(rad) + b
        c, s = np.cos(m * phi), np.sin(m * phi)
        wave[0] += np.outer(a * np.cos(lead), c) - np.outer(a * np.sin(lead), s)
        wave[1] += np.outer(a * np.sin(lead), c) + np.outer(a * np.cos(lead), s)
    cs = (p.sc_h / np.sqrt(rad))[:, None]
    f[:, 0] *= 1.0 + wave[0]
    f[:, 1] *= (1.0 + wave[0]) ** (p.gam if p.EOS else 1.0)
    f[:, 2] += cs * wave[1]
    f[:, 3] += 0.5 * cs * wave[0]
    if p.ndim == 3:
        f[:, 4] += 0.5 * cs * wave[1]
    return buf


class _Plane:
    """A plane of a run as torch takes it; it holds the run, whose memory it is, as long as a tensor lives."""

    def __init__(self, run, ptr, view):
        self.run, e = run, view.elem_bytes
        self.__cuda_array_interface__ = dict(
            data=(ptr, False), shape=(view.kmax, view.imax, view.jmax), typestr="<f%d" % e, version=3,
            strides=(e * view.slab_stride, e * view.row_stride, e))


def _planes(run):
    """The run's current Sigma, v_r, v_phi planes, where they lie on the device."""
    v = _lib.pg_device_view()
    assert _lib.lib().pg_device_view_get(run._h, v) == 0
    return [torch.as_tensor(_Plane(run, q, v), device="cuda") for q in (v.sigma, v.vr, v.vphi)]


def _pinned(nbytes):
    return torch.empty(nbytes, dtype=torch.uint8, pin_memory=True)


def prepare(case, seed):
    ps = _params(case, seed)
    runs = []
    for k, p in enumerate(ps):
        buf = _dump(p, seed + 1000 * k)
        run = pg.Run(p, 0)
        if case["kind"] == "job":
            src, dst = _pinned(len(buf)), _pinned(len(buf))
            src.numpy()[:] = np.frombuffer(buf, np.uint8)
            return dict(case=case, run=run, src=src, dst=dst)
        n = len(buf)
        run.load_from(np.frombuffer(buf, np.uint8).ctypes.data, n)
        if case["kind"] in ("advance", "batch"):
            run.clock_reset(0)
        runs.append(run)
    st = dict(case=case, runs=runs, run=runs[0], planes=[t for r in runs for t in _planes(r)])
    if case["kind"] == "batch":
        st["batch"] = pg.Batch(0)
        for r in runs:
            st["batch"].add(r)
    if case["kind"] == "reduce":
        st["planet"], _ = pg.init_planet(ps[0])
    return st


def run(state):
    case, r = state["case"], state["run"]
    kind, steps = case["kind"], case["steps"]
    if kind == "reduce":
        return [pg.GPU_output_reduction(r, state["planet"], 0.0, 0), pg.GPU_output_reduction(r, state["planet"], 0.0, 9)]
    if kind == "host":
        s, simtime, dt, planet, frrot = r.kernel_loop(steps)
        return state["planes"] + [simtime, planet.y, frrot]
    if kind == "batch":
        state["batch"].advance(steps, chunk=case["chunk"])
        state["batch"].sync()
        return state["planes"]
    if kind == "job":
        src, dst = state["src"], state["dst"]
        r.load_from(src.data_ptr(), src.numel())
        r.clock_reset(0)
        r.advance(steps, graph_chunk=case["chunk"])
        rows = r.history()
        r.save_to(dst.data_ptr(), dst.numel())
        return [dst.view(torch.float64), rows]
    r.advance(steps, graph_chunk=case["chunk"])
    # in 3D an even number of steps leaves the current planes where they were
    return state["planes"]


def work(case):
    """Each field read once and written once by each sweep; some 250 FP64 operations per cell and sweep."""
    if case["kind"] == "reduce":
        cells = case["nr"] * case["nphi"]
        return dict(bytes=2.0 * cells * (4 if case["precision"] else 8), flops=40.0 * cells)
    total = dict(bytes=0.0, flops=0.0)
    for p in _params(case, 0):
        cells = p.imax * p.jmax * p.kmax
        ns = p.ndim                                       # sweeps
        nf = 3 if p.ndim == 2 else 4                      # fields
        total["bytes"] += case["steps"] * cells * (2.0 * nf * ns * (4 if p.precision else 8))
        total["flops"] += case["steps"] * cells * 250.0 * ns
        if case["kind"] == "job":
            total["bytes"] += cells * (40.0 + 72.0)
    return total


# ---- the step in plain float64 ----------------------------------------------------
SMALL = 1.0e-15
PAD, REAL, ARR = 6, 116, 128


def _m(x):
    return torch.roll(x, 1, 0)       # value of cell n - 1 (the ends of a chunk are never used)


def _p(x):
    return torch.roll(x, -1, 0)      # value of cell n + 1


class _Disk:
    """One disk and its loop."""

    def __init__(self, p, buf):
        self.p, D = p, dict(dtype=torch.float64, device="cuda")
        self.D = D
        nr, nk, nphi = p.imax, p.kmax, p.jmax
        self.three = p.ndim == 3
        rb = 72 * nphi + 96
        f = torch.from_numpy(np.ascontiguousarray(_fields(buf, p))).to("cuda").reshape(nk, nr, 5, nphi)

        def ring(off):
            return np.ndarray((nr * nk,), np.float64, buf, offset=off, strides=(rb,)).reshape(nk, nr)

        x, dx = ring(40 * nphi)[0], ring(40 * nphi + 8)[0]
        z, dz = ring(72 * nphi + 32)[:, 0], ring(72 * nphi + 40)[:, 0]
        y = np.ndarray((2, nphi), np.float64, buf, offset=40 * nphi + 32)
        pads = np.arange(PAD)

        def padded(a, d):
            a = np.concatenate([a[0] - d[0] * (PAD - pads), a, a[-1] + d[-1] * (pads + 1)])
            return torch.tensor(a, **D), torch.tensor(np.concatenate([d[0] + 0 * pads, d, d[-1] + 0 * pads]), **D)

        self.x, self.dx = padded(x, dx)
        self.xc = self.x + 0.5 * self.dx
        self.y, self.dy = torch.tensor(y[0], **D), torch.tensor(y[1], **D)
        self.yc = self.y + 0.5 * self.dy
        if self.three:
            self.z, self.dz = padded(z, dz)
            self.zc = self.z + 0.5 * self.dz
            self.xvol = self.dx * (self.x * (self.x + self.dx) + self.dx ** 2 / 3.0)
        else:
            self.z = self.dz = self.zc = None
            self.xvol = self.dx * (self.x + 0.5 * self.dx)
        # profile at every ring (ghosts included), [nk (+12), nr + 12]
        sinz = torch.sin(self.zc) if self.three else torch.ones(1 + 2 * PAD, **D)
        cosz = torch.cos(self.zc) if self.three else torch.zeros(1 + 2 * PAD, **D)
        self.rc = self.xc[None, :] * sinz[:, None]
        self.prof_r, self.prof_p, self.prof_v = self._profile(sinz, cosz)
        self.nu = p.ss_alpha * p.sc_h ** 2 * self.rc ** p.p_alpha if p.visc_flag == 1 else None
        self.prof_u = (-1.5 * p.ss_alpha * p.sc_h ** 2 if p.visc_flag == 1 else 0.0) * self.rc ** (p.p_alpha - 1.0)
        self.cs2 = p.sc_h ** 2 * self.rc ** -p.p_beta
        ins = slice(PAD, PAD + nk)
        inr = slice(PAD, PAD + nr)
        self.ins, self.inr = ins, inr
        self.val = [a[ins, inr] for a in (self.prof_r, self.prof_u, self.prof_v)]
        # planes [nk, nr + 12, nphi] with the fixed radial ghost rings
        one = torch.ones(nphi, **D)

        def plane(k, ghost):
            a = ghost[ins][:, :, None] * one
            a[:, inr] = f[:, :, k]
            return a

        self.S = [plane(0, self.prof_r), plane(2, self.prof_u), plane(3, self.prof_v), plane(4, 0 * self.prof_r)]
        self.S = self.S if self.three else self.S[:3] + [torch.zeros_like(self.S[0])]
        self.p0 = plane(1, self.prof_p)
        self.rot_v = torch.zeros_like(self.prof_v[ins])
        self.rot_v[:, inr] = torch.tensor(ring(72 * nphi + 72), **D)
        self.res_v = torch.zeros_like(self.rot_v)
        self.inc = torch.zeros(nk, nr, dtype=torch.long, device="cuda")
        g = torch.zeros_like(self.xc[inr])
        r = self.xc[inr]
        if p.kill_rin > 0:
            g = torch.where(r < p.kill_rin, (p.kill_rin - r) / (p.kill_rin - p.xmin), g)
        if p.kill_rout > 0:
            g = torch.where(r > p.kill_rout, (r - p.kill_rout) / (p.xmax - p.kill_rout), g)
        self.damp = g * r ** -1.5
        self.pl = dict(m=p.M_p, x=p.R_p, y=PI, vx=0.0, vy=p.R_p ** -1.5, fx=0.0, fy=0.0)
        self.fr = self.pl["vy"] if p.FrRot_flag == 1 else 0.0
        self.pl["vy"] -= self.fr
        self._softening()
        self.simtime = 0.0

    def _profile(self, sinz, cosz):
        p = self.p
        gam, h2 = p.gam, p.sc_h ** 2

        def rho(R, Z):
            a = R ** -p.p_alpha
            return a * torch.exp((1.0 / torch.sqrt(R * R + Z * Z) - 1.0 / R) / (h2 * R ** -p.p_beta)) if self.three else a

        def pres(R, Z):
            d = rho(R, Z)
            return h2 * R ** -p.p_beta * (d if p.EOS == 0 else d ** gam / gam)

        R, Z = self.rc, self.xc[None, :] * cosz[:, None]
        if self.three:
            e = 1.27e-7
            s, c = sinz[:, None], cosz[:, None]
            dP = (pres((self.xc + e) * s, (self.xc + e) * c) - pres((self.xc - e) * s, (self.xc - e) * c)) / (2.0 * e)
        else:
            e = 1.27245e-8
            dP = (pres(R + e, Z) - pres(R - e, Z)) / 2.5449e-8
        d = rho(R, Z)
        return d, pres(R, Z), torch.sqrt(1.0 / self.xc + self.xc * dP / d)

    # -- planet --
    def _softening(self):
        p, x = self.p, self.pl["x"]
        self.pl["rs"] = p.rs_fac * math.sqrt(p.sc_h ** 2 * x ** -p.p_beta * x ** 3)

    def _kick(self, dt):
        b = self.pl
        b["vx"] += dt * b["fx"]
        b["vy"] += self.fr + dt * b["fy"] / b["x"] ** 2
        self.fr = b["vy"] if self.p.FrRot_flag == 1 else 0.0
        b["vy"] -= self.fr

    def _drift(self, dt):
        b, old = self.pl, self.pl["x"]
        b["x"] += dt * b["vx"]
        b["y"] += dt * b["vy"]
        b["vy"] = (b["vy"] + self.fr) * old ** 2 / b["x"] ** 2 - self.fr
        b["y"] += TWOPI if b["y"] < 0.0 else -TWOPI if b["y"] >= TWOPI else 0.0
        if self.p.plnt_flag == 2:
            self._softening()

    def _forces(self):
        b = self.pl
        b["fx"] = -1.0 / b["x"] ** 2 + b["x"] * (b["vy"] + self.fr) ** 2
        b["fy"] = 0.0
        if self.p.plnt_flag == 2:
            b["fx"] += self.p.Sigma_0 * self.reduce(8) / b["m"]
            b["fy"] = self.p.Sigma_0 * self.reduce(9) / b["m"]

    def reduce(self, mode):
        p, r = self.p, self.S[0][:, self.inr]
        vol = self.xvol[self.inr][None, :, None] * self.dy
        if mode == 0 or p.plnt_flag == 0:
            if self.three:
                vol = vol * (torch.cos(self.z) - torch.cos(self.z + self.dz))[self.ins][:, None, None]
            return float((r * vol).sum())
        if self.three:
            return 0.0
        rad = self.xc[self.inr][None, :, None]
        g = -self._grav(0 if mode == 8 else 1, rad, self.yc, None, 0.0)
        return float(((rad if mode == 9 else 1.0) * g * (r - rad ** -p.p_alpha) * vol).sum())

    def _grav(self, ax, rad, azi, pol, dt):
        """Planet (and, with a planet in 3D radial sweeps, star) acceleration at rad, azi, pol after dt."""
        b = self.pl
        px = b["x"]
        a = azi - (b["y"] + dt * b["vy"])
        c, s = torch.cos(a), torch.sin(a)
        if not self.three:
            R3 = torch.sqrt(rad * rad + px * px - 2.0 * px * rad * c + b["rs"] ** 2) ** 3
            if ax == 0:
                return -b["m"] * (rad - px * c) / R3 - b["m"] * c / px ** 2
            return -b["m"] * px * s / R3 + b["m"] * s / px ** 2
        st, ct = torch.sin(pol), torch.cos(pol)
        mass = b["m"] / (1.0 + b["m"])
        if ax == 1:
            rad = rad / st
        R3 = torch.sqrt(rad * rad + px * px - 2.0 * px * rad * c * st + b["rs"] ** 2) ** 3
        if ax == 0:
            return -mass * (rad - px * c * st) / R3 - 1.0 / (1.0 + b["m"]) / rad ** 2 - mass * st * c / px ** 2
        if ax == 1:
            return -mass * px * s / R3 + mass * st * s / px ** 2
        return mass * px * c * ct / R3 - mass * c * ct / (st * px ** 2)

    def _force(self, ax, rad, azi, pol, v, w, dt):
        """Acceleration along the sweep, centrifugal terms included."""
        planet = self.p.plnt_flag > 0
        if ax == 0 and not self.three:
            return (self._grav(0, rad, azi, pol, dt) if planet else 0.0) - 1.0 / rad ** 2 + v * v / rad ** 3
        if ax == 0:
            g = self._grav(0, rad, azi, pol, dt) if planet else -1.0 / rad ** 2
            return g + w * w / rad ** 3 + v * v / rad / (rad * torch.sin(pol)) ** 2
        if ax == 1:
            return self._grav(1, rad, azi, pol, dt) if planet else torch.zeros_like(v)
        g = self._grav(2, rad, azi, pol, dt) if planet else 0.0
        return g + w * w * torch.cos(pol) / (rad * torch.sin(pol)) ** 3

    # -- one chunk along dim 0 --
    @staticmethod
    def _paraset(d):
        a, b, c = d + _p(d), 2.0 * d + _p(d), d + 2.0 * _p(d)
        am, ap = _m(a), _p(a)
        q = 1.0 / (am + ap)
        c0 = d / a * (1.0 + 2.0 * q * _p(d) * (am / b - ap / c))
        e = d / (am + _p(d))
        return c0, -q * d * am / b, q * _p(d) * ap / c, e * _m(b) / a, e * c / am

    @staticmethod
    def _parabola(val, flat, par):
        c0, c1, c2, c3, c4 = par
        dr, dl = _p(val) - val, val - _m(val)
        t = c3 * dr + c4 * dl
        lim = torch.minimum(t.abs(), 2.0 * torch.minimum(dl.abs(), dr.abs()))
        t = torch.where(dl * dr < 0.0, torch.zeros_like(t), torch.where(t < 0.0, -lim, lim))
        ar = val + c0 * dr + c1 * _p(t) + c2 * t
        xr = flat * val + (1.0 - flat) * ar
        la = flat * val + (1.0 - flat) * _m(ar)
        d, six = xr - la, 6.0 * (val - 0.5 * (xr + la))
        flatten = (xr - val) * (val - la) <= 0.0
        xr, la = torch.where(flatten, val, xr), torch.where(flatten, val, la)
        la, xr = (torch.where(d * d < d * six, 3.0 * val - 2.0 * xr, la),
                  torch.where(d * d < -d * six, 3.0 * val - 2.0 * la, xr))
        return la, xr, xr - la, 6.0 * (val - 0.5 * (xr + la))

    def _riemann(self, pl, rl, ul, pr, rr, ur):
        p = self.p
        if p.EOS == 0:
            t1 = 0.5 * (torch.sqrt(pl / rl) + torch.sqrt(pr / rr))
            pm = torch.sqrt(pl * pr) * torch.exp(-0.5 * (ur - ul) / t1)
            return ul - t1 * torch.log(pm / pl), pm.clamp_min(SMALL)
        g1, g2 = (p.gam + 1.0) / p.gam / 2.0, p.gam + 1.0
        cl, cr = torch.sqrt(p.gam * pl * rl), torch.sqrt(p.gam * pr * rr)
        pm = (pl + (pr - pl - cr * (ur - ul)) * cl / (cl + cr)).clamp_min(SMALL)
        live = torch.ones_like(pm, dtype=torch.bool)
        wl = wr = None
        for _ in range(10):
            wl_, wr_ = cl * torch.sqrt(1.0 + g1 * (pm - pl) / pl), cr * torch.sqrt(1.0 + g1 * (pm - pr) / pr)
            wl, wr = (wl_, wr_) if wl is None else (torch.where(live, wl_, wl), torch.where(live, wr_, wr))
            zl, zr = 4.0 / rl * wl * wl, 4.0 / rr * wr * wr
            zl, zr = -zl * wl / (zl - g2 * (pm - pl)), zr * wr / (zr - g2 * (pm - pr))
            new = (pm + ((ur + (pm - pr) / wr) - (ul - (pm - pl) / wl)) * (zr * zl) / (zr - zl)).clamp_min(SMALL)
            new = torch.where(live, new, pm)
            live = live & ~((new - pm).abs() / new < 1.0e-8)
            pm = new
        return 0.5 * ((ul - (pm - pl) / wl) + (ur + (pm - pr) / wr)), pm.clamp_min(SMALL)

    def _chunk(self, ax, dt, x, d0, dvol0, rad, azi, pol, vrot, r, p, u, v, w):
        """The Lagrange-remap chain; arrays [cells, ...].  Returns r, u, v, w, remapped for 6 <= n < L - 6."""
        L, P, three = r.shape[0], self.p, self.three
        n = torch.arange(L, device="cuda").reshape([L] + [1] * (r.dim() - 1))
        flat = torch.zeros_like(r)
        if P.flat_flag:
            d1, d2 = _p(p) - _m(p), _p(_p(p)) - _m(_m(p))
            d2 = torch.where(d2.abs() < SMALL, torch.full_like(d2, SMALL), d2)
            shock = (d1.abs() / torch.minimum(_p(p), _m(p)) > 0.33) & ~(_m(u) < _p(u)) & (n >= 2) & (n < L - 2)
            steep = torch.where(shock, ((d1 / d2 - 0.75) * 5.0).clamp_min(0.0), flat)
            flat = torch.maximum(torch.maximum(_m(steep), steep), _p(steep)).clamp_max(0.5)
            flat = torch.where((n >= 2) & (n < L - 2), flat, torch.zeros_like(flat))
        h = 0.5 * dt
        # faces: sound crossing, states, forces, Riemann problem
        if ax == 0:
            f = self._force(0, x, azi + h * vrot, pol, 0.5 * (v + _m(v)), 0.5 * (w + _m(w)), h)
        elif ax == 1:
            f = self._force(1, rad, x + h * vrot, pol, v, w, h)
        else:
            f = self._force(2, rad, azi + h * vrot, x, v, 0.5 * (w + _m(w)), h)
        cs = h * torch.sqrt(P.gam * p / r) / d0 / (rad if ax else 1.0)
        fac = 1.0 - 4.0 / 3.0 * cs
        par, left, right = self._paraset(d0), [], []
        for q in (p, r, u):
            la, xr, da, a6 = self._parabola(q, flat, par)
            left.append(_m(xr - cs * (da - fac * a6)))
            right.append(la + cs * (da + fac * a6))
        um, pm = self._riemann(left[0].clamp_min(SMALL), left[1].clamp_min(SMALL), left[2] + h * f,
                               right[0].clamp_min(SMALL), right[1].clamp_min(SMALL), right[2] + h * f)
        # Lagrangian step
        delx = dt * um if ax == 0 else dt * (um / rad - vrot - self.fr) if ax == 1 else dt * um / rad
        xa = x + delx
        dx = _p(xa) - xa
        xn = xa + 0.5 * dx
        if ax == 0:
            f1 = self._force(0, rad, azi, pol, v, w, 0.0)
            f2 = self._force(0, xn, azi + dt * vrot, pol, v, w, dt)
        elif ax == 1:
            f1 = self._force(1, rad, azi, pol, v, w, 0.0)
            f2 = self._force(1, rad, xn + dt * vrot, pol, v, w, dt)
        else:
            f1 = self._force(2, rad, azi, pol, v, w, 0.0)
            f2 = self._force(2, rad, azi + dt * vrot, xn, v, w, dt)
        xe = torch.where(n < L - 3, xa, x + 0 * xa)      # the last face's factor is taken at its start
        de = xe - x
        if ax == 0 and not three:
            dvol, vf, lvol = dx * (xa + 0.5 * dx), 0.5 * (xe + x), delx * (x + 0.5 * delx)
        elif ax == 0:
            dvol = dx * (xa * (xa + dx) + dx * dx / 3.0)
            vf, lvol = de * (de / 3.0 + x) + x * x, delx * (x * xa + delx * delx / 3.0)
        elif ax == 1:
            dvol, vf, lvol = dx * rad, torch.ones_like(dx), delx * rad
        else:
            dvol = 2.0 * torch.sin(xn) * torch.sin(0.5 * dx) * rad
            mid, half = torch.sin(x + 0.5 * de), torch.sin(0.5 * de)
            vf = torch.where(de == 0.0, torch.sin(x) + 0 * de, 2.0 * mid * half / torch.where(de == 0.0, de + 1.0, de))
            lvol = 2.0 * torch.sin(x + 0.5 * delx) * torch.sin(0.5 * delx) * rad
        u = u + 0.5 * dt * (f1 + f2) - dt / (r * dvol0) * (_p(pm) - pm) * 0.5 * (_p(vf) + vf)
        r = (r * (dvol0 / dvol)).clamp_min(SMALL)
        # remap
        par, up = self._paraset(dx), delx >= 0.0
        e = 0.5 * delx / torch.where(up, _m(dx), dx)
        e2 = torch.where(up, 1.0 - 4.0 / 3.0 * e, 1.0 + 4.0 / 3.0 * e)
        flux, fields = [], [r, u, v, w]
        for k, q in enumerate(fields):
            la, xr, da, a6 = self._parabola(q, flat, par)
            t = torch.where(up, _m(xr) - e * (_m(da) - e2 * _m(a6)), la - e * (da + e2 * a6))
            flux.append(t * (lvol if k == 0 else flux[0]))
        mass, inside = r * dvol, (n >= 6) & (n < L - 6)
        rn = ((mass + flux[0] - _p(flux[0])) / dvol0).clamp_min(SMALL)
        out = [torch.where(inside, rn, r)]
        for q, g in zip(fields[1:], flux[1:]):
            out.append(torch.where(inside, (q * mass + g - _p(g)) / (rn * dvol0), q))
        return out

    @staticmethod
    def _derivs(x, q):
        x2, x3 = x - _m(x), _p(x) - _m(x)
        h2, h3 = (q - _m(q)) / x2, (_p(q) - _m(q)) / x3
        a = (h3 - h2) / (x3 - x2)
        return 2.0 * a * x2 + (x3 * h2 - x2 * h3) / (x3 - x2), 2.0 * a

    def _pressure(self, r, cs2):
        return r * cs2 if self.p.EOS == 0 else cs2 * r ** self.p.gam / self.p.gam

    def _chunks(self, n):
        for l in range(n // REAL + (1 if n % REAL else 0)):
            last = REAL * (l + 1) >= n
            if last and n % REAL == 0:
                continue                                  # the reference leaves a full last chunk as it is
            yield REAL * l, (n % REAL + 2 * PAD) if last else ARR

    def sweep_x(self, dt):
        p, S = self.p, self.S
        out = [a.clone() for a in S]
        cs2 = self.cs2[self.ins]
        P = self.p0 if self.p0 is not None else self._pressure(S[0], cs2[:, :, None])
        ghost = torch.ones_like(self.x, dtype=torch.bool)
        ghost[self.inr] = False
        P = torch.where(ghost[None, :, None], self.prof_p[self.ins][:, :, None] + 0 * P, P)
        for a, L in self._chunks(p.imax):
            s = slice(a, a + L)

            def col(t):
                return t[s][:, None, None]

            def cut(t):
                return t[:, s].transpose(0, 1)

            rc, rad = self.rc[self.ins][:, s].t()[:, :, None], col(self.xc)
            vrot = (self.res_v / self.rc[self.ins])[:, s].t()[:, :, None]
            pol = self.zc[self.ins][None, :, None] if self.three else None
            r, u, v, w = self._chunk(0, dt, col(self.x), col(self.dx), col(self.xvol), rad, self.yc, pol, vrot, cut(S[0]),
                                     cut(P), cut(S[1]), cut(S[2]) * rc, cut(S[3]) * rad if self.three else cut(S[3]))
            if self.nu is not None:
                x, nr, om, dtr = col(self.x), self.nu[self.ins][:, s].t()[:, :, None] * r, v / rc ** 2, dt / r
                dn, du, dv, dw = (self._derivs(x, q) for q in (nr, u, om, w))
                un = u + dtr * (2 * nr * du[1] + 2 * dn[0] * du[0] + 2 * nr * du[0] / rc - 2 * nr * u / rc ** 2)
                v = (om * rc + dtr * (rc * nr * dv[1] + rc * dn[0] * dv[0] + 3 * nr * dv[0])) * rc
                w = w + dtr * (nr * dw[1] + dn[0] * dw[0] + nr * dw[0] / rc)
                u = un
            for o, q in zip(out, (r, u, v / rc, w / rad)):
                o[:, a + PAD:a + L - PAD] = q[PAD:L - PAD].transpose(0, 1)
        self.S, self.p0 = out, None

    def sweep_y(self, dt):
        p, S = self.p, self.S
        out = [a.clone() for a in S]
        I = (self.ins, self.inr)
        rc, cs2 = self.rc[I], self.cs2[I]
        vrot = self.res_v[:, self.inr] / rc
        pol = self.zc[self.ins][:, None] if self.three else None
        for a, L in self._chunks(p.jmax):
            j = torch.arange(a - PAD, a - PAD + L, device="cuda")
            turn = TWOPI * torch.div(j, p.jmax, rounding_mode="floor").double()
            jw = j % p.jmax

            def col(t):
                return t[jw][:, None, None]

            def cut(t):
                return t[:, self.inr][:, :, jw].permute(2, 0, 1)

            shift = turn[:, None, None]
            x = col(self.y) + shift
            r0 = cut(S[0])
            r, u, v, w = self._chunk(1, dt, x, col(self.dy), col(self.dy) * rc, rc + 0 * r0, col(self.yc) + shift, pol, vrot,
                                     r0, self._pressure(r0, cs2), cut(S[2]), cut(S[3]), cut(S[1]))
            if self.nu is not None:
                nr, dtr = self.nu[I] * r, dt / r
                dn, du, dv, dw = (self._derivs(x * rc, q) for q in (nr, u, v, w))
                u, v, w = (u + dtr * (2 * nr * du[1] + 2 * dn[0] * du[0]), v + dtr * (nr * dv[1] + dn[0] * dv[0]),
                           w + dtr * (nr * dw[1] + dn[0] * dw[0]))
            for o, q in zip(out, (r, w, u, v)):
                o[:, self.inr, a:a + L - 2 * PAD] = q[PAD:L - PAD].permute(1, 2, 0)
        self.S = out

    def sweep_z(self, dt):
        p, S, D = self.p, self.S, self.D
        nk, out = p.kmax, [a.clone() for a in S]
        rad = self.xc[self.inr][None, :, None]
        low = slice(0, PAD)
        cs2 = self.cs2[self.ins][:, self.inr, None]
        inner = [q[:, self.inr] for q in S]
        P = self._pressure(inner[0], cs2)
        up = torch.arange(nk - 1, nk - 1 - PAD, -1, device="cuda")
        rcg = self.rc[:, self.inr][:, :, None]
        vr_in = (self.res_v[:, self.inr] / self.rc[self.ins][:, self.inr])[:, :, None]

        def ext(q, ghost, sign=1.0):
            g = ghost[low][:, self.inr, None] + 0 * q[:1]
            return torch.cat([g, q, sign * q[up]])

        r, P = ext(inner[0], self.prof_r), ext(P, self.prof_p)
        ur, vp, vt = ext(inner[1], self.prof_u), ext(inner[2], self.prof_v), ext(inner[3], 0 * self.prof_r, -1.0)
        vrot = torch.cat([0 * vr_in[:1].expand(PAD, -1, -1), vr_in, vr_in[up]])
        zvol = 2.0 * torch.sin(self.zc) * torch.sin(0.5 * self.dz)
        for a, L in self._chunks(nk):
            s = slice(a, a + L)

            def col(t):
                return t[s][:, None, None]

            g = self._chunk(2, dt, col(self.z), col(self.dz), col(zvol) * rad, rad + 0 * r[s], self.yc, col(self.zc), vrot[s],
                            r[s], P[s], vt[s], ur[s], vp[s] * rcg[s])
            rn, u, v, w = g
            if self.nu is not None:
                x, nr, dtr = col(self.z) * rad, self.nu[s][:, self.inr, None] * rn, dt / rn
                dn, du, dv = (self._derivs(x, q) for q in (nr, u, v))
                u, v = u + dtr * (2 * nr * du[1] + 2 * dn[0] * du[0]), v + dtr * (nr * dv[1] + dn[0] * dv[0])
            for o, q in zip(out, (rn, v, w / rcg[s], u)):
                o[a:a + L - 2 * PAD, self.inr] = q[PAD:L - PAD]
        self.S = out

    # -- the loop --
    def rate(self):
        p, (r, u, v, w) = self.p, [q[:, self.inr] for q in self.S]
        rc = self.rc[self.ins][:, self.inr, None]
        P = self.p0[:, self.inr] if self.p0 is not None else self._pressure(r, self.cs2[self.ins][:, self.inr, None])
        cs = torch.sqrt(p.gam * P / r)
        t = (u.abs() + cs) / self.dx[self.inr][None, :, None]
        t = torch.maximum(t, ((v - self.rot_v[:, self.inr, None] - self.fr * rc).abs() + cs) / (self.dy * rc))
        if self.three:
            t = torch.maximum(t, (w.abs() + cs) / (self.dz[self.ins][:, None, None] * self.xc[self.inr][None, :, None]))
        return float(t.max())

    def advance(self, steps):
        p = self.p
        dt = p.endtime
        if p.plnt_flag:
            self._forces()
        for _ in range(steps):
            dt = min(1.1 * dt, p.courant / self.rate())
            wid = self.xc[self.inr][None, :] * self.dy[0] / dt
            jp = self.rot_v[:, self.inr] / wid
            self.inc = torch.where(jp >= 0, torch.floor(jp + 0.5), torch.ceil(jp - 0.5)).long()
            self.res_v[:, self.inr] = torch.floor(jp + 0.5) * wid
            self.rot_v[:, self.inr] = self.val[2] - self.fr * self.xc[self.inr]
            if p.plnt_flag:
                self._kick(0.5 * dt)
            self.sweep_x(dt)
            self.sweep_y(dt)
            if self.three:
                self.sweep_z(dt)
            src = (torch.arange(p.jmax, device="cuda") - self.inc[:, :, None]) % p.jmax
            for q in self.S:
                q[:, self.inr] = torch.gather(q[:, self.inr], 2, src)
            f = (dt * self.damp)[None, :, None]
            for q, t in zip(self.S, self.val + [torch.zeros_like(self.val[0])]):
                q[:, self.inr] += f * (t[:, :, None] - q[:, self.inr])
            self.simtime += dt
            if p.plnt_flag:
                self._drift(dt)
                self._forces()
                self._kick(0.5 * dt)

    def planes(self):
        r, u, v = (q[:, self.inr] for q in self.S[:3])
        if self.p.precision:
            r, v = r - self.val[0][:, :, None], v - self.val[2][:, :, None]
        return [r, u, v]


def exact(case, seed):
    if case["kind"] == "job":
        return None
    out = []
    for k, p in enumerate(_params(case, seed)):
        d = _Disk(p, _dump(p, seed + 1000 * k))
        if case["kind"] == "reduce":
            return [d.reduce(0), d.reduce(9)]
        d.advance(case["steps"])
        out += d.planes()
        if case["kind"] == "host":
            out += [d.simtime, d.pl["y"], d.fr]
    return out
