// pg_step.cu -- what happens between the sweeps: dt, Index_Shift, the planet,
// the diagnostics and the clock of main.cu:343-441, and the ring reductions.
//
//   k_between   one launch from the end of a step to the start of the next:
//               rotate_rings, time, planet drift/forces/kick and bookkeeping of
//               the finished step, its mass and torque sums and history row
//               where it prints, then the next step's dt, half kick and
//               Index_Shift
//   k_moving    moving planet: drift, the disk's forces on the drifted planet
//               (reductions 8 and 9), kick
//   k_reduce    output_lv1/lv2/lv3 (device_func.cu:49-167) of a run
//   kb_between  k_between of every member of a batch
//
// Every CTA of a run forms the scalar part from the clock as it was before the
// launch, in its own copy; each does its share of the rings; the last CTA to
// finish (a counter, no waiting) adds the sums up and stores the clock.  One
// launch takes the place of five (poststep, two sums, record, prestep) that
// took 20 us of the 128x384 disk's step and 40 us of the 128x1024x32 disk's,
// where one CTA went over 4096 rings.  Step launched call by call, 136x203:
// 64 -> 34 us; in graphs, 256x768: 46 -> 42 us; moving planet 251x767: 143 ->
// 59 us (its two force sums took 16 us each with one 1024-thread CTA per ring,
// cos, sin and divisions per cell).  Latency bound: one thread's chain of FP64
// divisions.
//
// Sums take one CTA of 8 warps per ring: thread (w, L) holds the cells
// L + 32 (w + 8 q), q = 0..3, of a 1024-cell block of the reference's tree
// (list[t] += list[t + half]).  The levels 512 and 256 pair values of a thread,
// 128..32 values of a lane in different warps (through shared memory) and 16..1
// values of different lanes (by shuffle), every addition with the tree's two
// operands, so the order is the reference's bit for bit.
// The planet's force on a cell takes cos and sin of its azimuth from the
// column tables and one reciprocal square root.
//
// Compiled without contraction, as the host arithmetic it restates.
#include "pg_warp.cuh"

namespace pgd {

// Index_Shift orbital_advection.cu:12-43
__device__ __forceinline__ void index_shift_ring(const Tables &T, int t, double dt, double FrRot, int fargo) {
  const int k = t / T.nr, i = t % T.nr;
  const int row = i + NPAD, rk = k * T.nrg + row;
  const double xc = T.rxc[row];
  const double widthy = xc * T.dy[0] / dt;
  double rot_v;
  if (fargo == 1) rot_v = fma(-FrRot, xc, T.val_v[rk]);   // contracted in the reference's build
  else if (fargo == 2) rot_v = (1.0 - FrRot) * xc;
  else rot_v = 0.0;
  const double jp = T.rot_v[rk] / widthy;
  T.inc_j[rk] = jp >= 0.0 ? (int)(jp + 0.5) : (int)(jp - 0.5);
  T.res_v[rk] = floor(jp + 0.5) * widthy;
  T.rot_v[rk] = rot_v;
  set_shift(T, rk, T.inc_j[rk], T.rot_j[rk]);
}
// what the device loop's last sweep needs of a ring: this step's damping
// factor, the frame offset of the next get_dt's azimuthal rate and (polar) the
// planet's turn against it in half a step
__device__ __forceinline__ void finish_ring(const Tables &T, int t, double dt, double frrot_next, double vy, int ndim) {
  const int rk = t / T.nr * T.nrg + t % T.nr + NPAD;
  const double g = T.damp_g[rk];
  T.ro[rk].f = g > 0.0 ? g * (dt * T.damp_pw[rk]) : 0.0;
  T.ro[rk].off = fma(frrot_next, T.radc[rk], T.rot_v[rk]);
  if (ndim == 3) T.turn[rk] = turn_of(dt, T.res_v[rk], T.irc[rk], vy);
}
// rotate_rings ppm.cu:309-322, and also where a ring turns more than once in a
// step (a cold disk of few rings): dumps and sums index by rot_j
__device__ __forceinline__ int rotated(const Tables &T, int rk) {
  const int j = wrap1(T.rot_j[rk] + T.inc_j[rk], T.nphi);
  return (unsigned)j < (unsigned)T.nphi ? j : wrapm(j, T.nphi);
}

__global__ void k_index(Tables T, double dt, double frrot, int fargo) {
  after_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < T.nr * T.nk) index_shift_ring(T, t, dt, frrot, fargo);
}
__global__ void k_rotate(Tables T) {
  after_previous();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= T.nr * T.nk) return;
  const int rk = t / T.nr * T.nrg + t % T.nr + NPAD;
  const int rot = rotated(T, rk);
  T.rot_j[rk] = rot;
  set_shift(T, rk, T.inc_j[rk], rot);
}

// ---------------------------------------------------------------------------
// ring sums
constexpr int ST = 256, SWARPS = ST / 32;    // threads and warps of this file's CTAs

// the tree of a block whose thread (w, L) holds v[q] = list[L + 32 (w + 8 q)];
// thread 0 has the sum.  red: 256 doubles of shared memory.
__device__ __forceinline__ double cta_tree1024(double (&v)[4], double *red) {
  red[threadIdx.x] = (v[0] + v[2]) + (v[1] + v[3]);
  __syncthreads();
  double x = 0.0;
  if (threadIdx.x < 32) {
    double w[8];
#pragma unroll
    for (int m = 0; m < 8; m++) w[m] = red[threadIdx.x + 32 * m];
#pragma unroll
    for (int h = 4; h >= 1; h >>= 1) {
#pragma unroll
      for (int m = 0; m < h; m++) w[m] = w[m] + w[m + h];
    }
    x = w[0];
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) {
      const double y = __shfl_down_sync(0xffffffffu, x, d);
      if ((int)threadIdx.x < d) x = x + y;
    }
  }
  __syncthreads();
  return x;
}

// What a ring's sum needs of the planet (modes 8 and 9)
struct RingForce {
  double m, x, y, ix2, b2, cy, sy, exclude2;
  __device__ __forceinline__ RingForce(const Body &b, double exclude) {
    m = b.m; x = b.x; y = b.y;
    ix2 = 1.0 / (b.x * b.x);
    b2 = fma(b.x, b.x, b.rs * b.rs);
    sincos(b.y, &sy, &cy);
    exclude2 = exclude * exclude;
  }
};

// output_lv1 of ring rt (ring i of layer k), rotated by rot: mode 0 mass, 8
// radial force, 9 torque of the disk on the planet (2D).  The CTA's work;
// thread 0 has the sum.
template <class RT>
__device__ __forceinline__ double ring_sum(const Tables &T, const RT *R, int rt, int rot, int mode, int ndim,
                                           const RingForce &F, double *red) {
  const int i = rt % T.nr, k = rt / T.nr, nphi = T.nphi;
  const int row = i + NPAD, rk = k * T.nrg + row;
  const size_t base = (size_t)rk * nphi;
  const double rad = T.rxc[row], xvol = T.rxvol[row], zvol = ndim == 3 ? T.zvol[k + NPAD] : 1.0;
  const double bs = sizeof(RT) == 4 ? T.sbg[rk] : 0.0;
  const bool force = mode != 0;
  const double r0 = T.rpa[row], dx = rad - F.x, bq = fma(rad, rad, F.b2);
  double val = 0.0;
#pragma unroll 1
  for (int l = 0; l < nphi; l += 1024) {
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int j = l + threadIdx.x + ST * q;    // storage index
      double x = 0.0;
      if (j < nphi) {
        const int j0 = wrap1(j + rot, nphi);
        const double r = load_r(R[base + j0], bs), yv = T.yvol[j0];
        if (!force) {
          x = r * xvol * yv * zvol;
        } else {
          const double d = T.yc[j0] - F.y;
          if (fma(dx, dx, rad * rad * (d * d)) > F.exclude2) {
            const double cy = T.cyc[j0], sy = T.syc[j0];
            const double c = fma(cy, F.cy, sy * F.sy), s = fma(sy, F.cy, -(cy * F.sy));
            const double y = rsq(fma(-2.0 * F.x * rad, c, bq)), y3 = y * y * y;
            const double w = (r - r0) * xvol * yv;
            if (mode == 8) x = F.m * fma(rad - F.x * c, y3, c * F.ix2) * w;
            else x = F.m * s * fma(F.x, y3, -F.ix2) * rad * w;
          }
        }
      }
      v[q] = x;
    }
    val += cta_tree1024(v, red);
  }
  return val;
}

// output_lv2 (3D: round_reduc_sum over k per ring, reduction.cu:77-100) and
// output_lv3 over the rings in blocks of 1024 (the reference supports one),
// by the CTA; thread 0 has the sum.
__device__ __forceinline__ double ring_total(const Tables &T, const volatile double *part, int ndim, double *red) {
  const int nr = T.nr, nk = T.nk;
  double total = 0.0;
  for (int b = 0; b < nr; b += 1024) {
    double v[4];
#pragma unroll
    for (int q4 = 0; q4 < 4; q4++) {
      const int ii = b + threadIdx.x + ST * q4;
      v[q4] = 0.0;
      if (ii < nr) {
        if (ndim == 3) {
          double acc[64];
          const int kk = nk < 64 ? nk : 64;
          for (int q = 0; q < kk; q++) acc[q] = part[ii + nr * q];
          int len = 1;
          while (len < nk) len *= 2;
          while (len > 1) {
            const int half = len / 2;
            for (int q = 0; q < half; q++) if (q + half < kk) acc[q] += acc[q + half];
            len = half;
          }
          v[q4] = acc[0];
        } else {
          v[q4] = part[ii];
        }
      }
    }
    total += cta_tree1024(v, red);
  }
  return 0.0 + total;
}

// true in every thread of the last of nb CTAs to come here
__device__ __forceinline__ bool last_cta(unsigned *counter, unsigned nb) {
  __shared__ bool is_last;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    is_last = atomicAdd(counter, 1u) == nb - 1;
    if (is_last) *counter = 0u;
  }
  __syncthreads();
  if (is_last) __threadfence();
  return is_last;
}

template <class RT>
__global__ void __launch_bounds__(ST) k_reduce(Tables T, const RT *R, Body pl, double exclude, int mode, int plnt,
                                               int ndim, double *part, unsigned *counter, double *out) {
  after_previous();
  __shared__ double red[ST];
  const bool zero = mode != 0 && plnt && ndim != 2;     // the reference's force sums are 2D
  const RingForce F(pl, exclude);
  for (int rt = blockIdx.x; rt < T.nr * T.nk; rt += gridDim.x) {
    const int rk = rt / T.nr * T.nrg + rt % T.nr + NPAD;
    const double x = zero ? 0.0 : ring_sum<RT>(T, R, rt, T.rot_j[rk], plnt ? mode : 0, ndim, F, red);
    if (threadIdx.x == 0) part[rt] = x;
  }
  if (!last_cta(counter, gridDim.x)) return;
  const double x = ring_total(T, part, ndim, red);
  if (threadIdx.x == 0) *out = x;
}

// ---------------------------------------------------------------------------
// planet (planet.cu:28-93), device copies of the host arithmetic
__device__ double d_set_M_p(const DevClock &c, double t) {
  if (t < c.t_growth) return fmax(c.M_p * sin(3.1415926535897932384626433832795 * t / (2.0 * c.t_growth)), 0.01 * 0.000003);
  return c.M_p;
}
__device__ void d_kick(Body &pl, double &FrRot, double dt, int frflag) {
  pl.vx += dt * pl.fx;
  // without a force (fixed planet) the quotients are the same zero
  pl.vy += FrRot + (pl.fy == 0.0 && pl.x > 0.0 ? dt * pl.fy : dt * pl.fy / pl.x / pl.x);
  FrRot = (frflag == 1) ? pl.vy : 0.0;
  pl.vy -= FrRot;
}
// The planet's arithmetic is host code in the reference (planet.cu), whose
// compiler folds pow with the constant exponents 0, 1, -1 and 2 into 1, x,
// 1/x and x*x; the device copies below use the same forms (other exponents
// stay pow calls).
__device__ __forceinline__ double pow_host_form(double x, double y) {
  if (y == 0.0) return 1.0;
  if (y == 1.0) return x;
  if (y == -1.0) return 1.0 / x;
  if (y == 2.0) return x * x;
  return pow(x, y);
}
// moving planet: the drift moves x, and the softening follows it as
// kick_drift_kick does on the host, rs = rs_fac h(x), h = sqrt(cs2(x) x^3)
// with cs2 = sc_h^2 x^-p_beta (disk_profile.cu:39-52)
__device__ void d_drift_moving(Body &pl, double FrRot, double dt, const DevClock &c) {
  double old_rad = pl.x;
  pl.x += dt * pl.vx;
  pl.y += dt * pl.vy;
  pl.vy = ((pl.vy + FrRot) * old_rad * old_rad / pl.x / pl.x) - FrRot;
  if (pl.y < 0.0) pl.y += 6.283185307179586476925286766559;
  if (pl.y >= 6.283185307179586476925286766559) pl.y -= 6.283185307179586476925286766559;
  pl.rs = c.rs_fac * sqrt(c.sc2 * pow_host_form(pl.x, -c.p_beta) * pl.x * pl.x * pl.x);
}

// ---------------------------------------------------------------------------
// The scalar parts of a step, on a CTA's copy of the clock: its end
// (main.cu:378-412) with a moving planet, in two parts around the disk's force
// sums (planet.cu:54-93); with a fixed one see step_scalars.
__device__ __forceinline__ void step_time(DevClock &c) {
  c.simtime += c.dt_step;
  c.timem += c.dt_step;
  c.ncycle += 1;
  c.ncycp += 1;
}
__device__ __forceinline__ void step_books(DevClock &c) {
  if (c.ncycp == c.nprin) { c.ncycp = 0; c.prin = 1; }
  if (c.make_pict) {
    c.timem = 0.0;
    c.make_pict = 0;
    c.dt = c.old_dt;
    c.halted = 1;   // the host dumps before continuing
  }
  if (c.done) c.halted = 1;
}

// a diagnostics row (main.cu:414-428) of the finished step's planet and time
__device__ __forceinline__ void record_row(DevClock &c, const Body &p, double frrot, double simtime) {
  if (!c.hist || c.hist_count >= c.hist_cap) return;
  double *h = c.hist + (size_t)HIST_COLS * c.hist_count;
  const double vy = p.vy + frrot;
  const double L = vy * p.x * p.x;                                        // get_L planet.cu:11-15
  const double E = (p.vx * p.vx + vy * vy * p.x * p.x) / 2.0 - 1.0 / p.x; // get_E planet.cu:17-21
  h[0] = simtime;
  h[1] = c.mass;
  h[2] = c.torque / c.hist_norm;
  h[3] = p.x; h[4] = p.y; h[5] = p.vx; h[6] = p.vy; h[7] = p.fx; h[8] = p.fy;
  h[9] = sqrt(1.0 + (2.0 * E * L * L));
  h[10] = -1.0 / (2.0 * E);
  c.hist_count += 1;
}

constexpr int CLK_WORDS = sizeof(DevClock) / 8;
static_assert(sizeof(DevClock) % 8 == 0 && CLK_WORDS <= ST, "the clock is copied by words");
struct StepShm {
  DevClock c;
  Body planet;            // of the finished step, for its sums and history row
  double frrot, simtime, frrot_pre;
  int print, run;
  double red[ST];
};
__device__ __forceinline__ void clock_in(StepShm &S, const DevClock *clk) {
  if (threadIdx.x < CLK_WORDS)
    reinterpret_cast<unsigned long long *>(&S.c)[threadIdx.x] = reinterpret_cast<const unsigned long long *>(clk)[threadIdx.x];
  __syncthreads();
}
__device__ __forceinline__ void clock_out(StepShm &S, DevClock *clk) {
  __syncthreads();
  if (threadIdx.x < CLK_WORDS)
    reinterpret_cast<unsigned long long *>(clk)[threadIdx.x] = reinterpret_cast<const unsigned long long *>(&S.c)[threadIdx.x];
}

// drift's new place of the planet (planet.cu:54-60)
__device__ __forceinline__ double drift_y(const Body &p, double dt) {
  double y = p.y + dt * p.vy;
  if (y < 0.0) y += 6.283185307179586476925286766559;
  if (y >= 6.283185307179586476925286766559) y -= 6.283185307179586476925286766559;
  return y;
}
// The end of a step with a fixed planet (post; main.cu:378-412: time, drift,
// forces, kick, books) and the start of the next (BETWEEN_PRE; get_dt's host
// part, the dt clipping and the half kick, main.cu:345-370), by a whole warp:
// the divisions that do not wait for one another are done side by side, a lane
// each, so that the chain has four of them one after another instead of
// seventeen at some 200 cycles each.  The planet's cos and sin come from
// another warp.  Every operation is the scalar code's, so are the bits.
__device__ __forceinline__ void step_scalars(StepShm &S, int fl, bool post) {
  DevClock &c = S.c;
  const int lane = threadIdx.x & 31;
  const bool pln = c.plnt_flag > 0;
  const double ds = c.dt_step, courant = c.courant, endtime = c.endtime, tmovie = c.tmovie;
  Body p = c.planet;
  double fr = c.frrot, simtime = c.simtime, timem = c.timem, cdt = c.dt, old_dt = c.old_dt;
  long long ncycle = c.ncycle, ncycp = c.ncycp;
  int prin = c.prin, make_pict = c.make_pict, done = c.done, halted = c.halted, status = c.status;
  double x1 = p.x, y1 = p.y;
  if (post) {
    simtime += ds;
    timem += ds;
    ncycle += 1;
    ncycp += 1;
    if (pln) {
      x1 = p.x + ds * p.vx;
      y1 = drift_y(p, ds);
      p.m = d_set_M_p(c, simtime);
    }
  }
  double n = 1.0, d1 = 1.0, d2 = 1.0;
  if (lane == 0) { n = (p.vy + fr) * p.x * p.x; d1 = d2 = x1; }             // drift's v_phi
  if (lane == 1) { n = -1.0; d1 = d2 = x1; }                                // the star's pull
  if (lane == 2) { n = courant; d1 = __longlong_as_double((long long)c.cfl_bits); }   // dt_lv3 timestep.cu:105
  if (lane == 3) d1 = x1 * x1;
  if (lane == 4 && c.ndim == 3) d1 = 1.0 + p.m;
  double q = n / d1 / d2;
  const double hdt = __shfl_sync(0xffffffffu, q, 2), ix2 = __shfl_sync(0xffffffffu, q, 3), stm = __shfl_sync(0xffffffffu, q, 4);
  {
    const double v = __shfl_sync(0xffffffffu, q, 0), g = __shfl_sync(0xffffffffu, q, 1);
    if (post && pln) {
      p.x = x1;
      p.y = y1;
      p.vy = v - fr;
      p.fx = g + p.x * pow_host_form(p.vy + fr, 2.0);
      p.fy = 0.0;
      d_kick(p, fr, 0.5 * ds, c.frrot_flag);
    }
  }
  if (post) {                              // step_books
    if (ncycp == c.nprin) { ncycp = 0; prin = 1; }
    if (make_pict) {
      timem = 0.0;
      make_pict = 0;
      cdt = old_dt;
      halted = 1;
    }
    if (done) halted = 1;
  }
  const bool print = (fl & BETWEEN_DIAG) && prin;
  if (print) prin = 0;
  if (print && lane == 0) {
    S.planet = p;
    S.frrot = fr;
    S.simtime = simtime;
  }
  bool run = (fl & BETWEEN_PRE) && !halted && !done;
  if (run && status != 0) {
    halted = 1;
    run = false;
  }
  double dt = 1.1 * cdt;                   // timestep.cu:135-141
  dt = (hdt < dt) ? hdt : dt;
  const double dt0 = dt;
  bool last = false, out = false;
  if (ncycle == c.ncycend) last = true;
  double od = old_dt;
  bool end = false, pict = false;
  if (simtime + dt >= endtime) { od = dt; dt = endtime - simtime; end = pict = true; }
  if (timem + dt >= tmovie) { od = dt; dt = tmovie - timem; pict = true; }
  out = last || end;
  // kick_drift_kick(planet, FrRot, ..., 0.5*dt, true) main.cu:370
  Body k = p;
  double fk = fr;
  if (pln) d_kick(k, fk, 0.5 * dt, c.frrot_flag);
  // FrRot at the next get_dt, for the fused CFL: drift and kick replayed on
  // copies (fixed planet: its forces are analytic and leave v_phi alone)
  n = 1.0; d1 = 1.0; d2 = 1.0;
  if (lane == 0) { n = (k.vy + fk) * k.x * k.x; d1 = d2 = k.x + dt * k.vx; }
  if (lane == 1) { n = dt0; d1 = endtime; }
  q = n / d1 / d2;
  double frn = fk;
  {
    const double v = __shfl_sync(0xffffffffu, q, 0), rel = __shfl_sync(0xffffffffu, q, 1);
    if (pln) frn = c.frrot_flag == 1 ? (v - fk) + (fk + 0.0) : 0.0;
    if (run && (rel < 1.0e-12 || !(dt0 > 0.0))) {
      status = 4;
      halted = 1;
      run = false;
    }
  }
  if (lane == 0) {
    c.simtime = simtime;
    c.timem = timem;
    c.ncycle = ncycle;
    c.ncycp = ncycp;
    c.halted = halted;
    c.status = status;
    S.print = print;
    S.run = run;
    if (run) {
      S.frrot_pre = fr;                    // as Index_Shift sees it
      c.prin = out;
      if (out) done = 1;
      if (pict) make_pict = 1;
      c.old_dt = od;
      c.dt = c.dt_step = dt;
      c.planet = k;
      c.frrot = fk;
      c.frrot_next = frn;
      c.cfl_bits = 0ull;
      PlanetC &e = c.pc;                   // planet_consts; cy, sy: between_body
      e.m = k.m * stm;
      e.x = k.x;
      e.ix2 = ix2;
      e.b2 = fma(k.x, k.x, k.rs * k.rs);
      e.star = pln ? stm : 1.0;
      e.y = k.y;
      e.vy = k.vy;
      e.turn = c.ndim == 3 ? turn_of(dt, 0.0, 0.0, k.vy) : make_double2(1.0, 0.0);
    } else {
      c.prin = prin;
      c.dt = cdt;
      c.planet = p;
      c.frrot = fr;
    }
    c.done = done;
    c.make_pict = make_pict;
  }
}

// CTA b of a run's nb.  fl: BETWEEN_POST the end of a step with a fixed planet,
// BETWEEN_DIAG its diagnostics, BETWEEN_PRE the start of the next.
template <class RT>
__device__ __forceinline__ void between_body(StepShm &S, const Tables &T, const RT *R, DevClock *clk, double *part,
                                             unsigned *counter, int fargo, int torque, int ndim, int fl, int b,
                                             int nb) {
  const int rings = T.nr * T.nk, tid = threadIdx.x;
  clock_in(S, clk);
  const bool off = S.c.halted && !(fl & BETWEEN_DIAG && S.c.prin);
  if (off) return;                       // every CTA of the run alike
  const bool post = (fl & BETWEEN_POST) && !S.c.halted;
  const double py = post && S.c.plnt_flag > 0 ? drift_y(S.c.planet, S.c.dt_step) : S.c.planet.y;
  double sy = 0.0, cy = 1.0;
  __syncthreads();
  if (tid < 32) step_scalars(S, fl, post);
  else if (tid == 32) sincos(py, &sy, &cy);
  __syncthreads();
  if (tid == 32 && S.run) {
    S.c.pc.sy = sy;
    S.c.pc.cy = cy;
  }
  if (S.print) {
    const RingForce F(S.planet, 0.0);
    for (int rt = b; rt < rings; rt += nb) {
      const int rk = rt / T.nr * T.nrg + rt % T.nr + NPAD, rot = post ? rotated(T, rk) : T.rot_j[rk];
      const double m = ring_sum<RT>(T, R, rt, rot, 0, ndim, F, S.red);
      const double t = torque ? ring_sum<RT>(T, R, rt, rot, 9, ndim, F, S.red) : 0.0;
      if (tid == 0) {
        part[rt] = m;
        part[rings + rt] = t;
      }
    }
  }
  // a thread per ring; in a step that sums the CTA's own rings, which it alone
  // has read
  const int first = S.print ? b + tid * nb : b * ST + tid, by = nb * ST;
  for (int rt = first; rt < rings; rt += by) {
    const int rk = rt / T.nr * T.nrg + rt % T.nr + NPAD;
    if (post) T.rot_j[rk] = rotated(T, rk);
    if (S.run) {
      index_shift_ring(T, rt, S.c.dt_step, S.frrot_pre, fargo);
      finish_ring(T, rt, S.c.dt_step, S.c.frrot_next, S.c.planet.vy, ndim);
    }
  }
  if (nb > 1 && !last_cta(counter, nb)) return;
  __syncthreads();
  if (S.print) {
    const double m = ring_total(T, part, ndim, S.red);
    const double t = torque ? ring_total(T, part + rings, ndim, S.red) : 0.0;
    if (tid == 0) {
      S.c.mass = m;
      if (torque) S.c.torque = t;
      record_row(S.c, S.planet, S.frrot, S.simtime);
    }
  }
  clock_out(S, clk);
}

template <class RT>
__global__ void __launch_bounds__(ST) k_between(Tables T, const RT *R, DevClock *clk, double *part, unsigned *counter,
                                                int fargo, int torque, int ndim, int fl) {
  after_previous();
  __shared__ StepShm S;
  between_body<RT>(S, T, R, clk, part, counter, fargo, torque, ndim, fl, blockIdx.x, gridDim.x);
}

// members' CTAs by the queue's prefix sums
template <class RT>
__global__ void __launch_bounds__(ST) kb_between(BatchQueue q, int fl) {
  after_previous();
  __shared__ StepShm S;
  const int r = batch_find(q, blockIdx.x);
  const BatchRun &b = q.runs[r];
  const RT *R;
  if constexpr (sizeof(RT) == 4) R = (const RT *)b.QX.r;   // a 2D step ends in its first planes
  else R = (const RT *)b.PX.r;
  between_body<RT>(S, b.T, R, b.clk, b.ring_part, b.counter, b.fargo, b.plnt, 2, fl, blockIdx.x - q.start[r],
                   q.start[r + 1] - q.start[r]);
}

// moving planet: the step's end up to the kick
template <class RT>
__global__ void __launch_bounds__(ST) k_moving(Tables T, const RT *R, DevClock *clk, double *part, unsigned *counter,
                                               int ndim) {
  after_previous();
  __shared__ StepShm S;
  const int rings = T.nr * T.nk, tid = threadIdx.x;
  clock_in(S, clk);
  if (S.c.halted) return;
  __syncthreads();
  if (tid == 0) {
    step_time(S.c);
    d_drift_moving(S.c.planet, S.c.frrot, S.c.dt_step, S.c);
    S.c.planet.m = d_set_M_p(S.c, S.c.simtime);
  }
  __syncthreads();
  const RingForce F(S.c.planet, 0.0);
  for (int rt = blockIdx.x; rt < rings; rt += gridDim.x) {
    const int rk = rt / T.nr * T.nrg + rt % T.nr + NPAD, rot = rotated(T, rk);
    const double f8 = ndim == 2 ? ring_sum<RT>(T, R, rt, rot, 8, ndim, F, S.red) : 0.0;
    const double f9 = ndim == 2 ? ring_sum<RT>(T, R, rt, rot, 9, ndim, F, S.red) : 0.0;
    if (tid == 0) {
      part[rt] = f8;
      part[rings + rt] = f9;
      T.rot_j[rk] = rot;
    }
  }
  if (!last_cta(counter, gridDim.x)) return;
  const double f8 = ring_total(T, part, ndim, S.red), f9 = ring_total(T, part + rings, ndim, S.red);
  if (tid == 0) {
    // planet_forces planet.cu:58-59 with the disk sums of this state
    DevClock &c = S.c;
    Body &p = c.planet;
    c.f8 = f8;
    c.f9 = f9;
    p.fx = c.Sigma_0 * f8 / p.m - 1.0 / p.x / p.x + p.x * pow_host_form(p.vy + c.frrot, 2.0);
    p.fy = c.Sigma_0 * f9 / p.m;
    d_kick(p, c.frrot, 0.5 * c.dt_step, c.frrot_flag);
    c.frrot_next = c.frrot;      // the CFL of the next get_dt runs after this kernel
    step_books(c);
  }
  clock_out(S, clk);
}

}  // namespace pgd

namespace pgk {
using namespace pgd;

// A CTA per ring up to four per SM of a B200, then each several: for the sums of
// k_reduce and k_moving, and between steps, where a step that prints sums (one
// in nprin) and one that does not takes as long with 16 CTAs as with 592.  With
// a CTA per 8 rings, at most 148, and Index_Shift by the thread that stored the
// sum, a printing step took, us: 128x384 54.6, now 35.1; 1536x4608 895, 776;
// 128x1024x32 1019, 943 (without printing 30, 655 and 893 both ways).  k_reduce
// with at most 296 and 1184 CTAs instead of 592: 1536x4608 torque 76 and 54 us
// for 52.
static int ring_ctas(int rings) { return rings < 592 ? rings : 592; }
// of a batch member, whose fellows fill the GPU
int between_ctas(int rings) {
  const int n = (rings + SWARPS - 1) / SWARPS;
  return n < 148 ? n : 148;
}

void index_shift(const Tables &T, double dt, double frrot, int fargo, cudaStream_t s) {
  launch(k_index, (T.nr * T.nk + 127) / 128, 128, 0, s, T, dt, frrot, fargo);
}
void rotate(const Tables &T, cudaStream_t s) { launch(k_rotate, (T.nr * T.nk + 127) / 128, 128, 0, s, T); }

template <class RT>
void reduce(const Tables &T, const RT *r, const Body &pl, double exclude, int mode, int plnt, int ndim,
            double *part, unsigned *counter, double *out, cudaStream_t s) {
  launch(k_reduce<RT>, ring_ctas(T.nr * T.nk), ST, 0, s, T, r, pl, exclude, mode, plnt, ndim, part, counter, out);
}
template <class RT>
void between(const Tables &T, const RT *r, DevClock *clk, double *part, unsigned *counter, int fargo,
             int plnt, int ndim, int fl, cudaStream_t s) {
  launch(k_between<RT>, ring_ctas(T.nr * T.nk), ST, 0, s, T, r, clk, part, counter, fargo, plnt && ndim == 2, ndim, fl);
}
template <class RT>
void moving(const Tables &T, const RT *r, DevClock *clk, double *part, unsigned *counter, int ndim,
            cudaStream_t s) {
  launch(k_moving<RT>, ring_ctas(T.nr * T.nk), ST, 0, s, T, r, clk, part, counter, ndim);
}
template <class RT>
void batch_between(const BatchQueue &q, int fl, cudaStream_t s) {
  if (q.total > 0) launch(kb_between<RT>, q.total, ST, 0, s, q, fl);
}
#define PG_STEP(RT)                                                                                                      \
  template void reduce<RT>(const Tables &, const RT *, const Body &, double, int, int, int, double *, unsigned *, \
                           double *, cudaStream_t);                                                                      \
  template void between<RT>(const Tables &, const RT *, DevClock *, double *, unsigned *, int, int, int, int,    \
                            cudaStream_t);                                                                               \
  template void moving<RT>(const Tables &, const RT *, DevClock *, double *, unsigned *, int, cudaStream_t);     \
  template void batch_between<RT>(const BatchQueue &, int, cudaStream_t);
PG_STEP(double)
PG_STEP(float)

}  // namespace pgk
