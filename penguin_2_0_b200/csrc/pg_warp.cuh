// pg_warp.cuh -- the ppmlr chain (ppmlr.cu:2-56) of one pencil chunk as one
// warp's work.
//
// A chunk is 116 interior cells and 6 ghost cells on each side (n_pad 6,
// arrsize 128 of variable_types.h:13-16).  A lane owns C neighbouring cells
// (C = 4: 32 lanes hold a full chunk); a shorter chunk takes G = ceil(lim / C)
// lanes and several pencils share a warp.  A stage works on a lane's cells in
// registers and reads the neighbours at their two ends by one shuffle per
// value; between stages the fields rest in the warp's slots of shared memory
// (each lane on its own cells, so without bank conflicts or barriers).
//
// What bounds it: instruction issue.  The sweeps read and write each field once
// (DRAM far from its limit).  Measured with 16 warps per SM: an FP64
// instruction keeps a scheduler from issuing for two cycles, any other for one
// (32 DFMA take 64 cycles, with 32 LOP3 between them 97), and with that the
// sweeps run at 78-85 % of what their instructions allow.  So what counts is
// the number of instructions per cell, FP64 ones twice, and that they come from
// the SM's instruction cache: straight-line code of more than 2048 instructions
// (32 KB) was measured to issue at 1.2-1.9 instructions per cycle and SM
// against 3.85 below that, whatever the number of warps, and the chain with
// every stage unrolled over 4 cells and all fields is 4700 instructions long.
// So the stages that repeat per field (edges, fluxes) are loops over fields.
// The faces (forces, Riemann problem) as a loop over pairs of cells as well were
// 3 % slower: the moves that it takes cost more than the shorter code gains.
// The number of operations is kept down by
//   * edge values as differences from the cell value (edges below): the
//     monotonicity rules of parabola.cu:70-133 become comparisons of the two
//     half jumps, and the interface value itself is never formed;
//   * no parabola of p in an isothermal azimuthal sweep: p = cs2 rho with one
//     cs2 per ring, and the parabola's rules commute with a constant factor;
//   * a Riemann solution that needs log(p_r / p_l) and exp(t) of small
//     arguments only (series below; other arguments take log and exp);
//   * the planet's angle at every cell by angle addition from one cosine and
//     sine per pencil or per azimuth cell;
//   * grid-only factors (paraset's coefficients, the viscosity's difference
//     weights, reciprocal widths and volumes) from per-axis tables;
//   * reciprocals and square roots as one third-order step on the hardware's
//     approximations (rcp, rsq below).
// Times against the chain of one thread per cell that it replaced are with
// the sweep kernels in pg_sweep.cu.
//
// Index ranges, update rules and the order of the physical steps are the
// reference's (cited beside each stage).  Differences that leave results to
// rounding:
//  * chunks of a pencil are independent warps reading the pre-sweep state
//    from a separate buffer (ppm.cu:43-157 carries pre-update values, so the
//    result is the same Jacobi update);
//  * the q remap (remap.cu:123-142) and the q of evolve (evolve.cu:131-135)
//    are skipped: the store derives p from the EOS relation (ppm.cu:138-143).
// Cells outside a stage's range hold values that no cell inside uses.
//
// This file is compiled without contraction (-fmad=false): fused operations
// are written out, so a cell's bits do not depend on the kernel around it.
#pragma once
#include "pg_kernels.cuh"

namespace pgd {

// Series coefficients as operands from the constant bank: as immediates each
// takes two moves before its use.
__constant__ double kSin[4] = {1.0 / 362880.0, -1.0 / 5040.0, 1.0 / 120.0, -1.0 / 6.0};
__constant__ double kCos[3] = {1.0 / 40320.0, -1.0 / 720.0, 1.0 / 24.0};
__constant__ double kLog[8] = {1.0 / 17.0, 1.0 / 15.0, 1.0 / 13.0, 1.0 / 11.0, 1.0 / 9.0, 1.0 / 7.0, 1.0 / 5.0, 1.0 / 3.0};
__constant__ double kExp[8] = {1.0 / 3628800.0, 1.0 / 362880.0, 1.0 / 40320.0, 1.0 / 5040.0,
                               1.0 / 720.0,     1.0 / 120.0,    1.0 / 24.0,    1.0 / 6.0};

// 1 / b: PTX's rcp.approx.ftz.f64 (relative error 2^-20 or less) and one
// third-order Newton step (Householder), y (1 + e + e^2) with e = 1 - b y:
// the error of the step is e^3 < 2^-60.  Zero, subnormal and infinite b give
// a NaN, which the sweeps' finiteness check reports.
__device__ __forceinline__ double rcp(double b) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  const double e = fma(-b, y, 1.0);
  return fma(y, fma(e, e, e), y);
}
// 1 / sqrt(x), x > 0 and normal: rsqrt.approx.ftz.f64 and one third-order
// step of the same kind (Householder), y (1 + e/2 + 3 e^2/8) with e = 1 - x y^2
__device__ __forceinline__ double rsq(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-(x * y), y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}
// sqrt(x) by rsq where x is positive and normal, else (zero, as where a dump holds
// no pressure) by CUDA's, out of line
static __device__ __noinline__ double sqrt_call(double x) { return sqrt(x); }
__device__ __forceinline__ double root(double x) {
  return (unsigned)(__double2hiint(x) - 0x00100000) < 0x7fe00000u ? x * rsq(x) : sqrt_call(x);
}

// a / b from ib = 1 / b to rounding: the quotient corrected by its remainder
// (Markstein).  Where the same b divides step after step (a cell's volume, a
// ring's radius), a product with the rounded reciprocal would drift: its error
// has the same sign each time.
__device__ __forceinline__ double quot(double a, double b, double ib) {
  const double q = a * ib;
  return fma(fma(-q, b, a), ib, q);
}

// sin(x) and cos(x) for the small angles of a step (fractions of a cell).
// Taylor to x^9 and x^8: for |x| <= 0.05 the first omitted terms are below 1e-19
// of sin's x and of cos's 1.  Larger angles take sincos, but not those of the
// cells that pad a pencil to whole lanes of three (live): any value will do
// there, and one of them sent its whole warp the long way (polar sweep of the
// 128x1024x32 disk 436 -> 423 us).  With four cells per lane the check costs
// what it saves: 1 % more at 24 and 16 layers, 1 % less at 14.
static __device__ __noinline__ double2 sincos_call(double x) {
  double s, c;
  sincos(x, &s, &c);
  return make_double2(s, c);
}
// |x| above 0.05, by the high word: 0.05 less 4e-8 at the least
__device__ __forceinline__ bool wide(double x) { return (__double2hiint(x) & 0x7fffffff) >= 0x3fa99999; }
__device__ __forceinline__ void sincos_near(double x, double &s, double &c, bool live = true) {
  const double z = x * x;
  s = fma(x * z, fma(z, fma(z, fma(z, kSin[0], kSin[1]), kSin[2]), kSin[3]), x);
  c = fma(z, fma(z, fma(z, fma(z, kCos[0], kCos[1]), kCos[2]), -0.5), 1.0);
  if (wide(x) && live) {
    const double2 t = sincos_call(x);
    s = t.x;
    c = t.y;
  }
}

// sin(x) / x of such an angle
__device__ __forceinline__ double sinc_near(double x, bool live) {
  if (wide(x) && live) return sincos_call(x).x / x;
  const double z = x * x;
  return fma(z, fma(z, fma(z, fma(z, kSin[0], kSin[1]), kSin[2]), kSin[3]), 1.0);
}
static __device__ __noinline__ double pow_call(double x, double y) { return pow(x, y); }

// Arrays of an axis table (Tables::ax): chunk l of the axis holds A_COUNT
// arrays of ARR entries, one per cell of the chunk (ghost cells included), the
// lane's C cells placed so that a warp reads whole lines (k_axis_table).
enum AxisEntry {
  A_XF,                                  // left face coordinate (azimuth: unwrapped)
  A_IW,                                  // 1 / width
  A_C0, A_C1, A_C2, A_C3, A_C4,          // Eulerian paraset coefficients (parabola.cu:138-176)
  A_VA, A_VB, A_VC, A_VD,                // derivs' weights: first = VA D+ + VB D-, second = VC D+ - VD D-
  A_VOL, A_IVOL, A_XC,                   // cell volume along the axis, its reciprocal, cell centre
  A_E0, A_E1, A_E2, A_E3, A_E4, A_E5,    // radial: 1/face, 1/centre; azimuth: cos, sin of face and centre;
  A_COUNT                                // polar: sin, cos of face and centre, 1/sin of face and centre
};

#define PG_CELLS _Pragma("unroll") for (int c = 0; c < C; c++)

__device__ __forceinline__ double from_left(double x) { return __shfl_up_sync(0xffffffffu, x, 1); }
__device__ __forceinline__ double from_right(double x) { return __shfl_down_sync(0xffffffffu, x, 1); }

// o[n] = a[n - 1], o[n] = a[n + 1]
template <int C>
__device__ __forceinline__ void left_of(const double (&a)[C], double (&o)[C]) {
  const double l = from_left(a[C - 1]);
  PG_CELLS o[c] = c ? a[c > 0 ? c - 1 : 0] : l;
}
template <int C>
__device__ __forceinline__ void right_of(const double (&a)[C], double (&o)[C]) {
  const double r = from_right(a[0]);
  PG_CELLS o[c] = c < C - 1 ? a[c < C - 1 ? c + 1 : 0] : r;
}

// cos and sin of the planet's angle's change against a ring in half a step
// (res_v and 1/r_cyl of the ring)
__device__ __forceinline__ double2 turn_of(double dt, double res, double irc, double vy) {
  double2 t;
  sincos_near(0.5 * dt * (res * irc - vy), t.y, t.x);
  return t;
}
static __device__ __noinline__ double2 turn_call(double dt, double res, double irc, double vy) {
  return turn_of(dt, res, irc, vy);
}

__device__ __forceinline__ PlanetC planet_consts(const Body &b, bool three, bool plnt, double dt) {
  PlanetC p;
  const double stm = three ? 1.0 / (1.0 + b.m) : 1.0;
  p.m = b.m * stm;
  p.x = b.x;
  p.ix2 = 1.0 / (b.x * b.x);
  p.b2 = fma(b.x, b.x, b.rs * b.rs);
  p.star = plnt ? stm : 1.0;
  p.y = b.y;
  p.vy = b.vy;
  sincos(b.y, &p.sy, &p.cy);
  p.turn = three ? turn_of(dt, 0.0, 0.0, b.vy) : make_double2(1.0, 0.0);
  return p;
}

// Slots of a warp's workspace: one double per cell of each lane.
enum Slot {
  W_R, W_U, W_V, W_W,                    // density, sweep velocity, transverse slots
  W_SLR, W_SRR,                          // density left and right of each cell's left face
  W_OMF,                                 // 1 - flat, where a cell of the warp is flattened
  W_SLP, W_SRP,                          // pressure left and right of each cell's left face
  W_COUNT,
  W_P = W_SLP                            // the pressure, until its states take the slot
};
// Place of cell c of a lane in a slot, from the lane's own base (ws_lane):
// pairs of cells (C = 4) or single cells (C = 3) of all lanes side by side,
// PIECE apart.  Pieces, slots and warps are padded so that a tile's loads
// and stores (neighbouring threads on neighbouring columns, that is warps)
// fall in different banks.
constexpr int SLOT = 132;
constexpr int WS = W_COUNT * SLOT + 16;  // doubles of a warp's workspace: 4 mod 16
constexpr int WS_ISO_Y = W_SLP * SLOT;   // of an isothermal azimuthal sweep, which keeps no pressure
template <int C>
constexpr int PIECE = C == 4 ? 66 : 34;
template <int C>
__device__ __forceinline__ constexpr int ws_lane(int lane) { return C == 4 ? 2 * lane : lane; }

// What a lane knows of its pencil and its cells.
template <int C>
struct Lane {
  int n0, lim;              // first cell of the lane in the chunk, cells of the chunk
  const double *tab;        // axis table of the chunk at the lane's first cell
  int half;                 // distance of the lane's next piece (a pair of cells for C = 4, else one cell)
  double *ws;               // the warp's workspace at the lane's base
  const double *row;        // radial, polar: per-row values (RowEntry) at the lane's first cell, placed as the axis table's
  double dt, frrot;
  double c0, s0;            // radial, polar: cos and sin of phi - phi_planet at the step's start (radial: times sin theta)
  double ca, sa, cb, sb, cc, sc;   // azimuthal: rotations of the planet's angle at t, t + dt/2 and t + dt
  double rad, irad;         // azimuthal: cylindrical radius of the ring; polar: r of the ring
  double sp, isp2;          // radial: 1 / sin^2 theta; azimuthal: sin theta
  double bq;                // azimuthal, polar: r^2 + x_p^2 + rs^2
  double vr;                // azimuthal: res_v / r_cyl of the ring
  double cs2, ciso;         // azimuthal, isothermal: cs2 and its root, the high word above which
  int low;                  // both rho and cs2 rho are above 1e-14
  __device__ __forceinline__ int n(int c) const { return n0 + c; }
  // lo <= n < lim - hi
  __device__ __forceinline__ bool in(int c, int lo, int hi) const {
    return (unsigned)(n0 + c - lo) < (unsigned)(lim - hi - lo);
  }
};

template <int C>
__device__ __forceinline__ void get(const Lane<C> &L, int slot, double (&o)[C]) {
  const double *q = L.ws + slot * SLOT;
  if constexpr (C == 4) {
    const double2 x = *reinterpret_cast<const double2 *>(q), y = *reinterpret_cast<const double2 *>(q + PIECE<4>);
    o[0] = x.x; o[1] = x.y; o[2] = y.x; o[3] = y.y;
  } else {
    PG_CELLS o[c] = q[c * PIECE<C>];
  }
}
template <int C>
__device__ __forceinline__ void put(const Lane<C> &L, int slot, const double (&o)[C]) {
  double *q = L.ws + slot * SLOT;
  if constexpr (C == 4) {
    *reinterpret_cast<double2 *>(q) = make_double2(o[0], o[1]);
    *reinterpret_cast<double2 *>(q + PIECE<4>) = make_double2(o[2], o[3]);
  } else {
    PG_CELLS q[c * PIECE<C>] = o[c];
  }
}
// per-row values of a radial or polar tile (one ring of one layer per row)
enum RowEntry {
  R_SND, R_CH, R_SH, R_NU, R_RC, R_IRC,   // R_CH, R_SH: cos and sin of the planet's angle's change in dt/2
  R_COUNT
};
// the lane's entries of one array of the axis table, and of the per-row values
template <int C>
__device__ __forceinline__ void ld(const Lane<C> &L, int a, double (&o)[C]) {
  const double *q = L.tab + a * ARR;
  if constexpr (C == 4) {
    const double2 x = *reinterpret_cast<const double2 *>(q), y = *reinterpret_cast<const double2 *>(q + L.half);
    o[0] = x.x; o[1] = x.y; o[2] = y.x; o[3] = y.y;
  } else {
    PG_CELLS o[c] = q[c * L.half];
  }
}
template <int C>
__device__ __forceinline__ void ld_row(const Lane<C> &L, int a, double (&o)[C]) {
  const double *q = L.row + a * ARR;
  if constexpr (C == 4) {
    const double2 x = *reinterpret_cast<const double2 *>(q), y = *reinterpret_cast<const double2 *>(q + L.half);
    o[0] = x.x; o[1] = x.y; o[2] = y.x; o[3] = y.y;
  } else {
    PG_CELLS o[c] = q[c * L.half];
  }
}
template <int C>
struct ParC { double c0[C], c1[C], c2[C], c3[C], c4[C]; };

__device__ __forceinline__ bool opposite(double a, double b) { return (__double2hiint(a) ^ __double2hiint(b)) < 0; }
// 2 x by its exponent, or (zero) a number below 2^-1021 of either sign: as a
// bound for an edge difference as good as zero, at one integer operation
__device__ __forceinline__ double twice(double x, bool zero) {
  return __hiloint2double(zero ? 0 : __double2hiint(x) + 0x00100000, __double2loint(x));
}

// CW84 parabola of a field (parabola.cu:70-133): d1 = right edge - value and
// d2 = value - left edge after flattening and limiting.  Then the jump over
// the cell is d1 + d2 and a6 = 3 (d2 - d1).  parabola's rules in these terms:
// an extremum has d1 and d2 of opposite sign and takes both zero; u2 < u1 is
// |d2| > 2 |d1| and sets d2 = 2 d1; u2 < -u1 is |d1| > 2 |d2| and sets
// d1 = 2 d2.  flat: whether a cell of the warp is flattened (W_OMF is set).
// ODD: some ghost cells hold no state (NaN, or beyond 1e154), and the slopes beside
// them are parabola's by its own comparisons (min3 of simple_func.cu:1-14).
template <bool ODD, int C>
__device__ __forceinline__ void edges(const Lane<C> &L, const double (&a)[C], const ParC<C> &k, bool flat, double (&d1)[C],
                                      double (&d2)[C]) {
  double dr[C], dl[C], t[C], tr[C], s[C];
  right_of<C>(a, dr);
  PG_CELLS dr[c] = dr[c] - a[c];
  left_of<C>(dr, dl);
  PG_CELLS {
    const double x = fma(k.c3[c], dr[c], k.c4[c] * dl[c]);
    if (ODD) {
      const double l2 = 2.0 * fabs(dl[c]), r2 = 2.0 * fabs(dr[c]), q = fabs(x) < l2 ? fabs(x) : l2;
      t[c] = r2 < q ? r2 : q;
      t[c] = x < 0.0 ? -t[c] : t[c];
      if (dl[c] * dr[c] < 0.0) t[c] = 0.0;
    } else {
      double q = fabs(dl[c]) < fabs(dr[c]) ? fabs(dl[c]) : fabs(dr[c]);
      q = twice(q, opposite(dl[c], dr[c]));
      q = fabs(x) < q ? fabs(x) : q;
      t[c] = copysign(q, x);
    }
  }
  right_of<C>(t, tr);
  PG_CELLS s[c] = fma(k.c0[c], dr[c], fma(k.c1[c], tr[c], k.c2[c] * t[c]));
  left_of<C>(s, d2);
  PG_CELLS {
    d1[c] = s[c];
    d2[c] = dl[c] - d2[c];
  }
  if (flat) {
    double o[C];
    get<C>(L, W_OMF, o);
    PG_CELLS {
      d1[c] *= o[c];
      d2[c] *= o[c];
    }
  }
  PG_CELLS {
    const double x1 = d1[c], x2 = d2[c];
    if (ODD) {
      const double j = x1 + x2, jj = j * j, j6 = j * (3.0 * (x2 - x1));
      if (x1 * x2 <= 0.0) d1[c] = d2[c] = 0.0;
      if (jj < j6) d2[c] = 2.0 * d1[c];
      if (jj < -j6) d1[c] = 2.0 * d2[c];
      continue;
    }
    const bool ext = opposite(x1, x2);
    const double y1 = twice(x1, ext), y2 = twice(x2, ext);
    d1[c] = fabs(x1) > fabs(y2) ? y2 : x1;
    d2[c] = fabs(x2) > fabs(y1) ? y1 : x2;
  }
}

// Planet (and star) acceleration along the radius (forces.cu:185-264): radius
// x and 1/x, cf = cos(phi - phi_p) sin(theta), angular momentum v and w = r
// v_theta
template <bool THREED, bool ODD>
__device__ __forceinline__ double force_r(double x, double ix, double cf, double v, double w, const PlanetC &P, int plnt,
                                          double isp2) {
  double t = v * v;
  if (THREED) t = fma(w, w, t * isp2);
  // ODD: a ghost face at radius 0 has no force (inf - inf), as the reference's terms;
  // without a planet its 2D star pulls towards radius 0 from either side
  const double i2 = ODD && !THREED && !plnt ? ix * fabs(ix) : ix * ix;
  const double f = ODD ? t * (ix * ix * ix) - P.star * i2 : i2 * fma(ix, t, -P.star);
  if (!plnt) return f;
  const double xc = P.x * cf;
  const double y = rsq(fma(x, fma(-2.0, xc, x), P.b2));
  return f - P.m * fma(x - xc, y * y * y, cf * P.ix2);
}
// azimuthal (forces.cu:265-296): bq = r^2 + x_p^2 + rs^2, r cylindrical radius
__device__ __forceinline__ double force_phi(double rad, double bq, double sp, double cf, double sf, const PlanetC &P) {
  const double y = rsq(fma(-2.0 * P.x * rad, cf, bq));
  return P.m * sf * fma(sp, P.ix2, -(P.x * (y * y * y)));
}
// polar (forces.cu:298-372): sine and cosine of the angle, 1 / (r sin) and
// 1 / sin, angular momentum w
__device__ __forceinline__ double force_theta(double rad, double bq, double sp, double cp, double irc, double isp, double cf,
                                              double w, const PlanetC &P, int plnt) {
  const double f = w * w * cp * (irc * irc * irc);
  if (!plnt) return f;
  const double y = rsq(fma(-2.0 * P.x * rad * sp, cf, bq));
  return fma(P.m * cf * cp, fma(P.x, y * y * y, -(isp * P.ix2)), f);
}

// Isothermal Riemann problem (riemann.cu:45-53) in full, with the reference's
// bounds on p and rho: states outside the series' range below.
static __device__ __noinline__ double2 riemann_iso_call(double pl, double rl, double ul, double pr, double rr, double ur) {
  pl = pl > kSmallp ? pl : kSmallp;
  pr = pr > kSmallp ? pr : kSmallp;
  rl = rl > kSmallr ? rl : kSmallr;
  rr = rr > kSmallr ? rr : kSmallr;
  const double t1 = 0.5 * (sqrt(pl / rl) + sqrt(pr / rr));
  const double pm = sqrt(pl * pr) * exp(-0.5 * (ur - ul) / t1);
  return make_double2(0.5 * (ul + ur) - 0.5 * t1 * log(pr / pl), pm > kSmallp ? pm : kSmallp);
}
// The usual case.  With w = 2 t1, t1 the mean of sqrt(p/rho) of both sides:
// p* = sqrt(p_l p_r) exp(t), t = -(u_r - u_l) / w, and u* = u_l - t1 log(p*/p_l)
// = (u_l + u_r)/2 - t1 log(p_r/p_l)/2.  log(p_r/p_l) = 2 atanh(z),
// z = (p_r - p_l)/(p_r + p_l).  Series to z^17 and t^10 for |z|, |t| <= 1/8
// (omitted terms below 4e-18).  a, b: p or, where p = cs2 rho with the same
// cs2 on both sides, rho; s: sqrt(p_l p_r).  False outside the range.
__device__ __forceinline__ bool riemann_near(double a, double b, double s, double w, double ul, double ur, double &um,
                                             double &pm) {
  const double t = (ul - ur) * rcp(w);
  const double z = (b - a) * rcp(b + a), z2 = z * z;
  double q = fma(z2, kLog[0], kLog[1]);
#pragma unroll
  for (int i = 2; i < 8; i++) q = fma(z2, q, kLog[i]);
  double e = fma(t, kExp[0], kExp[1]);
#pragma unroll
  for (int i = 2; i < 8; i++) e = fma(t, e, kExp[i]);
  e = fma(t, e, 0.5);
  e = fma(t, e, 1.0);
  e = fma(t, e, 1.0);
  um = fma(-0.5 * w, fma(z * z2, q, z), 0.5 * (ul + ur));
  pm = s * e;
  return fabs(z) <= 0.125 && fabs(t) <= 0.125;
}
// a double's high word as an integer grows with it; kTiny: that of 1e-14, an
// order of magnitude above the bounds kSmallp and kSmallr
constexpr int kTiny = 0x3d06849b;
// x above kSmallr (by its high word: false from 1e-15 (1 + 1e-6) down, and for what is not finite)
__device__ __forceinline__ bool above_bound(double x) {
  return (unsigned)(__double2hiint(x) - 0x3cd203b0) < 0x7ff00000u - 0x3cd203b0u;
}

// Isentropic Riemann problem (riemann.cu:75-111): van Leer's (1979) Newton
// iteration for the contact pressure, at most 10 passes, relative tolerance
// 1e-8.  Out of line: one copy for the lane's cells.
static __device__ __noinline__ double2 riemann_isen(double pl, double rl, double ul, double pr, double rr, double ur,
                                                    double gam, double g1, double g2) {
  pl = pl > kSmallp ? pl : kSmallp;
  pr = pr > kSmallp ? pr : kSmallp;
  rl = rl > kSmallr ? rl : kSmallr;
  rr = rr > kSmallr ? rr : kSmallr;
  double xl = gam * pl * rl, xr = gam * pr * rr;
  const double cl = xl * rsq(xl), cr = xr * rsq(xr);
  const double vl = 4.0 * rcp(rl), vr = 4.0 * rcp(rr), ipl = rcp(pl), ipr = rcp(pr);
  double pm = pr - pl - cr * (ur - ul);
  pm = pl + pm * cl * rcp(cl + cr);
  pm = pm > kSmallp ? pm : kSmallp;
  double wl = 0.0, wr = 0.0;
  for (int it = 0; it < 10; it++) {
    const double prev = pm;
    xl = fma(g1 * (pm - pl), ipl, 1.0);
    xr = fma(g1 * (pm - pr), ipr, 1.0);
    wl = cl * (xl * rsq(xl));
    wr = cr * (xr * rsq(xr));
    double zl = vl * wl * wl, zr = vr * wr * wr;
    zl = -zl * wl * rcp(zl - g2 * (pm - pl));
    zr = zr * wr * rcp(zr - g2 * (pm - pr));
    const double uml = ul - (pm - pl) * rcp(wl), umr = ur + (pm - pr) * rcp(wr);
    pm = pm + (umr - uml) * (zr * zl) * rcp(zr - zl);
    pm = pm > kSmallp ? pm : kSmallp;
    if (fabs(pm - prev) < 1.0e-8 * pm) break;
  }
  const double um = 0.5 * ((ul - (pm - pl) * rcp(wl)) + (ur + (pm - pr) * rcp(wr)));
  return make_double2(um, pm);
}

// ---------------------------------------------------------------------------
// The chain.  On entry the warp's slots hold the chunk's density, sweep
// velocity and the two transverse slots (radial: angular momentum r_cyl v_phi
// and r v_theta; azimuthal: v_theta and v_r; polar: v_r and the angular
// momentum) and, but in an isothermal azimuthal sweep, the pressure; cs is the
// sound crossing number dt/2 c / width.  On return the slots of cells
// 6 <= n < lim - 6 hold the remapped values, the others the Lagrangian ones,
// which is what the viscosity's stencil reads at the chunk's ends
// (remap.cu:94, viscosity.cu:370-472).  All lanes of the warp call it.
template <int AXIS, bool THREED, int EOS, bool ODD, int C>
__device__ __forceinline__ void warp_chain(const Lane<C> &L, const PlanetC &P, const Phys &ph, const double (&cs)[C]) {
  constexpr bool PAR_P = !(AXIS == 1 && EOS == 0);      // p has a parabola of its own
  const int lim = L.lim;
  const double dt = L.dt, hdt = 0.5 * dt;

  // ---- flatten flatten.cu:7-40 ----
  // A shock needs |dp1| / min(p) > 0.33, a ratio of the outer pressures above
  // 1.33: their high words then differ by more than 0.32 * 2^20 (the least is
  // 0.33 * 2^20, at mantissas near 1 and 2).  Warps without such a cell skip
  // the rest.  The azimuthal sweep takes ratios of rho for those of p.
  bool flat = false;
  if (ph.flat) {
    double p[C];
    get<C>(L, PAR_P ? W_P : W_R, p);
    int hi[C];
    bool any = false;
    PG_CELLS hi[c] = __double2hiint(p[c]);
    const int hl = __shfl_up_sync(0xffffffffu, hi[C - 1], 1), hr = __shfl_down_sync(0xffffffffu, hi[0], 1);
    PG_CELLS {
      const int d = (c < C - 1 ? hi[c < C - 1 ? c + 1 : 0] : hr) - (c ? hi[c ? c - 1 : 0] : hl);
      any = any || (abs(d) > 335544 && L.in(c, 2, 2));
    }
    if (__any_sync(0xffffffffu, any)) {
      double u[C], pl[C], pr[C], ul[C], ur[C], pll[C], prr[C], st[C], sl[C], sr[C];
      get<C>(L, W_U, u);
      left_of<C>(p, pl);
      right_of<C>(p, pr);
      left_of<C>(u, ul);
      right_of<C>(u, ur);
      left_of<C>(pl, pll);
      right_of<C>(pr, prr);
      any = false;
      // smallp bounds the pressure's difference: with rho in place of p, 1e-15 / cs2
      const double small = PAR_P ? kSmallp : kSmallp / L.cs2;
      PG_CELLS {
        const double m = pr[c] < pl[c] ? pr[c] : pl[c];
        // velocities that the limiter left at 1e-308 for zero are equal
        const bool shock = fabs(pr[c] - pl[c]) > 0.33 * m && m >= 0.0 && !(ul[c] + 1.0e-290 < ur[c]) && L.in(c, 2, 2);
        double dp2 = prr[c] - pll[c];
        if (fabs(dp2) < small) dp2 = small;
        const double x = ((pr[c] - pl[c]) / dp2 - 0.75) * 5.0;
        st[c] = (shock && x > 0.0) ? x : 0.0;
        any = any || shock;
      }
      left_of<C>(st, sl);
      right_of<C>(st, sr);
      PG_CELLS {
        double m = sl[c] > st[c] ? sl[c] : st[c];
        m = m > sr[c] ? m : sr[c];
        m = m < 0.5 ? m : 0.5;
        st[c] = L.in(c, 2, 2) ? 1.0 - m : 1.0;
      }
      put<C>(L, W_OMF, st);
      flat = __any_sync(0xffffffffu, any);
    }
  }


  // ---- states states.cu:3-73 ----
  double um[C], pm[C];
  {
    double sl[C], sr[C];
    {
      ParC<C> k;
      ld<C>(L, A_C0, k.c0);
      ld<C>(L, A_C1, k.c1);
      ld<C>(L, A_C2, k.c2);
      ld<C>(L, A_C3, k.c3);
      ld<C>(L, A_C4, k.c4);
#pragma unroll 1
      for (int f = PAR_P ? 0 : 1; f < 3; f++) {
        double a[C], d1[C], d2[C], e[C];
        get<C>(L, f == 0 ? (int)W_P : f == 1 ? (int)W_R : (int)W_U, a);
        edges<ODD, C>(L, a, k, flat, d1, d2);
        PG_CELLS {
          const double d = d1[c] + d2[c], a6 = 3.0 * (d2[c] - d1[c]), fac = fma(-kFourthd, cs[c], 1.0);
          e[c] = a[c] + fma(-cs[c], fma(-fac, a6, d), d1[c]);          // at the right face
          sr[c] = a[c] + fma(cs[c], fma(fac, a6, d), -d2[c]);          // at the left face
        }
        left_of<C>(e, sl);
        if (f < 2) {                       // the velocity's stay in registers
          put<C>(L, f == 0 ? (int)W_SLP : (int)W_SLR, sl);
          put<C>(L, f == 0 ? (int)W_SRP : (int)W_SRR, sr);
        }
      }
    }

    // ---- forces at the faces, t + dt/2 ----
    double f[C];
    if (AXIS == 0) {
      double x[C], ix[C], v[C], w[C], vl[C], wl[C], ch[C], sh[C];
      ld_row<C>(L, R_CH, ch);
      ld_row<C>(L, R_SH, sh);
      ld<C>(L, A_XF, x);
      ld<C>(L, A_E0, ix);
      get<C>(L, W_V, v);
      left_of<C>(v, vl);
      if (THREED) {
        get<C>(L, W_W, w);
        left_of<C>(w, wl);
      }
      PG_CELLS f[c] = force_r<THREED, ODD>(x[c], ix[c], fma(L.c0, ch[c], -(L.s0 * sh[c])), 0.5 * (v[c] + vl[c]),
                                           THREED ? 0.5 * (w[c] + wl[c]) : 0.0, P, ph.plnt, L.isp2);
    } else if (AXIS == 1) {
      PG_CELLS f[c] = 0.0;
      if (ph.plnt) {
        double k[C], s[C];
        ld<C>(L, A_E0, k);
        ld<C>(L, A_E1, s);
        PG_CELLS f[c] = force_phi(L.rad, L.bq, L.sp, fma(k[c], L.cb, -(s[c] * L.sb)), fma(s[c], L.cb, k[c] * L.sb), P);
      }
    } else {
      double w[C], wl[C], sf[C], cf[C], is[C], ch[C], sh[C];
      ld_row<C>(L, R_CH, ch);
      ld_row<C>(L, R_SH, sh);
      ld<C>(L, A_E0, sf);
      ld<C>(L, A_E1, cf);
      ld<C>(L, A_E4, is);
      get<C>(L, W_W, w);
      left_of<C>(w, wl);
      PG_CELLS f[c] = force_theta(L.rad, L.bq, sf[c], cf[c], is[c] * L.irad, is[c], fma(L.c0, ch[c], -(L.s0 * sh[c])),
                                  0.5 * (w[c] + wl[c]), P, ph.plnt);
    }

    // ---- riemann riemann.cu:3-115 at the left face of each cell ----
    double pl[C], pr[C], rl[C], rr[C];
    PG_CELLS {
      sl[c] = fma(hdt, f[c], sl[c]);
      sr[c] = fma(hdt, f[c], sr[c]);
    }
    get<C>(L, W_SLR, rl);
    get<C>(L, W_SRR, rr);
    if (PAR_P) {
      get<C>(L, W_SLP, pl);
      get<C>(L, W_SRP, pr);
    }
    if (EOS == 0) {
      bool far[C], any = false;
      PG_CELLS {
        int low = min(__double2hiint(rl[c]), __double2hiint(rr[c]));
        bool ok;
        if (PAR_P) {
          low = min(low, min(__double2hiint(pl[c]), __double2hiint(pr[c])));
          const double w = fma(pl[c], rsq(pl[c] * rl[c]), pr[c] * rsq(pr[c] * rr[c])), pp = pl[c] * pr[c];
          ok = riemann_near(pl[c], pr[c], pp * rsq(pp), w, sl[c], sr[c], um[c], pm[c]) && low > kTiny;
        } else {
          // sqrt(p / rho) is the ring's
          const double pp = rl[c] * rr[c];
          ok = riemann_near(rl[c], rr[c], L.cs2 * (pp * rsq(pp)), 2.0 * L.ciso, sl[c], sr[c], um[c], pm[c]) && low > L.low;
        }
        far[c] = !ok && L.in(c, 3, 2);
        any = any || far[c];
      }
      if (any) {
        PG_CELLS {
          if (far[c]) {
            const double2 t = PAR_P ? riemann_iso_call(pl[c], rl[c], sl[c], pr[c], rr[c], sr[c])
                                    : riemann_iso_call(L.cs2 * rl[c], rl[c], sl[c], L.cs2 * rr[c], rr[c], sr[c]);
            um[c] = t.x;
            pm[c] = t.y;
          }
        }
      }
    } else {
      PG_CELLS {
        um[c] = 0.0;
        pm[c] = 1.0;
        if (L.in(c, 3, 2)) {
          const double2 t = riemann_isen(pl[c], rl[c], sl[c], pr[c], rr[c], sr[c], ph.gam, ph.gamfac1, ph.gamfac2);
          um[c] = t.x;
          pm[c] = t.y;
        }
      }
    }
  }

  // ---- evolve evolve.cu:3-166 ----
  // dvol and the remap's overlap volume lvol leave out the factor r that the
  // azimuthal and polar volumes share with dvol0
  double dx[C], lvol[C], del[C], m[C];
  {
    double xf[C], xa[C], xr[C], vf[C], f1[C], f2[C], dvol[C];
    ld<C>(L, A_XF, xf);
    PG_CELLS {
      double d;
      if (AXIS == 0) d = dt * um[c];
      else if (AXIS == 1) d = dt * (um[c] * L.irad - L.vr - L.frrot);
      else d = dt * um[c] * L.irad;
      xa[c] = xf[c] + d;
    }
    right_of<C>(xa, xr);
    PG_CELLS dx[c] = xr[c] - xa[c];
    if (AXIS == 0) {
      double xc[C], ixc[C], v[C], w[C], ch[C], sh[C];
      ld_row<C>(L, R_CH, ch);
      ld_row<C>(L, R_SH, sh);
      ld<C>(L, A_XC, xc);
      ld<C>(L, A_E1, ixc);
      get<C>(L, W_V, v);
      if (THREED) get<C>(L, W_W, w);
      PG_CELLS {
        const double s = 2.0 * sh[c] * ch[c], k = fma(-2.0 * sh[c], sh[c], 1.0);    // the change in dt
        const double xn = fma(0.5, dx[c], xa[c]), wc = THREED ? w[c] : 0.0;
        f1[c] = force_r<THREED, ODD>(xc[c], ixc[c], L.c0, v[c], wc, P, ph.plnt, L.isp2);
        f2[c] = force_r<THREED, ODD>(xn, rcp(xn), fma(L.c0, k, -(L.s0 * s)), v[c], wc, P, ph.plnt, L.isp2);
        const double d = xa[c] - xf[c];
        const double xe = L.n(c) < lim - 3 ? xa[c] : xf[c];         // the last face keeps its start (evolve.cu:36-44)
        if (!THREED) {
          dvol[c] = dx[c] * fma(0.5, dx[c], xa[c]);
          vf[c] = 0.5 * (xe + xf[c]);
          lvol[c] = d * fma(0.5, d, xf[c]);
        } else {
          dvol[c] = dx[c] * fma(xa[c], xa[c] + dx[c], dx[c] * dx[c] * kThird);
          const double de = xe - xf[c];
          vf[c] = fma(de, fma(kThird, de, xf[c]), xf[c] * xf[c]);
          lvol[c] = d * fma(xf[c], xa[c], kThird * (d * d));
        }
        del[c] = d;
      }
    } else if (AXIS == 1) {
      PG_CELLS f1[c] = f2[c] = 0.0;
      if (ph.plnt) {
        double k[C], s[C], xc[C];
        ld<C>(L, A_E2, k);
        ld<C>(L, A_E3, s);
        ld<C>(L, A_XC, xc);
        PG_CELLS {
          f1[c] = force_phi(L.rad, L.bq, L.sp, fma(k[c], L.ca, -(s[c] * L.sa)), fma(s[c], L.ca, k[c] * L.sa), P);
          // the centre moves by a fraction of a cell: one more rotation
          double se, ce;
          sincos_near(fma(0.5, dx[c], xa[c]) - xc[c], se, ce, C == 4 || L.n(c) < lim);
          const double cr = fma(L.cc, ce, -(L.sc * se)), sn = fma(L.sc, ce, L.cc * se);
          f2[c] = force_phi(L.rad, L.bq, L.sp, fma(k[c], cr, -(s[c] * sn)), fma(s[c], cr, k[c] * sn), P);
        }
      }
      PG_CELLS {
        del[c] = xa[c] - xf[c];
        dvol[c] = dx[c];
        lvol[c] = del[c];
      }
    } else {
      double sf[C], cf[C], sc[C], cc[C], isc[C], xc[C], w[C], chr[C], shr[C];
      ld_row<C>(L, R_CH, chr);
      ld_row<C>(L, R_SH, shr);
      ld<C>(L, A_E0, sf);
      ld<C>(L, A_E1, cf);
      ld<C>(L, A_E2, sc);
      ld<C>(L, A_E3, cc);
      ld<C>(L, A_E5, isc);
      ld<C>(L, A_XC, xc);
      get<C>(L, W_W, w);
      PG_CELLS {
        const double s = 2.0 * shr[c] * chr[c], k = fma(-2.0 * shr[c], shr[c], 1.0);   // the change in dt
        double se, ce;
        f1[c] = force_theta(L.rad, L.bq, sc[c], cc[c], isc[c] * L.irad, isc[c], L.c0, w[c], P, ph.plnt);
        sincos_near(fma(0.5, dx[c], xa[c]) - xc[c], se, ce, C == 4 || L.n(c) < lim);
        const double sn = fma(sc[c], ce, cc[c] * se), cn = fma(cc[c], ce, -(sc[c] * se)), is = rcp(sn);
        f2[c] = force_theta(L.rad, L.bq, sn, cn, is * L.irad, is, fma(L.c0, k, -(L.s0 * s)), w[c], P, ph.plnt);
        // cos(a) - cos(a + dx) = 2 sin(a + dx/2) sin(dx/2); the faces move by
        // a fraction of a cell, so their sines come from the Eulerian face's
        dvol[c] = sn * dx[c] * sinc_near(0.5 * dx[c], C == 4 || L.n(c) < lim);
        const double d = xa[c] - xf[c], h = 0.5 * d;
        double sh, ch;
        sincos_near(h, sh, ch, C == 4 || L.n(c) < lim);
        const double sm = fma(sf[c], ch, cf[c] * sh);               // sin of the mid angle
        const double g = sm * sinc_near(h, C == 4 || L.n(c) < lim);
        lvol[c] = d * g;
        vf[c] = L.n(c) < lim - 3 ? g : sf[c];                       // the last face keeps its start (evolve.cu:36-44)
        del[c] = d;
      }
    }
    double vol[C], ivol[C], pr[C], vr[C], r[C], u[C];
    ld<C>(L, A_VOL, vol);
    ld<C>(L, A_IVOL, ivol);
    get<C>(L, W_R, r);
    get<C>(L, W_U, u);
    right_of<C>(pm, pr);
    if (AXIS != 1) right_of<C>(vf, vr);
    bool low = false;                     // a density below its bound: an emptied cell, or one whose faces crossed
    PG_CELLS {
      const double dm = dt * ivol[c] * (AXIS == 0 ? 1.0 : L.irad) * rcp(r[c]);     // dt / (r dvol0)
      double a = dm * (pr[c] - pm[c]);
      if (AXIS != 1) a *= 0.5 * (vr[c] + vf[c]);
      u[c] = u[c] + fma(hdt, f1[c] + f2[c], -a);
      m[c] = r[c] * vol[c];               // the cell's mass, which the Lagrangian step keeps
      r[c] = m[c] * rcp(dvol[c]);
      low = low || (!above_bound(r[c]) && L.n(c) < lim - 3);
    }
    if (low) {
      // the bound takes its place, and its mass is the bound's times the moved
      // volume (evolve.cu:137, remap.cu:94-99)
      PG_CELLS {
        const bool held = r[c] > kSmallr;
        m[c] = held ? m[c] : kSmallr * dvol[c];
        r[c] = held ? r[c] : kSmallr;
      }
    }
    put<C>(L, W_R, r);
    put<C>(L, W_U, u);
  }

  // ---- remap remap.cu:14-226 ----
  // paraset on the Lagrangian widths, then field by field the parabola and
  // the flux through each left face from its upwind cell (get_flux
  // remap.cu:1-10), density first: its flux carries the others.
  ParC<C> k;
  double e[C];                            // half the face's displacement over the donor's width
  {
    double xm[C], xp[C], a[C], am[C], ap[C], ia[C], im[C];
    left_of<C>(dx, xm);
    right_of<C>(dx, xp);
    PG_CELLS {
      a[c] = dx[c] + xp[c];
      ia[c] = rcp(a[c]);
    }
    left_of<C>(a, am);
    right_of<C>(a, ap);
    left_of<C>(ia, im);
    PG_CELLS {
      const double ib = rcp(a[c] + dx[c]), g = a[c] + xp[c], ig = rcp(g);
      const double d = rcp(am[c] + ap[c]);
      const double mb = am[c] * ib, pg_ = ap[c] * ig, dp = d * xp[c];
      k.c0[c] = dx[c] * ia[c] * fma(2.0 * dp, mb - pg_, 1.0);
      k.c1[c] = -d * dx[c] * mb;
      k.c2[c] = dp * pg_;
      const double h = dx[c] * rcp(am[c] + xp[c]);
      k.c3[c] = h * (am[c] + xm[c]) * ia[c];
      k.c4[c] = h * g * im[c];
      e[c] = 0.5 * del[c] * rcp(del[c] >= 0.0 ? xm[c] : dx[c]);
    }
  }
  // 1 / mass after the remap (per dvol's unit, as m), whose sign says which way
  // the left face moved: e's own turns around with a crossed donor's width; mass flux
  double im[C], mf[C];
  PG_CELLS {
    im[c] = del[c];
    mf[c] = lvol[c];
  }
  // 2D leaves out the slot that stays zero: w of the radial sweep, v of the
  // azimuthal one
  constexpr int NF = THREED ? 4 : 3;
#pragma unroll 1
  for (int f = 0; f < NF; f++) {
    const int slot = (AXIS == 1 && !THREED && f == 2) ? (int)W_W : f;
    double a[C], d1[C], d2[C], al[C], l1[C], l2[C], fl[C], fr[C];
    get<C>(L, slot, a);
    edges<ODD, C>(L, a, k, flat, d1, d2);
    left_of<C>(a, al);
    left_of<C>(d1, l1);
    left_of<C>(d2, l2);
    PG_CELLS {
      const bool up = __double2hiint(im[c]) >= 0;
      const double q = up ? al[c] : a[c], x1 = up ? l1[c] : d1[c], x2 = up ? l2[c] : d2[c];
      // t = edge - e (da - s a6), s = 1 - 4/3 e from the left cell, -(1 + 4/3 e) from the right one
      const double s3 = fma(-4.0, e[c], up ? 3.0 : -3.0);
      const double t = q + fma(-e[c], fma(-s3, x2 - x1, x1 + x2), up ? x1 : -x2);
      fl[c] = t * mf[c];
    }
    right_of<C>(fl, fr);
    if (f == 0) {
      double ivol[C], vol[C];
      ld<C>(L, A_IVOL, ivol);
      ld<C>(L, A_VOL, vol);
      PG_CELLS {
        double q = quot(m[c] + fl[c] - fr[c], vol[c], ivol[c]);
        q = q > kSmallr ? q : kSmallr;
        a[c] = L.in(c, NPAD, NPAD) ? q : a[c];
        im[c] = copysign(rcp(a[c] * vol[c]), im[c]);
        mf[c] = fl[c];
      }
    } else {
      PG_CELLS {
        const double q = fma(a[c], m[c], fl[c] - fr[c]) * fabs(im[c]);
        a[c] = L.in(c, NPAD, NPAD) ? q : a[c];
      }
    }
    put<C>(L, slot, a);
  }
}

// first and second derivative of a field on the faces' coordinates (derivs
// viscosity.cu:2-18), from the axis table's weights of the two differences
template <int C>
struct Deriv {
  double a[C], b[C], p[C], q[C];
  __device__ __forceinline__ void load(const Lane<C> &L) {
    ld<C>(L, A_VA, a);
    ld<C>(L, A_VB, b);
    ld<C>(L, A_VC, p);
    ld<C>(L, A_VD, q);
  }
  __device__ __forceinline__ void of(const double (&f)[C], double (&d1)[C], double (&d2)[C]) const {
    double dr[C], dl[C];
    right_of<C>(f, dr);
    PG_CELLS dr[c] = dr[c] - f[c];
    left_of<C>(dr, dl);
    PG_CELLS {
      d1[c] = fma(a[c], dr[c], b[c] * dl[c]);
      d2[c] = fma(p[c], dr[c], -(q[c] * dl[c]));
    }
  }
};

}  // namespace pgd
