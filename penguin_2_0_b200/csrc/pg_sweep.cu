// pg_sweep.cu -- the directional sweeps: each chunk of a pencil is one warp's
// work (pg_warp.cuh), in FP64 arithmetic on FP64 or FP32 state planes.
//
//   k_sweep_x   radial sweep (ppm.cu:26-160)
//   k_sweep_y   azimuthal sweep (ppm.cu:162-307); FARGO integer shift
//               (rotate_rings, ppm.cu:309-322) at its store; optional fused
//               epilogue: wave damping, CFL rate max (dt_lv1,
//               timestep.cu:12-73), finiteness check into the status word
//   k_sweep_z   polar sweep (3D), same store and epilogue
//   kb_sweep_*  the radial and azimuthal sweeps of every 2D member of a batch
//
// FP32 planes hold dS = Sigma - S_bg(ring) and dv = v_phi - v_bg(ring); a
// sweep adds the FP64 ring values at its loads and rounds the differences at
// its stores, so both plane types run the same chain.
//
// A CTA of 4 warps takes one tile.  Radial and polar tiles are 4 P adjacent
// azimuth columns of one chunk (P pencils per warp: one full chunk, or as
// many short ones as 32 lanes hold); the CTA moves them between global and
// shared memory with neighbouring threads on neighbouring columns, where a
// lane that read its own rows would use 8 of each 32-byte sector.  Azimuthal
// pencils lie along the rows: each warp reads its cells directly and passes
// its results through shared memory, so that a store instruction covers 256
// contiguous bytes.
//
// What bounds them and what they measured (B200, event-timed per sweep, FP64):
// instruction issue (pg_warp.cuh) at 2.2-2.4 of 4 per cycle and SM, FP64 pipe
// 43-51 %, DRAM below 15 %.  Against one thread per cell, the chain through
// shared memory and 22 CTA barriers per chunk:
//   128x1024x32  radial 628 -> 268 us, azimuthal 554 -> 194, polar 698 -> 422
//   1536x4608    radial 836 -> 346 us, azimuthal 906 -> 312
//   256x768      radial  46 ->  21 us, azimuthal  37 ->  21
// Of the radial sweep's 162 M instructions on the 3D disk 26 M are the tile's
// loads and stores and what they need, of the azimuthal one's 131 M 17 M, of
// the polar one's 285 M some 55 M.
// 4 warps per CTA, 4 CTAs per SM at 128 registers.  A thread reloads 44-96 bytes of
// spills in the radial sweep, 120-160 in the azimuthal one, 24-32 in the polar one
// with 3 cells per lane and 156-244 with 4, 284-320 in the batch's kernels, whose
// tables are behind a pointer.  3 CTAs ran 2-13 % longer but on the smallest grids,
// 5 CTAs 5-25 %, 8 warps per CTA 5 %, 16 warps 30 %.  Loading the tile in one go before the first use took
// the radial sweep from 344 to 328 us, cutting the workspace from 11 to 9 slots
// (which leaves L1 room for the axis tables) from 308 to 284, planet constants
// from the clock and quotients by multiplication (tiles formed on the host) to
// 268.
#include "pg_warp.cuh"

namespace pgd {

constexpr int NW = 4;                    // warps per CTA
constexpr int NT = 32 * NW;
constexpr int MINB = 4;                  // CTAs per SM

struct StepIn {
  double dt, frrot, frrot_next;
  Body pl;
};
// the step's dt, planet and frame rotation: launch arguments or the device clock
__device__ __forceinline__ bool load_step(const SweepCtl &c, StepIn &s) {
  if (c.clk) {
    // all loads at once: one round trip to L2
    s.dt = c.clk->dt_step;
    s.frrot = c.clk->frrot;
    s.frrot_next = c.clk->frrot_next;
    s.pl = c.clk->planet;
    return !c.clk->halted;
  } else {
    s.dt = c.dt;
    s.frrot = c.frrot;
    s.frrot_next = c.frrot;
    s.pl = c.planet;
  }
  return true;
}

// Keeps the loads before it ahead of what follows: a tile's loads do not wait
// for the look at the clock.
__device__ __forceinline__ void in_flight() { asm volatile("" ::: "memory"); }

// The planet's constants into shared memory: from the clock, or (calls with a
// planet of their own) formed by one thread while the others load.
template <bool THREED>
__device__ __forceinline__ void planet_shm(PlanetC &S, const SweepCtl &ctl, const StepIn &st, const Phys &ph) {
  constexpr int N = sizeof(PlanetC) / sizeof(double);
  const int t = (int)threadIdx.x - (NT - 32);
  if (ctl.clk) {
    if (t >= 0 && t < N) reinterpret_cast<double *>(&S)[t] = reinterpret_cast<const double *>(&ctl.clk->pc)[t];
  } else if (t == 0) {
    S = planet_consts(st.pl, THREED, ph.plnt, st.dt);
  }
}

// ---------------------------------------------------------------------------
// axis tables (pg_warp.cuh AxisEntry): chunk l of an axis holds A_COUNT
// arrays of ARR entries, cell n = C g + c stored so that a lane's C entries
// are read in whole lines by the warp (table_pos)
__device__ __forceinline__ int table_pos(int n, int C, int G) {
  const int g = n / C, c = n % C;
  return C == 4 ? (c >> 1) * 2 * G + 2 * g + (c & 1) : c * G + g;
}

__global__ void k_axis_table(Tables T, int axis, int C, double *out) {
  const Chunking &ch = axis == 0 ? T.cx : axis == 1 ? T.cy : T.cz;
  const int nn = axis == 0 ? T.nr : axis == 1 ? T.nphi : T.nk;
  const int l = blockIdx.x, n = threadIdx.x, N = nn + 2 * NPAD;
  const int lim = l == ch.loop - 1 ? ch.lim_last : ARR;
  const int G = (lim + C - 1) / C;
  if (n >= C * G) return;
  auto clampe = [&](int e) { return e < 0 ? 0 : e >= N ? N - 1 : e; };
  auto turn = [&](int e) { return e < NPAD ? -1 : e >= nn + NPAD ? 1 : 0; };
  auto face = [&](int e) {
    e = clampe(e);
    if (axis == 0) return T.rx[e];
    if (axis == 2) return T.z[e];
    return T.y[e - NPAD - turn(e) * nn] + turn(e) * kTwoPi;
  };
  auto width = [&](int e) {
    e = clampe(e);
    if (axis == 0) return T.rdx[e];
    if (axis == 2) return T.dz[e];
    return T.dy[e - NPAD - turn(e) * nn];
  };
  const int e = clampe(REAL * l + n);
  const double xm = width(e - 1), x = width(e), xp = width(e + 1), xpp = width(e + 2);
  const double a = x + xp, b = a + x, c = a + xp, am = xm + x, ap = xp + xpp;
  const double d = 1.0 / (am + ap);
  double o[A_COUNT] = {};
  o[A_XF] = face(e);
  o[A_IW] = 1.0 / x;
  o[A_C0] = x / a * (1.0 + 2.0 * d * xp * (am / b - ap / c));
  o[A_C1] = -d * x * am / b;
  o[A_C2] = d * xp * ap / c;
  const double h = x / (am + xp);
  o[A_C3] = h * (am + xm) / a;
  o[A_C4] = h * c / am;
  // derivs (viscosity.cu:2-18) on faces at distances f1 to the left and f2 to
  // the right: first = (f1/f2 D+ + f2/f1 D-)/(f1+f2), second = 2 (D+/f2 - D-/f1)/(f1+f2)
  const double f1 = face(e) - face(e - 1), f2 = face(e + 1) - face(e), fs = f1 + f2;
  if (f1 > 0.0 && f2 > 0.0) {
    o[A_VA] = f1 / (f2 * fs);
    o[A_VB] = f2 / (f1 * fs);
    o[A_VC] = 2.0 / (f2 * fs);
    o[A_VD] = 2.0 / (f1 * fs);
  }
  o[A_VOL] = axis == 0 ? T.rxvol[e] : axis == 2 ? T.zvol[e] : T.yvol[e - NPAD - turn(e) * nn];
  o[A_IVOL] = 1.0 / o[A_VOL];
  o[A_XC] = axis == 0 ? T.rxc[e] : axis == 2 ? T.zc[e] : T.yc[e - NPAD - turn(e) * nn] + turn(e) * kTwoPi;
  if (axis == 0) {
    o[A_E0] = 1.0 / o[A_XF];
    o[A_E1] = 1.0 / o[A_XC];
  } else {
    const bool az = axis == 1;
    sincos(o[A_XF], &o[az ? A_E1 : A_E0], &o[az ? A_E0 : A_E1]);
    sincos(o[A_XC], &o[az ? A_E3 : A_E2], &o[az ? A_E2 : A_E3]);
    if (!az) {
      o[A_E4] = 1.0 / o[A_E0];
      o[A_E5] = 1.0 / o[A_E2];
    }
  }
  double *q = out + (size_t)l * A_COUNT * ARR + table_pos(n, C, G);
  for (int i = 0; i < A_COUNT; i++) q[i * ARR] = o[i];
}

// ---------------------------------------------------------------------------
// Shared block of a radial or polar tile: the warps' workspaces and the
// per-row values
struct __align__(16) TileShm {
  double ws[NW][WS];
  double row[R_COUNT][ARR];
  PlanetC pl;
};
// Place of cell n of column cl of a tile in a slot of its warp's workspace
struct ColMap {
  int w, l0;                             // the column's warp and first lane
  __device__ __forceinline__ ColMap(const Tile &M, int cl) : w(quot16(cl, M.mP)), l0((cl - w * M.P) * M.G) {}
  template <int C>
  __device__ __forceinline__ int at(int n) const {
    const int g = n / C, c = n - g * C;
    return ws_lane<C>(l0 + g) + (C == 4 ? (c >> 1) * PIECE<4> + (c & 1) : c * PIECE<3>);
  }
};
// Threads of a tile's loads and stores: thread t keeps column t % cols and
// takes rows t / cols, t / cols + step, ...; threads past the last whole row idle.
struct TileWalk {
  int cl, n;
  __device__ __forceinline__ TileWalk(const Tile &M, int tid) {
    n = quot16(tid, M.mC);
    cl = tid - n * M.cols;
    if (n >= M.step) n = 1 << 20;
  }
};

// The lane's place in a chunk of lim cells.  Lanes past the warp's last pencil
// compute on a uniform state of their own, out of every range.
template <int C, bool HAS_P = true>
__device__ __forceinline__ int place_lane(Lane<C> &L, const Tile &M, int pw, const double *tab, const double *row,
                                          double *ws, int lane) {
  const int g = min(lane - pw * M.G, M.G - 1);
  const bool idle = lane >= M.P * M.G;
  L.n0 = idle ? 1 << 20 : C * g;
  L.lim = M.lim;
  L.tab = tab + (C == 4 ? 2 * g : g);
  L.row = row + (C == 4 ? 2 * g : g);
  L.half = C == 4 ? 2 * M.G : M.G;
  L.ws = ws + ws_lane<C>(lane);
  if (idle) {
    double one[C], zero[C];
    PG_CELLS {
      one[c] = 1.0;
      zero[c] = 0.0;
    }
    put<C>(L, W_R, one);
    if (HAS_P) put<C>(L, W_P, one);
    put<C>(L, W_U, zero);
    put<C>(L, W_V, zero);
    put<C>(L, W_W, zero);
  }
  return C * g;
}

// ---------------------------------------------------------------------------
// radial sweep: tile t of the run
template <class RT, bool THREED, int EOS, bool ODD>
__device__ __forceinline__ void sweep_x_tile(TileShm &S, const Tables &T, const PlanesT<RT> &P, const Phys &ph,
                                             const SweepCtl &ctl, const StepIn &st, int t) {
  constexpr int C = 4;
  const int nphi = T.nphi, nrg = T.nrg, full = T.cx.loop - 1, tid = threadIdx.x;
  const int nfull = full * T.tx[0].ng * T.nk;
  const bool last = t >= nfull;
  const Tile &M = T.tx[last];
  if (last) t -= nfull;
  int q = quot40(t, M.ng, M.mng);
  const int j0 = (t - q * M.ng) * M.cols;
  const int k = last ? q : q / full, l = last ? full : q - k * full;
  if (last && T.cx.stuck) {
    // ppm.cu:48 gives this chunk lim = 12: its rings keep their values
#pragma unroll 1
    for (int e = tid; e < REAL * NW; e += NT) {
      const int i = REAL * l + e / NW, j = j0 + e % NW;
      if (i >= T.nr || j >= nphi) continue;
      const size_t o = ((size_t)k * nrg + i + NPAD) * nphi + j;
      P.ro[o] = P.r[o]; P.uo[o] = P.u[o]; P.vo[o] = P.v[o];
      if (THREED) P.wo[o] = P.w[o];
    }
    return;
  }
  const int lim = M.lim, row0 = REAL * l, rows = C * M.G;
  const TileWalk W(M, tid);
  const ColMap cm(M, W.cl);
  double *const cw = S.ws[cm.w];
  // every load of the tile in flight before the first is used
  RT a[4][4];
  double rc[4], cs2[4], p0[4], bs[4], bv[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int n = W.n + i * M.step;
    if (n >= rows) break;
    const int rk = k * nrg + min(row0 + n, nrg - 1);
    const size_t o = (size_t)rk * nphi + min(j0 + W.cl, nphi - 1);
    a[i][0] = __ldcg(&P.r[o]);
    a[i][1] = __ldcg(&P.u[o]);
    a[i][2] = __ldcg(&P.v[o]);
    if (THREED) a[i][3] = __ldcg(&P.w[o]);
    if (P.p0) p0[i] = P.p0[o];
    rc[i] = T.radc[rk];
    cs2[i] = T.cs2[rk];
    if (sizeof(RT) == 4) {
      bs[i] = T.sbg[rk];
      bv[i] = T.vbg[rk];
    }
  }
  if (tid < rows) {
    const int rk = k * nrg + min(row0 + tid, nrg - 1);
    const double snd = T.snd[rk], nu = T.nu[rk], r = T.radc[rk], irc = T.irc[rk], res = T.res_v[rk];
    const int q = table_pos(tid, C, M.G);
    S.row[R_SND][q] = 0.5 * st.dt * snd;
    double sh, ch;
    sincos_near(0.5 * st.dt * (res * irc - st.pl.vy), sh, ch);
    S.row[R_CH][q] = ch;
    S.row[R_SH][q] = sh;
    S.row[R_NU][q] = nu;
    S.row[R_RC][q] = r;
    S.row[R_IRC][q] = irc;
  }
  planet_shm<THREED>(S.pl, ctl, st, ph);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int n = W.n + i * M.step;
    if (n >= rows) break;
    const int s = cm.at<C>(n);
    const double r = load_r(a[i][0], bs[i]);
    cw[W_R * SLOT + s] = r;
    cw[W_U * SLOT + s] = (double)a[i][1];
    cw[W_V * SLOT + s] = load_r(a[i][2], bv[i]) * rc[i];
    if (THREED) cw[W_W * SLOT + s] = (double)a[i][3];
    cw[W_P * SLOT + s] = P.p0 ? p0[i] : EOS == 0 ? r * cs2[i] : cs2[i] * pow_call(r, ph.gam) / ph.gam;
  }
  __syncthreads();
  {
    const int lane = tid & 31, wid = tid >> 5, pw = min(quot16(lane, M.mG), M.P - 1);
    const PlanetC pl = S.pl;
    Lane<C> L;
    place_lane<C>(L, M, pw, T.ax[0] + (size_t)l * A_COUNT * ARR, S.row[0], S.ws[wid], lane);
    L.dt = st.dt;
    {
      // cos and sin of the column's azimuth less the planet's
      const int j = min(j0 + wid * M.P + pw, nphi - 1);
      const double cy = T.cyc[j], sy = T.syc[j];
      L.sp = THREED ? T.szc[k + NPAD] : 1.0;
      L.isp2 = THREED ? rcp(L.sp * L.sp) : 1.0;
      L.c0 = fma(cy, pl.cy, sy * pl.sy) * L.sp;
      L.s0 = fma(sy, pl.cy, -(cy * pl.sy)) * L.sp;
    }
    if (THREED) {
      double x[C], w[C];
      ld<C>(L, A_XC, x);
      get<C>(L, W_W, w);
      PG_CELLS w[c] *= x[c];
      put<C>(L, W_W, w);
    }
    {
      double cs[C];
      ld<C>(L, A_IW, cs);
      if (EOS == 0 && !P.p0 && !ODD) {
        double snd[C];
        ld_row<C>(L, R_SND, snd);
        PG_CELLS cs[c] = snd[c] * cs[c];
      } else {
        double p[C], r[C];
        get<C>(L, W_P, p);
        get<C>(L, W_R, r);
        PG_CELLS {
          const double x = ph.gam * p[c] * rcp(r[c]);
          cs[c] = 0.5 * st.dt * root(x) * cs[c];
        }
      }
      warp_chain<0, THREED, EOS, ODD, C>(L, pl, ph, cs);
    }
    // device_viscosity_r viscosity.cu:370-421; the stored v_phi is v / r_cyl
    double irc[C], rc[C], v[C];
    ld_row<C>(L, R_IRC, irc);
    ld_row<C>(L, R_RC, rc);
    get<C>(L, W_V, v);
    PG_CELLS v[c] = quot(v[c], rc[c], irc[c]);
    if (ph.visc) {
      double a[C], nr[C], n1[C], d1[C], d2[C], dtr[C];
      Deriv<C> D;
      D.load(L);
      get<C>(L, W_R, a);
      ld_row<C>(L, R_NU, nr);
      PG_CELLS {
        nr[c] *= a[c];
        dtr[c] = st.dt * rcp(a[c]);
      }
      D.of(nr, n1, d2);
      get<C>(L, W_U, a);
      D.of(a, d1, d2);
      PG_CELLS a[c] = fma(2.0 * dtr[c], fma(nr[c], fma(irc[c], fma(-a[c], irc[c], d1[c]), d2[c]), n1[c] * d1[c]), a[c]);
      put<C>(L, W_U, a);
      PG_CELLS a[c] = v[c] * irc[c];
      D.of(a, d1, d2);
      PG_CELLS {
        const double x = fma(rc[c], fma(nr[c], d2[c], n1[c] * d1[c]), 3.0 * nr[c] * d1[c]);
        v[c] = fma(dtr[c], x, v[c]);
      }
      if (THREED) {
        get<C>(L, W_W, a);
        D.of(a, d1, d2);
        PG_CELLS a[c] = fma(dtr[c], fma(nr[c], fma(d1[c], irc[c], d2[c]), n1[c] * d1[c]), a[c]);
        put<C>(L, W_W, a);
      }
    }
    put<C>(L, W_V, v);
    if (THREED) {
      double w[C], x[C], ix[C];
      get<C>(L, W_W, w);
      ld<C>(L, A_XC, x);
      ld<C>(L, A_E1, ix);
      PG_CELLS w[c] = quot(w[c], x[c], ix[c]);
      put<C>(L, W_W, w);
    }
  }
  __syncthreads();
  if (j0 + W.cl < nphi) {
#pragma unroll 2
    for (int n = W.n + 4; n < lim - NPAD; n += M.step) {
      if (n < NPAD) continue;          // a warp's rows start with a lane's cells: different banks
      const int rk = k * nrg + row0 + n;
      const size_t o = (size_t)rk * nphi + j0 + W.cl;
      const double bs = sizeof(RT) == 4 ? T.sbg[rk] : 0.0, bv = sizeof(RT) == 4 ? T.vbg[rk] : 0.0;
      const int s = cm.at<C>(n);
      P.ro[o] = store_r<RT>(cw[W_R * SLOT + s], bs);
      P.uo[o] = (RT)cw[W_U * SLOT + s];
      P.vo[o] = store_r<RT>(cw[W_V * SLOT + s], bv);
      if (THREED) P.wo[o] = (RT)cw[W_W * SLOT + s];
    }
  }
}

template <class RT, bool THREED, int EOS, bool ODD>
__global__ void __launch_bounds__(NT, MINB) k_sweep_x(Tables T, PlanesT<RT> P, Phys ph, SweepCtl ctl) {
  extern __shared__ __align__(16) unsigned char shm[];
  after_previous();
  StepIn st;
  if (!load_step(ctl, st)) return;
  sweep_x_tile<RT, THREED, EOS, ODD>(*reinterpret_cast<TileShm *>(shm), T, P, ph, ctl, st, blockIdx.x);
}

// ---------------------------------------------------------------------------
// The last sweep's epilogue on one finished cell of ring rk, layer k: damping
// on the stored state, the next get_dt's CFL rate and the finiteness check.
// Values are those that the separate kernels (k_damp, k_cfl) form.
template <class RT>
struct Finish {
  RingOut o;
  double tr, tu, tv;                     // damping targets
  double bs, bv, cs2;
  template <bool POLAR>
  __device__ __forceinline__ void ring(const Tables &T, const SweepCtl &ctl, int rk) {
    bs = sizeof(RT) == 4 ? T.sbg[rk] : 0.0;
    bv = sizeof(RT) == 4 ? T.vbg[rk] : 0.0;
    o.shift = make_int2(0, 0);
    if (!ctl.fuse) {
      if (ctl.shift) o.shift = T.ro[rk].shift;
      if (POLAR) {
        o.rc = T.ro[rk].rc;
        o.irc = T.ro[rk].irc;
      }
      return;
    }
    o = T.ro[rk];
    if (o.f != 0.0) {
      tr = T.val_r[rk]; tu = T.val_u[rk]; tv = T.val_v[rk];
    }
    cs2 = T.cs2[rk];
  }
  __device__ __forceinline__ int shift(const SweepCtl &ctl) const { return ctl.shift ? o.shift.x : 0; }
  // stores the cell at offset at (azimuth column jo) and returns its CFL rate
  template <bool THREED, int EOS>
  __device__ __forceinline__ double cell(const Tables &T, const PlanesT<RT> &P, const SweepCtl &ctl, const Phys &ph, size_t at,
                                         int jo, double r, double u, double v, double w, bool &bad) const {
    RT sr = store_r<RT>(r, bs), su = (RT)u, sv = store_r<RT>(v, bv), sw = (RT)w;
    double rate = 0.0;
    if (ctl.fuse) {
      if (o.f != 0.0) {
        sr = store_r<RT>(damped(load_r(sr, bs), tr, o.f), bs);
        su = (RT)damped((double)su, tu, o.f);
        sv = store_r<RT>(damped(load_r(sv, bv), tv, o.f), bv);
        if (THREED) sw = (RT)damped((double)sw, 0.0, o.f);
      }
      r = load_r(sr, bs);
      v = load_r(sv, bv);
      if (!ctl.nocfl) {
        const double a = EOS == 0 ? o.cs : sound_speed(r, eos_p<EOS>(r, cs2, ph), ph);
        int js = jo - o.shift.y;
        if (js < 0) js += T.nphi;
        rate = cfl_rate<THREED>(a, (double)su, o.irdx, v - o.off, T.idy[js] * o.irc, (double)sw, o.iwz);
      }
      if (!(r > 0.0) || !isfinite(r) || !isfinite((double)su) || !isfinite(v)) bad = true;
    }
    P.ro[at] = sr; P.uo[at] = su; P.vo[at] = sv;
    if (THREED) P.wo[at] = sw;
    return rate;
  }
};

// a warp's CFL maximum and failure flag into the clock
__device__ __forceinline__ void report(const SweepCtl &ctl, double rate, bool bad) {
  for (int o = 16; o > 0; o >>= 1) {
    const double x = __shfl_down_sync(0xffffffffu, rate, o);
    rate = (x > rate || x != x) ? x : rate;
  }
  bad = __any_sync(0xffffffffu, bad);
  if ((threadIdx.x & 31) == 0) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(rate);
    // NaN sorts above every number; most warps are below the maximum so far
    if ((rate > 0.0 || rate != rate) && b > *(volatile unsigned long long *)&ctl.clk->cfl_bits)
      atomicMax(&ctl.clk->cfl_bits, b);
    if (bad) atomicExch(&ctl.clk->status, 3);
  }
}

// ---------------------------------------------------------------------------
// azimuthal sweep: warp task t of the run
template <int EOS>
struct __align__(16) YShm {
  double ws[NW][EOS ? WS : WS_ISO_Y];
  PlanetC pl;
};
template <class RT, bool THREED, int EOS>
__device__ __forceinline__ void sweep_y_task(double *ws, const PlanetC &SP, const Tables &T, const PlanesT<RT> &P,
                                             const Phys &ph, const SweepCtl &ctl, const StepIn &st, bool run, int t) {
  constexpr int C = 4;
  const int nphi = T.nphi, nrg = T.nrg, full = T.cy.loop - 1, rings = T.nr * T.nk, lane = threadIdx.x & 31;
  // rings of one chunk side by side: the warps of an SM share its tables.  The
  // tasks of full chunks fill whole CTAs, so that a CTA's warps take the
  // barrier together; tasks past the last ring compute and store nothing.
  const int nfull = full * T.ty[0].ng * NW;
  const bool last = t >= nfull;
  const Tile &M = T.ty[last];
  int l = full, ring;
  if (!last) {
    const int cta = t / NW;
    l = quot40(cta, M.ng, M.mng);
    ring = t - l * M.ng * NW;
  } else {
    ring = (t - nfull) * M.P;
  }
  const int lim = M.lim;
  if (last && T.cy.stuck) {
    if (ring >= rings || !run) return;
    // ppm.cu:196 gives this chunk lim = 12: its cells keep their values and
    // only move with the ring's rotation
    const int k = ring / T.nr, row = ring % T.nr + NPAD, rk = k * nrg + row;
    const size_t base = (size_t)rk * nphi;
    Finish<RT> F;
    F.template ring<false>(T, ctl, rk);
    const int inc = F.shift(ctl);
    double rate = 0.0;
    bool bad = false;
#pragma unroll 1
    for (int j = REAL * l + lane; j < nphi; j += 32) {
      int jo = j + inc;
      if (jo >= nphi) jo -= nphi;
      const size_t s = base + j;
      const double x = F.template cell<THREED, EOS>(T, P, ctl, ph, base + jo, jo, load_r(P.r[s], F.bs), (double)P.u[s],
                                                    load_r(P.v[s], F.bv), THREED ? (double)P.w[s] : 0.0, bad);
      rate = (x > rate || x != x) ? x : rate;
    }
    if (ctl.fuse) report(ctl, rate, bad);
    return;
  }
  {
    const int pw = min(quot16(lane, M.mG), M.P - 1);
    const int q = min(ring + pw, rings - 1), k = quot40(q, T.nr, T.mnr), row = q - k * T.nr + NPAD, rk = k * nrg + row;
    Lane<C> L;
    const int n0 = place_lane<C, (EOS != 0)>(L, M, pw, T.ax[1] + (size_t)l * A_COUNT * ARR, ws, ws, lane);
    // all loads in flight before the first is used; the four cells of a lane
    // share their sectors in L1
    const size_t base = (size_t)rk * nphi;
    RT x[4][C];
    PG_CELLS {
      int j = REAL * l - NPAD + n0 + c;
      j = j < 0 ? j + nphi : j >= nphi ? j - nphi : j;
      x[0][c] = P.r[base + j];
      x[1][c] = P.v[base + j];
      if (THREED) x[2][c] = P.w[base + j];
      x[3][c] = P.u[base + j];
    }
    const double bs = sizeof(RT) == 4 ? T.sbg[rk] : 0.0, bv = sizeof(RT) == 4 ? T.vbg[rk] : 0.0;
    L.dt = st.dt;
    L.frrot = st.frrot;
    L.rad = T.radc[rk];
    L.irad = T.irc[rk];
    L.sp = THREED ? T.szc[k + NPAD] : 1.0;
    const double res = T.res_v[rk];
    L.vr = res * L.irad;
    L.cs2 = T.cs2[rk];
    const double snd = T.snd[rk], rs = T.rxc[row];
    in_flight();
    if (!run) return;
    __syncthreads();                     // the planet's constants
    const PlanetC pl = SP;
    {
      L.bq = fma(rs, rs, pl.b2);         // the planet's distance sees the spherical radius in 3D
      L.ca = pl.cy; L.sa = -pl.sy;
      double c, s;
      sincos_near(0.5 * st.dt * (L.vr - pl.vy), s, c);
      L.cb = fma(L.ca, c, -(L.sa * s)); L.sb = fma(L.sa, c, L.ca * s);
      L.cc = fma(L.cb, c, -(L.sb * s)); L.sc = fma(L.sb, c, L.cb * s);
    }
    {
      double q[C];
      PG_CELLS q[c] = load_r(x[0][c], bs);
      put<C>(L, W_R, q);
      PG_CELLS q[c] = load_r(x[1][c], bv);
      put<C>(L, W_U, q);
      if (THREED) {
        PG_CELLS q[c] = (double)x[2][c];
        put<C>(L, W_V, q);
      }
      PG_CELLS q[c] = (double)x[3][c];
      put<C>(L, W_W, q);
    }
    double cs[C];
    {
      ld<C>(L, A_IW, cs);
      if (EOS == 0) {
        L.ciso = L.cs2 * rsq(L.cs2);
        L.low = max(kTiny, __double2hiint(1.0e-14 * rcp(L.cs2)) + 1);
        const double a = 0.5 * st.dt * snd * L.irad;
        PG_CELLS cs[c] *= a;
      } else {
        double p[C], r[C];
        get<C>(L, W_R, r);
        PG_CELLS {
          p[c] = L.cs2 * pow_call(r[c], ph.gam) / ph.gam;
          const double x2 = ph.gam * p[c] * rcp(r[c]);
          cs[c] *= 0.5 * st.dt * root(x2) * L.irad;
        }
        put<C>(L, W_P, p);
      }
    }
    warp_chain<1, THREED, EOS, false, C>(L, pl, ph, cs);
    // device_viscosity_p viscosity.cu:423-472 on x = r_cyl phi
    if (ph.visc) {
      const double nu = T.nu[rk], ir = L.irad;
      double a[C], nr[C], n1[C], d1[C], d2[C], dtr[C];
      Deriv<C> D;
      D.load(L);
      get<C>(L, W_R, a);
      PG_CELLS {
        nr[c] = nu * a[c];
        dtr[c] = st.dt * (ir * ir) * rcp(a[c]);
      }
      D.of(nr, n1, d2);
#pragma unroll 1
      for (int f = W_U; f <= W_W; f++) {
        if (!THREED && f == W_V) continue;
        const double two = f == W_U ? 2.0 : 1.0;
        get<C>(L, f, a);
        D.of(a, d1, d2);
        PG_CELLS a[c] = fma(two * dtr[c], fma(nr[c], d2[c], n1[c] * d1[c]), a[c]);
        put<C>(L, f, a);
      }
    }
  }
  __syncwarp();
  double rate = 0.0;
  bool bad = false;
  const int len = lim - 2 * NPAD;
#pragma unroll 1
  for (int b = 0; b < M.P && ring + b < rings; b++) {
    const int q = ring + b, k = quot40(q, T.nr, T.mnr), row = q - k * T.nr + NPAD, rk = k * nrg + row;
    const size_t base = (size_t)rk * nphi;
    const ColMap cm(M, b);
    Finish<RT> F;
    F.template ring<false>(T, ctl, rk);
    const int im = F.shift(ctl);
#pragma unroll 1
    for (int m = lane; m < len; m += 32) {
      const int s = cm.at<C>(m + NPAD);
      int jo = REAL * l + m + im;
      if (jo >= nphi) jo -= nphi;
      const double x = F.template cell<THREED, EOS>(T, P, ctl, ph, base + jo, jo, ws[W_R * SLOT + s], ws[W_W * SLOT + s],
                                                    ws[W_U * SLOT + s], THREED ? ws[W_V * SLOT + s] : 0.0, bad);
      rate = (x > rate || x != x) ? x : rate;
    }
  }
  if (ctl.fuse) report(ctl, rate, bad);
}

template <class RT, bool THREED, int EOS>
__global__ void __launch_bounds__(NT, MINB) k_sweep_y(Tables T, PlanesT<RT> P, Phys ph, SweepCtl ctl) {
  extern __shared__ __align__(16) unsigned char shm[];
  after_previous();
  YShm<EOS> &S = *reinterpret_cast<YShm<EOS> *>(shm);
  StepIn st;
  const bool run = load_step(ctl, st);
  planet_shm<THREED>(S.pl, ctl, st, ph);
  const int wid = threadIdx.x >> 5;
  sweep_y_task<RT, THREED, EOS>(S.ws[wid], S.pl, T, P, ph, ctl, st, run, blockIdx.x * NW + wid);
}

// ---------------------------------------------------------------------------
// polar-angle sweep (3D, ngeomz 5): no reference kernel exists
// (bundle_sweep3D is called at main.cu:376 and never defined).  Modelled on
// the radial sweep: pencils along k for one (i, phi column), fixed lower
// layers (init.cpp:415-476) and a reflecting midplane (boundary.cu:412-418,
// mirror with v_theta negated) or fixed upper layers.  Slots: u <- v_theta,
// v <- v_r, w <- r sin(theta) v_phi (so get_fz's w^2 cos/(r sin)^3 is the
// centrifugal term); viscosity follows device_viscosity_p's pattern on the
// arc length r*theta.  A tile is 4 P columns of one ring, so its row values
// (one layer per row) are shared by the whole CTA.
template <class RT, int EOS, bool ODD, int C>
__device__ __forceinline__ void sweep_z_tile(TileShm &S, const Tables &T, const PlanesT<RT> &P, const Phys &ph,
                                             const SweepCtl &ctl, const StepIn &st, bool run, int ntop, int t) {
  const int nphi = T.nphi, nrg = T.nrg, nk = T.nk, full = T.cz.loop - 1, tid = threadIdx.x;
  const int nfull = full * T.tz[0].ng * T.nr;
  const bool last = t >= nfull;
  const Tile &M = T.tz[last];
  if (last) t -= nfull;
  int q = quot40(t, M.ng, M.mng);
  const int j0 = (t - q * M.ng) * M.cols;
  const int l = last ? full : q / T.nr, i = last ? q : q - l * T.nr, row = i + NPAD;
  if (last && T.cz.stuck) {
    if (!run) return;
#pragma unroll 1
    for (int e = tid; e < REAL * NW; e += NT) {
      const int k = REAL * l + e / NW, j = j0 + e % NW;
      if (k >= nk || j >= nphi) continue;
      const int rk = k * nrg + row;
      int jo = j + (ctl.shift ? T.ro[rk].shift.x : 0);
      if (jo >= nphi) jo -= nphi;
      const size_t s = (size_t)rk * nphi + j, o = (size_t)rk * nphi + jo;
      P.ro[o] = P.r[s]; P.uo[o] = P.u[s]; P.vo[o] = P.v[s]; P.wo[o] = P.w[s];
    }
    return;
  }
  const int lim = M.lim, k0 = REAL * l - NPAD, rows = C * M.G;
  const double rad = T.rxc[row];
  const TileWalk W(M, tid);
  const ColMap cm(M, W.cl);
  double *const cw = S.ws[cm.w];
  // every load of the tile in flight before the first is used; a ghost layer
  // below or a fixed one above comes from the ghost tables (no FARGO
  // residual), a mirrored one from its mirror image
  RT a[C][4];
  double rc[C], cs2[C], bs[C], bv[C];
#pragma unroll
  for (int i4 = 0; i4 < C; i4++) {
    const int kr = min(k0 + W.n + i4 * M.step, nk + NPAD - 1);
    rc[i4] = (kr >= 0 && kr < nk) ? T.radc[kr * nrg + row] : rad * T.szc[kr + NPAD];
    if (kr >= 0 && (kr < nk || ntop == 0)) {
      const int km = kr >= nk ? 2 * nk - 1 - kr : kr, rk = km * nrg + row;
      const size_t o = (size_t)rk * nphi + min(j0 + W.cl, nphi - 1);
      a[i4][0] = __ldcg(&P.r[o]);
      a[i4][1] = __ldcg(&P.u[o]);
      a[i4][2] = __ldcg(&P.v[o]);
      a[i4][3] = __ldcg(&P.w[o]);
      cs2[i4] = T.cs2[rk];
      bs[i4] = sizeof(RT) == 4 ? T.sbg[rk] : 0.0;
      bv[i4] = sizeof(RT) == 4 ? T.vbg[rk] : 0.0;
    }
  }
  double snd = 0.0, nu = 0.0;            // of row tid: sound speed (a fixed layer: its square over gamma), viscosity
  double2 turn = make_double2(0.0, 0.0);
  bool fixed = false;
  if (tid < rows) {
    const int kr = min(k0 + tid, nk + NPAD - 1);
    fixed = kr < 0 || (kr >= nk && ntop != 0);
    const int km = kr >= nk ? 2 * nk - 1 - kr : kr, rk = km * nrg + row;
    const int gq = (kr < 0 ? kr + NPAD : kr - nk + NPAD) * T.nr + i;
    snd = fixed ? T.csg[gq] : T.snd[rk];
    turn = !ctl.clk ? turn_call(st.dt, fixed ? 0.0 : T.res_v[rk], fixed ? 0.0 : T.irc[rk], st.pl.vy)
           : fixed  ? ctl.clk->pc.turn
                    : T.turn[rk];
    nu = (kr >= 0 && kr < nk) ? T.nu[rk] : T.nug[gq];
  }
  planet_shm<true>(S.pl, ctl, st, ph);
  in_flight();
  if (!run) return;
  if (tid < rows) {
    const int q = table_pos(tid, C, M.G);
    S.row[R_SND][q] = fixed ? sqrt(ph.gam * snd) : snd;
    S.row[R_CH][q] = turn.x;
    S.row[R_SH][q] = turn.y;
    S.row[R_NU][q] = nu;
  }
#pragma unroll
  for (int i4 = 0; i4 < C; i4++) {
    const int n = W.n + i4 * M.step;
    if (n >= rows) break;
    const int kr = min(k0 + n, nk + NPAD - 1), s = cm.at<C>(n);
    double r, p, vt, vr, vp;
    if (kr < 0 || (kr >= nk && ntop != 0)) {
      const double *g = T.tg + ((size_t)(kr < 0 ? kr + NPAD : NPAD + kr - nk) * T.nr + i) * 4;
      r = g[0]; p = g[1]; vr = g[2]; vp = g[3];
      vt = 0.0;
    } else {
      r = load_r(a[i4][0], bs[i4]);
      vr = (double)a[i4][1];
      vp = load_r(a[i4][2], bv[i4]);
      vt = kr >= nk ? -(double)a[i4][3] : (double)a[i4][3];
      p = EOS == 0 ? r * cs2[i4] : cs2[i4] * pow_call(r, ph.gam) / ph.gam;
    }
    cw[W_R * SLOT + s] = r;
    cw[W_U * SLOT + s] = vt;
    cw[W_V * SLOT + s] = vr;
    cw[W_W * SLOT + s] = vp * rc[i4];
    cw[W_P * SLOT + s] = p;
  }
  __syncthreads();
  {
    const int lane = tid & 31, wid = tid >> 5, pw = min(quot16(lane, M.mG), M.P - 1);
    const PlanetC pl = S.pl;
    Lane<C> L;
    place_lane<C>(L, M, pw, T.ax[2] + (size_t)l * A_COUNT * ARR, S.row[0], S.ws[wid], lane);
    L.dt = st.dt;
    L.rad = rad;
    L.irad = T.irxc[row];
    L.bq = fma(rad, rad, pl.b2);
    {
      const int j = min(j0 + wid * M.P + pw, nphi - 1);
      const double cy = T.cyc[j], sy = T.syc[j];
      L.c0 = fma(cy, pl.cy, sy * pl.sy);
      L.s0 = fma(sy, pl.cy, -(cy * pl.sy));
    }
    {
      double cs[C];
      ld<C>(L, A_IW, cs);
      const double a = 0.5 * st.dt * L.irad;
      if (EOS == 0 && !ODD) {
        double snd[C];
        ld_row<C>(L, R_SND, snd);
        PG_CELLS cs[c] = a * snd[c] * cs[c];
      } else {
        double p[C], r[C];
        get<C>(L, W_P, p);
        get<C>(L, W_R, r);
        PG_CELLS {
          const double x = ph.gam * p[c] * rcp(r[c]);
          cs[c] = a * root(x) * cs[c];
        }
      }
      warp_chain<2, true, EOS, ODD, C>(L, pl, ph, cs);
    }
    if (ph.visc) {
      double a[C], nr[C], n1[C], d1[C], d2[C], dtr[C];
      Deriv<C> D;
      D.load(L);
      get<C>(L, W_R, a);
      ld_row<C>(L, R_NU, nr);
      PG_CELLS {
        nr[c] *= a[c];
        dtr[c] = st.dt * (L.irad * L.irad) * rcp(a[c]);
      }
      D.of(nr, n1, d2);
#pragma unroll 1
      for (int f = W_U; f <= W_V; f++) {
        const double two = f == W_U ? 2.0 : 1.0;
        get<C>(L, f, a);
        D.of(a, d1, d2);
        PG_CELLS a[c] = fma(two * dtr[c], fma(nr[c], d2[c], n1[c] * d1[c]), a[c]);
        put<C>(L, f, a);
      }
    }
  }
  __syncthreads();
  // the polar sweep is the last of a 3D step: the FARGO integer shift of each
  // layer (rotate_rings, ppm.cu:309-322) is applied at this store
  const int len = lim - 2 * NPAD;
  double rate = 0.0;
  bool bad = false;
  if (j0 + W.cl < nphi) {
#pragma unroll 2
    for (int m = W.n; m < len; m += M.step) {
      const int k = k0 + m + NPAD, rk = k * nrg + row, s = cm.at<C>(m + NPAD);
      Finish<RT> F;
      F.template ring<true>(T, ctl, rk);
      int jo = j0 + W.cl + F.shift(ctl);
      if (jo >= nphi) jo -= nphi;
      const double x = F.template cell<true, EOS>(T, P, ctl, ph, (size_t)rk * nphi + jo, jo, cw[W_R * SLOT + s],
                                                  cw[W_V * SLOT + s], quot(cw[W_W * SLOT + s], F.o.rc, F.o.irc),
                                                  cw[W_U * SLOT + s], bad);
      rate = (x > rate || x != x) ? x : rate;
    }
  }
  if (ctl.fuse) report(ctl, rate, bad);
}

template <class RT, int EOS, bool ODD, int C>
__global__ void __launch_bounds__(NT, MINB) k_sweep_z(Tables T, PlanesT<RT> P, Phys ph, SweepCtl ctl, int ntop) {
  extern __shared__ __align__(16) unsigned char shm[];
  after_previous();
  StepIn st;
  const bool run = load_step(ctl, st);
  sweep_z_tile<RT, EOS, ODD, C>(*reinterpret_cast<TileShm *>(shm), T, P, ph, ctl, st, run, ntop, blockIdx.x);
}

// ---------------------------------------------------------------------------
// Batched 2D sweeps: one launch walks the tiles of every run of a group; CTA
// b takes tiles b, b + grid, ...  Each tile runs the same code as in the
// run's own launch, so a run's results depend on neither batch nor grid.
template <class RT>
__device__ __forceinline__ const PlanesT<RT> &batch_planes(const BatchRun &b, int y) {
  if constexpr (sizeof(RT) == 4) return y ? b.QY : b.QX;
  else return y ? b.PY : b.PX;
}

template <class RT>
__global__ void __launch_bounds__(NT, MINB) kb_sweep_x(BatchQueue q) {
  extern __shared__ __align__(16) unsigned char shm[];
  after_previous();
  for (int t = blockIdx.x; t < q.total; t += gridDim.x) {
    const int r = batch_find(q, t);
    const BatchRun &b = q.runs[r];
    SweepCtl ctl{};
    ctl.clk = b.clk;
    StepIn st;
    if (load_step(ctl, st)) {
      PlanesT<RT> P = batch_planes<RT>(b, 0);
      P.p0 = (sizeof(RT) == 8 && b.p0 && b.clk->ncycle == b.p0_cycle) ? b.p0 : nullptr;
      sweep_x_tile<RT, false, 0, false>(*reinterpret_cast<TileShm *>(shm), b.T, P, b.ph, ctl, st, t - q.start[r]);
    }
    __syncthreads();
  }
}

template <class RT>
__global__ void __launch_bounds__(NT, MINB) kb_sweep_y(BatchQueue q) {
  extern __shared__ __align__(16) unsigned char shm[];
  after_previous();
  YShm<0> &S = *reinterpret_cast<YShm<0> *>(shm);
  const int wid = threadIdx.x >> 5;
  for (int t = blockIdx.x; t < q.total; t += gridDim.x) {
    const int r = batch_find(q, t);
    const BatchRun &b = q.runs[r];
    SweepCtl ctl{};
    ctl.clk = b.clk;
    ctl.fuse = 1;
    ctl.shift = 1;
    StepIn st;
    const bool run = load_step(ctl, st);
    planet_shm<false>(S.pl, ctl, st, b.ph);
    sweep_y_task<RT, false, 0>(S.ws[wid], S.pl, b.T, batch_planes<RT>(b, 1), b.ph, ctl, st, run, (t - q.start[r]) * NW + wid);
    __syncthreads();
  }
}

}  // namespace pgd

// ---------------------------------------------------------------------------
namespace pgk {
using namespace pgd;

static int pencils_per_warp(int lim, int C) { return 32 / ((lim + C - 1) / C); }
static int groups(int n, int w) { return (n + w - 1) / w; }

// Cells per lane of the polar sweep: 3 or 4, whichever leaves fewer of the
// warp's cell slots empty.  The 32-layer disk's pencils of 44 cells fill 88 of
// 96 slots with 3 (two pencils of 15 lanes) and 88 of 128 with 4; 28 and 36
// cells fill 112 and 108 of 128 with 4.  Grids of more than one chunk take 4.
// Polar sweep with 3 and 4 cells, us: 128x1024x32 424, 578; 128x512 of 40 layers
// 422, 305; 24: 223, 209; 20: 214, 150; 16: 152, 154; 12: 114, 127.
int polar_cells(const Chunking &ch) {
  if (ch.loop > 1 || ch.stuck) return 4;
  const int lim = ch.lim_last;
  if (lim > 96) return 4;
  return 4 * pencils_per_warp(lim, 3) > 3 * pencils_per_warp(lim, 4) ? 3 : 4;
}

// tiles of a chunk of lim cells (idle: the last chunk of a multiple of 116,
// whose cells are copied) across n pencils
static Tile make_tile(int lim, bool idle, int C, int n) {
  Tile t{};
  t.lim = lim;
  t.G = (lim + C - 1) / C;
  t.P = idle ? 1 : 32 / t.G;
  t.cols = NW * t.P;
  t.step = NT / t.cols;
  t.ng = groups(n, t.cols);
  t.mG = 65536 / t.G + 1;
  t.mP = 65536 / t.P + 1;
  t.mC = 65536 / t.cols + 1;
  t.mng = (1ull << 40) / t.ng + 1;
  return t;
}
void make_tiles(Tables &T) {
  const int rings = T.nr * T.nk, C = polar_cells(T.cz);
  T.tx[0] = make_tile(ARR, false, 4, T.nphi);
  T.tx[1] = make_tile(T.cx.lim_last, T.cx.stuck, 4, T.nphi);
  T.ty[0] = make_tile(ARR, false, 4, rings);
  T.ty[1] = make_tile(T.cy.lim_last, T.cy.stuck, 4, rings);
  T.tz[0] = make_tile(ARR, false, 4, T.nphi);
  T.tz[1] = make_tile(T.cz.lim_last, T.cz.stuck, C, T.nphi);
  T.mnr = (1ull << 40) / T.nr + 1;
}

// CTAs of a run's radial, azimuthal and polar sweep
int tiles_x(const Tables &T) { return T.nk * ((T.cx.loop - 1) * T.tx[0].ng + T.tx[1].ng); }
int tiles_y(const Tables &T) { return (T.cy.loop - 1) * T.ty[0].ng + T.ty[1].ng; }
static int tiles_z(const Tables &T) { return T.nr * ((T.cz.loop - 1) * T.tz[0].ng + T.tz[1].ng); }

// The sweeps' kernels, by plane type, dimension, equation of state, cells per lane
// and whether ghost cells hold no state (Tables::odd).
template <class RT>
using SweepK = void (*)(Tables, PlanesT<RT>, Phys, SweepCtl);
template <class RT>
using SweepZK = void (*)(Tables, PlanesT<RT>, Phys, SweepCtl, int);
template <class RT, bool ODD>
static SweepK<RT> kernel_x(bool three, int eos) {
  if constexpr (sizeof(RT) == 8) {
    if (eos) return three ? k_sweep_x<RT, true, 1, ODD> : k_sweep_x<RT, false, 1, ODD>;
  }
  return three ? k_sweep_x<RT, true, 0, ODD> : k_sweep_x<RT, false, 0, ODD>;
}
template <class RT>
static SweepK<RT> kernel_y(bool three, int eos) {
  if constexpr (sizeof(RT) == 8) {
    if (eos) return three ? k_sweep_y<RT, true, 1> : k_sweep_y<RT, false, 1>;
  }
  return three ? k_sweep_y<RT, true, 0> : k_sweep_y<RT, false, 0>;
}
template <class RT, bool ODD>
static SweepZK<RT> kernel_z(int C, int eos) {
  if constexpr (sizeof(RT) == 8) {
    if (eos) return C == 3 ? k_sweep_z<RT, 1, ODD, 3> : k_sweep_z<RT, 1, ODD, 4>;
  }
  return C == 3 ? k_sweep_z<RT, 0, ODD, 3> : k_sweep_z<RT, 0, ODD, 4>;
}

// The sweeps take their shared blocks as dynamic shared memory, 44.8 KB for a tile
// of 4 warps, below the default limit of 48 KiB.  Naming the kernels to the runtime
// here loads the module in a process's first pg_create (7.5-9 ms of it for 3.4-4.5);
// the first load then takes that much less, 6.5-8.5 ms for 9.5-12.
static_assert(sizeof(TileShm) <= 48 * 1024 && sizeof(YShm<1>) <= sizeof(TileShm), "within the default limit");
template <class RT>
static bool name_kernels() {
  bool ok = true;
  auto name = [&](const void *f) {
    ok = ok && cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TileShm)) == cudaSuccess;
  };
  for (int eos = 0; eos < (sizeof(RT) == 8 ? 2 : 1); eos++)
    for (bool three : {false, true}) {
      name((const void *)kernel_x<RT, false>(three, eos));
      name((const void *)kernel_y<RT>(three, eos));
      name((const void *)kernel_z<RT, false>(three ? 3 : 4, eos));
    }
  name((const void *)kb_sweep_x<RT>);
  name((const void *)kb_sweep_y<RT>);
  return ok;
}
int setup_device() { return name_kernels<double>() && name_kernels<float>() ? 0 : 1; }

void axis_tables(const Tables &T, int ndim, cudaStream_t s) {
  k_axis_table<<<T.cx.loop, ARR, 0, s>>>(T, 0, 4, const_cast<double *>(T.ax[0]));
  k_axis_table<<<T.cy.loop, ARR, 0, s>>>(T, 1, 4, const_cast<double *>(T.ax[1]));
  if (ndim == 3) k_axis_table<<<T.cz.loop, ARR, 0, s>>>(T, 2, polar_cells(T.cz), const_cast<double *>(T.ax[2]));
}
size_t axis_table_elems(const Chunking &ch) { return (size_t)ch.loop * A_COUNT * ARR; }

template <class RT>
void sweep_x(const Tables &T, const PlanesT<RT> &P, const Phys &ph, const SweepCtl &c, int ndim, cudaStream_t s) {
  launch(T.odd & 1 ? kernel_x<RT, true>(ndim == 3, ph.eos) : kernel_x<RT, false>(ndim == 3, ph.eos), tiles_x(T), NT,
         sizeof(TileShm), s, T, P, ph, c);
}

template <class RT>
void sweep_y(const Tables &T, const PlanesT<RT> &P, const Phys &ph, const SweepCtl &c, int ndim, cudaStream_t s) {
  launch(kernel_y<RT>(ndim == 3, ph.eos), tiles_y(T), NT, sizeof(RT) == 8 && ph.eos ? sizeof(YShm<1>) : sizeof(YShm<0>), s, T, P,
         ph, c);
}

template <class RT>
void sweep_z(const Tables &T, const PlanesT<RT> &P, const Phys &ph, const SweepCtl &c, int ntop, cudaStream_t s) {
  const int C = polar_cells(T.cz);
  launch(T.odd & 2 ? kernel_z<RT, true>(C, ph.eos) : kernel_z<RT, false>(C, ph.eos), tiles_z(T), NT, sizeof(TileShm), s, T, P, ph,
         c, ntop);
}

template <class RT>
void batch_sweep_x(const BatchQueue &q, int grid, cudaStream_t s) {
  if (q.total > 0) launch(kb_sweep_x<RT>, grid > 0 && grid < q.total ? grid : q.total, NT, sizeof(TileShm), s, q);
}
template <class RT>
void batch_sweep_y(const BatchQueue &q, int grid, cudaStream_t s) {
  if (q.total > 0) launch(kb_sweep_y<RT>, grid > 0 && grid < q.total ? grid : q.total, NT, sizeof(YShm<0>), s, q);
}

#define PG_SWEEPS(RT)                                                                                              \
  template void sweep_x<RT>(const Tables &, const PlanesT<RT> &, const Phys &, const SweepCtl &, int, cudaStream_t); \
  template void sweep_y<RT>(const Tables &, const PlanesT<RT> &, const Phys &, const SweepCtl &, int, cudaStream_t); \
  template void sweep_z<RT>(const Tables &, const PlanesT<RT> &, const Phys &, const SweepCtl &, int, cudaStream_t); \
  template void batch_sweep_x<RT>(const BatchQueue &, int, cudaStream_t);                                            \
  template void batch_sweep_y<RT>(const BatchQueue &, int, cudaStream_t);
PG_SWEEPS(double)
PG_SWEEPS(float)

}  // namespace pgk
