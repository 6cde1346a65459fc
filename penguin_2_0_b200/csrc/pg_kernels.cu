// pg_kernels.cu -- sm_100a kernels around the sweeps (those are pg_sweep.cu).
//
//   k_tables    per-ring, per-column and per-layer tables
//   k_cfl       CFL rate max (dt_lv1, timestep.cu:12-73)
//   k_damp      wave damping
//   k_index     Index_Shift (orbital_advection.cu:12-43)
//   k_reduce    output_lv1/lv2/lv3 (device_func.cu:49-167) in the same tree
//               order, finished by the last CTA
//   k_prestep / k_poststep  the scalar part of main.cu:343-441 on device
#include "pg_kernels.cuh"

namespace pgd {

// ordered encoding of a non-negative double (NaN sorts above +inf)
__device__ __forceinline__ unsigned long long dbits(double x) {
  return (unsigned long long)__double_as_longlong(x);
}

__device__ __forceinline__ double block_max(double v, double *red) {
  // reduce within the CTA; only thread 0's result is meaningful
  for (int o = 16; o > 0; o >>= 1) {
    double t = __shfl_down_sync(0xffffffffu, v, o);
    v = (t > v || t != t) ? t : v;
  }
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) red[wid] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    int nw = (blockDim.x + 31) >> 5;
    for (int i = 1; i < nw; i++) v = (red[i] > v || red[i] != red[i]) ? red[i] : v;
  }
  return v;
}

// ---------------------------------------------------------------------------
// tables: cs2, nu and the damping factors per ring, on the device so that
// they carry the same bits as the reference's inline get_cs2/get_nu calls
__global__ void k_tables(Tables T, Phys ph, int ndim, double kill_rin, double kill_rout,
                         double xmin, double xmax) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  int n = T.nk * T.nrg;
  const int nz = T.nk + 2 * NPAD;
  if (t < nz) {
    const_cast<double *>(T.szc)[t] = sin(T.zc[t]);
    const_cast<double *>(T.idz)[t] = 1.0 / T.dz[t];
  }
  if (t < T.nrg) {
    const_cast<double *>(T.irdx)[t] = 1.0 / T.rdx[t];
    const_cast<double *>(T.irxc)[t] = 1.0 / T.rxc[t];
  }
  if (t < T.nphi) {
    const_cast<double *>(T.idy)[t] = 1.0 / T.dy[t];
    const_cast<double *>(T.cyc)[t] = cos(T.yc[t]);
    const_cast<double *>(T.syc)[t] = sin(T.yc[t]);
  }
  if (ndim == 3 && t < 2 * NPAD * T.nr) {
    // nu at r sin(theta) of the 12 polar ghost layers of ring i (slot g:
    // layer g - 6 below the grid, or layer nk + g - 6 above it), the
    // expression the polar viscosity uses for them (get_nu
    // disk_profile.cu:149-152)
    const int i = t % T.nr, g = t / T.nr;
    const int kz = (g < NPAD) ? g : T.nk + g;          // ghost layer + NPAD
    const double rcg = T.rxc[i + NPAD] * sin(T.zc[kz]);    // T.szc[kz], which this launch writes
    const_cast<double *>(T.nug)[t] = ph.vis_nu * pow(rcg, ph.p_alpha);
    // cs2 of the fixed layer's state, p = rho cs2 (used where the layer's
    // state is: isothermal runs)
    const_cast<double *>(T.csg)[t] = T.tg[4 * (size_t)t + 1] / T.tg[4 * (size_t)t];
  }
  if (t >= n) return;
  int k = t / T.nrg, row = t % T.nrg;
  double rad = T.rxc[row];
  double rc = rad;
  if (ndim == 3) rc *= sin(T.zc[k + NPAD]);
  double *radc = const_cast<double *>(T.radc);
  double *cs2 = const_cast<double *>(T.cs2);
  double *nu = const_cast<double *>(T.nu);
  double *dg = const_cast<double *>(T.damp_g);
  double *dp = const_cast<double *>(T.damp_pw);
  radc[t] = rc;
  cs2[t] = ph.sc2 * pow(rc, -ph.p_beta);          // get_cs2 disk_profile.cu:39-42
  const_cast<double *>(T.irc)[t] = 1.0 / rc;
  const_cast<double *>(T.snd)[t] = sqrt(ph.gam * cs2[t]);
  nu[t] = ph.vis_nu * pow(rc, ph.p_alpha);        // get_nu disk_profile.cu:149-152
  double g = 0.0;
  bool interior = row >= NPAD && row < T.nr + NPAD;
  if (interior) {
    double r = rad;
    if (kill_rin > 0.0 && r < kill_rin) g = (kill_rin - r) / (kill_rin - xmin);
    else if (kill_rout > 0.0 && r > kill_rout) g = (r - kill_rout) / (xmax - kill_rout);
  }
  dg[t] = g;
  dp[t] = pow(rad, -1.5);
}

// CFL rate (dt_lv1 timestep.cu:12-73), one CTA per ring.  In the device loop
// (clk) FrRot, the target and the halt flag come from the clock, the cells
// are checked, and rot_j may still lack the step's shift (rot_pending).
template <class RT>
__global__ void k_cfl(Tables T, const RT *R, const RT *U, const RT *V, const RT *W, const double *P0, Phys ph,
                      double frrot, int ndim, unsigned long long *out, DevClock *clk, int rot_pending) {
  __shared__ double red[32];
  if (clk) {
    if (clk->halted) return;
    frrot = clk->frrot_next;
    out = &clk->cfl_bits;
  }
  const int i = blockIdx.x, k = blockIdx.y;
  const int row = i + NPAD, rk = k * T.nrg + row;
  const size_t base = (size_t)rk * T.nphi;
  const double bs = sizeof(RT) == 4 ? T.sbg[rk] : 0.0, bv = sizeof(RT) == 4 ? T.vbg[rk] : 0.0;
  const double irdx = T.irdx[row], irc = T.irc[rk], off = __fma_rn(frrot, T.radc[rk], T.rot_v[rk]);
  const double iwz = ndim == 3 ? __dmul_rn(T.idz[k + NPAD], T.irxc[row]) : 0.0;
  const int rotn = T.rot_j[rk] + (rot_pending ? T.inc_j[rk] : 0);
  double rate = 0.0;
  bool bad = false;
  for (int j = threadIdx.x; j < T.nphi; j += blockDim.x) {
    // physical column j holds storage index js = j - rot_j
    const int js = wrapm(j - rotn, T.nphi);
    const double r = load_r(R[base + j], bs), v = load_r(V[base + j], bv), u = (double)U[base + j];
    const double cs = P0 ? sound_speed(r, P0[base + j], ph)
                         : ph.eos ? sound_speed(r, eos_p<1>(r, T.cs2[rk], ph), ph) : T.snd[rk];
    const double iwy = __dmul_rn(T.idy[js], irc);
    const double rt = ndim == 3 ? cfl_rate<true>(cs, u, irdx, __dsub_rn(v, off), iwy, (double)W[base + j], iwz)
                                : cfl_rate<false>(cs, u, irdx, __dsub_rn(v, off), iwy, 0.0, 0.0);
    rate = (rt > rate || rt != rt) ? rt : rate;
    if (!(r > 0.0) || !isfinite(r) || !isfinite(u) || !isfinite(v)) bad = true;
  }
  double m = block_max(rate, red);
  int anybad = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    if (m > 0.0 || m != m) atomicMax(out, dbits(m));
    if (clk && anybad) atomicExch(&clk->status, 3);
  }
}

// Index_Shift orbital_advection.cu:12-43 for every interior ring
__device__ __forceinline__ void index_shift_ring(const Tables &T, int t, double dt, double FrRot, int fargo) {
  int k = t / T.nr, i = t % T.nr;
  int row = i + NPAD, rk = k * T.nrg + row;
  double xc = T.rxc[row];
  double widthy = xc * T.dy[0] / dt;
  double rot_v;
  if (fargo == 1) rot_v = T.val_v[rk] - FrRot * xc;
  else if (fargo == 2) rot_v = (1.0 - FrRot) * xc;
  else rot_v = 0.0;
  double jp = T.rot_v[rk] / widthy;
  if (jp >= 0.0) { T.inc_j[rk] = (int)(jp + 0.5); T.res_v[rk] = floor(jp + 0.5) * widthy; }
  else { T.inc_j[rk] = (int)(jp - 0.5); T.res_v[rk] = floor(jp + 0.5) * widthy; }
  T.rot_v[rk] = rot_v;
}

__global__ void k_index(Tables T, double dt, double frrot, int fargo, const DevClock *clk) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (clk) {
    if (clk->halted) return;
    dt = clk->dt_step;
    frrot = clk->frrot_next;  // unused path; the fused loop shifts in k_prestep
  }
  if (t >= T.nr * T.nk) return;
  index_shift_ring(T, t, dt, frrot, fargo);
}

// rotate_rings ppm.cu:309-322
__global__ void k_rotate(Tables T, const DevClock *clk) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (clk && clk->halted) return;
  if (t >= T.nr * T.nk) return;
  int k = t / T.nr, i = t % T.nr;
  int rk = k * T.nrg + i + NPAD;
  int j = T.rot_j[rk] + T.inc_j[rk];
  T.rot_j[rk] = wrap1(j, T.nphi);
}

// wave damping by dt, or by the clock's step: the rule and the bits of the
// last sweep's epilogue
template <class RT>
__global__ void k_damp(Tables T, RT *R, RT *U, RT *V, RT *W, double dt, const DevClock *clk, int ndim) {
  if (clk) {
    if (clk->halted) return;
    dt = clk->dt_step;
  }
  const int i = blockIdx.x, k = blockIdx.y;
  const int rk = k * T.nrg + i + NPAD;
  const double g = T.damp_g[rk];
  if (!(g > 0.0)) return;
  const double f = g * (dt * T.damp_pw[rk]);
  const size_t base = (size_t)rk * T.nphi;
  const double vr = T.val_r[rk], vu = T.val_u[rk], vv = T.val_v[rk];
  const double bs = sizeof(RT) == 4 ? T.sbg[rk] : 0.0, bv = sizeof(RT) == 4 ? T.vbg[rk] : 0.0;
  for (int j = threadIdx.x; j < T.nphi; j += blockDim.x) {
    const size_t o = base + j;
    R[o] = store_r<RT>(damped(load_r(R[o], bs), vr, f), bs);
    U[o] = (RT)damped((double)U[o], vu, f);
    V[o] = store_r<RT>(damped(load_r(V[o], bv), vv, f), bv);
    if (ndim == 3) W[o] = (RT)damped((double)W[o], 0.0, f);
  }
}

// ---------------------------------------------------------------------------
// output_lv1 (per ring, 1024 threads, storage order, bin_reduc_sum per 1024
// cells, running sum across chunks), output_lv2 (3D: round_reduc_sum over
// k) and output_lv3 (bin_reduc_sum over <=1024 rings) of device_func.cu.
// The last CTA to finish does lv2/lv3, so one launch gives the final value.
__device__ __forceinline__ double tree1024(double *list) {
  for (int len = 1024; len > 1; len >>= 1) {
    int half = len >> 1;
    if ((int)threadIdx.x < half) list[threadIdx.x] += list[threadIdx.x + half];
    __syncthreads();
  }
  return list[0];
}

// Rings t0, t0 + tstep, ... (t = i + nr * k: ring i of polar layer k), each
// summed on its own as one CTA of the reference sums it; the last of the
// run's nblocks CTAs to finish adds up the run's partial sums.
template <typename RT>
__device__ __forceinline__ void reduce_body(const Tables &T, const RT *R, Body pl, const DevClock *clk,
                                            double exclude, int mode, int plnt, double p_alpha, int ndim,
                                            double *ring_part, unsigned int *counter, double *out,
                                            double *hist_row, int t0, int tstep, unsigned nblocks,
                                            bool every_step = false) {
  __shared__ double list[1024];
  __shared__ bool is_last;
  if (clk) {
    if (!every_step && !clk->prin) return;
    if (every_step && clk->halted) return;
    pl = clk->planet;
  }
  const int tt = threadIdx.x;
  for (int rt = t0; rt < T.nr * T.nk; rt += tstep) {
    const int i = rt % T.nr, k = rt / T.nr;
    const int row = i + NPAD, rk = k * T.nrg + row;
    const int nphi = T.nphi;
    const size_t base = (size_t)rk * nphi;
    const int rot = T.rot_j[rk];
    const double rad = T.rxc[row], xvol = T.rxvol[row];
    const double zvol = (ndim == 3) ? T.zvol[k + NPAD] : 1.0;
    // FP32 planes hold Sigma - S_bg(ring)
    const double r_off = (sizeof(RT) == 4) ? T.sbg[rk] : 0.0;
    const int loop = nphi / 1024 + (nphi % 1024 != 0);
    double val = 0.0;
    for (int l = 0; l < loop; l++) {
      int j = tt + 1024 * l;   // storage index
      double v = 0.0;
      if (j < nphi) {
        int j0 = wrap1(j + rot, nphi);
        double phi = T.yc[j0];
        double r = r_off + (double)R[base + j0];
        if (plnt) {
          if (mode == 0) v = r * xvol * T.yvol[j0] * zvol;
          else if (ndim == 2 && (mode == 8 || mode == 9)) {
            if ((rad - pl.x) * (rad - pl.x) + rad * rad * (phi - pl.y) * (phi - pl.y) > exclude * exclude) {
              if (mode == 8) {
                double t = -grav_rad_cyl(rad, phi, 0.0, pl, 0.0);
                t *= (r - pow(rad, -p_alpha)) * xvol * T.yvol[j0];
                v = t;
              } else {
                double t = -grav_azi_cyl(rad, phi, 0.0, pl, 0.0);
                t *= rad * (r - pow(rad, -p_alpha)) * xvol * T.yvol[j0];
                v = t;
              }
            }
          }
        } else {
          v = r * xvol * T.yvol[j0] * zvol;
        }
      }
      list[tt] = v;
      __syncthreads();
      double s = tree1024(list);
      if (tt == 0) val += s;
      __syncthreads();
    }
    if (tt == 0) ring_part[i + T.nr * k] = val;
  }
  if (tt == 0) {
    __threadfence();
    unsigned int prev = atomicAdd(counter, 1u);
    is_last = (prev == nblocks - 1);
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  // lv2 (3D): round_reduc_sum over k per ring i, reduction.cu:77-100
  const volatile double *part = ring_part;
  int nr = T.nr, nk = T.nk;
  // lv3: rings in chunks of 1024 (the reference supports iblk <= 1024)
  double total = 0.0;
  for (int base_i = 0; base_i < nr; base_i += 1024) {
    int ii = base_i + tt;
    double v = 0.0;
    if (ii < nr) {
      if (ndim == 3) {
        // pairwise tree over k with the reference's half-point order
        double acc[64];
        int kk = nk < 64 ? nk : 64;
        for (int q = 0; q < kk; q++) acc[q] = part[ii + nr * q];
        int len2 = 1;
        while (len2 < nk) len2 *= 2;
        while (len2 > 1) {
          int half = len2 / 2;
          for (int q = 0; q < half; q++) if (q + half < kk) acc[q] += acc[q + half];
          len2 = half;
        }
        v = acc[0];
      } else {
        v = part[ii];
      }
    }
    list[tt] = v;
    __syncthreads();
    double s = tree1024(list);
    if (tt == 0) total += s;
    __syncthreads();
  }
  if (tt == 0) {
    double res = 0.0 + total;
    if (out) *out = res;
    (void)hist_row;
    *counter = 0u;
  }
}

// ---------------------------------------------------------------------------
// Mass sums of runs with many rings: one warp per ring (RW rings per CTA).
// Lane L holds list[L + 32 m], m = 0..31, of a 1024-cell block, its 32 loads
// issued together; tree1024's levels 512..32 pair values inside a lane and
// levels 16..1 across lanes by shuffle.  Every addition has the same two
// operands as in tree1024, and __dadd_rn keeps the cell's product from being
// fused into the first one, so the sums are bitwise those of reduce_body.
// Used where cells are cheap (mass) and rings plentiful; the force sums and
// small runs keep reduce_body's one cell per thread.
constexpr int RW = 4;
__device__ __forceinline__ double warp_tree1024(double (&v)[32]) {
#pragma unroll
  for (int h = 16; h >= 1; h >>= 1) {
#pragma unroll
    for (int m = 0; m < h; m++) v[m] = __dadd_rn(v[m], v[m + h]);
  }
  double x = v[0];
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int d = 16; d >= 1; d >>= 1) {
    const double y = __shfl_down_sync(0xffffffffu, x, d);
    if (lane < d) x = __dadd_rn(x, y);
  }
  return x;   // lane 0: the block's sum
}

template <typename RT>
__global__ void __launch_bounds__(32 * RW) k_reduce_mass_w(Tables T, const RT *R, const DevClock *clk, int ndim,
                                                           double *ring_part, unsigned int *counter, double *out) {
  __shared__ double list[1024];
  __shared__ bool is_last;
  if (clk && !clk->prin) return;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int nr = T.nr, nk = T.nk, nphi = T.nphi;
  for (int rt = blockIdx.x * RW + w; rt < nr * nk; rt += gridDim.x * RW) {
    const int i = rt % nr, k = rt / nr;
    const int row = i + NPAD, rk = k * T.nrg + row;
    const size_t base = (size_t)rk * nphi;
    const int rot = T.rot_j[rk];
    const double xvol = T.rxvol[row];
    const double zvol = (ndim == 3) ? T.zvol[k + NPAD] : 1.0;
    // FP32 planes hold Sigma - S_bg(ring)
    const double r_off = (sizeof(RT) == 4) ? T.sbg[rk] : 0.0;
    const int loop = nphi / 1024 + (nphi % 1024 != 0);
    double val = 0.0;
    for (int l = 0; l < loop; l++) {
      double v[32];
#pragma unroll
      for (int m = 0; m < 32; m++) {
        const int j = lane + 32 * m + 1024 * l;   // storage index
        double x = 0.0;
        if (j < nphi) {
          const int j0 = wrap1(j + rot, nphi);
          const double r = r_off + (double)R[base + j0];
          x = r * xvol * T.yvol[j0] * zvol;
        }
        v[m] = x;
      }
      const double sum = warp_tree1024(v);
      if (lane == 0) val += sum;
    }
    if (lane == 0) ring_part[i + nr * k] = val;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    unsigned int prev = atomicAdd(counter, 1u);
    is_last = (prev == gridDim.x - 1);
  }
  __syncthreads();
  if (!is_last) return;
  __threadfence();
  // lv2 (3D: round_reduc_sum over k per ring, reduction.cu:77-100), then lv3
  // over the rings in blocks of 1024, as reduce_body
  const volatile double *part = ring_part;
  double total = 0.0;
  for (int base_i = 0; base_i < nr; base_i += 1024) {
    for (int q4 = threadIdx.x; q4 < 1024; q4 += 32 * RW) {
      const int ii = base_i + q4;
      double v = 0.0;
      if (ii < nr) {
        if (ndim == 3) {
          double acc[64];
          int kk = nk < 64 ? nk : 64;
          for (int q = 0; q < kk; q++) acc[q] = part[ii + nr * q];
          int len2 = 1;
          while (len2 < nk) len2 *= 2;
          while (len2 > 1) {
            int half = len2 / 2;
            for (int q = 0; q < half; q++) if (q + half < kk) acc[q] += acc[q + half];
            len2 = half;
          }
          v = acc[0];
        } else {
          v = part[ii];
        }
      }
      list[q4] = v;
    }
    __syncthreads();
    if (w == 0) {
      double v[32];
#pragma unroll
      for (int m = 0; m < 32; m++) v[m] = list[lane + 32 * m];
      const double sum = warp_tree1024(v);
      if (lane == 0) total += sum;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    double res = 0.0 + total;
    if (out) *out = res;
    *counter = 0u;
  }
}

template <typename RT>
__global__ void __launch_bounds__(1024) k_reduce(Tables T, const RT *R, Body pl, const DevClock *clk,
                                                 double exclude, int mode, int plnt, double p_alpha,
                                                 int ndim, double *ring_part, unsigned int *counter,
                                                 double *out, double *hist_row) {
  reduce_body<RT>(T, R, pl, clk, exclude, mode, plnt, p_alpha, ndim, ring_part, counter, out, hist_row,
                  blockIdx.x, gridDim.x, gridDim.x);
}

// moving planet: the disk's radial (mode 8) and azimuthal (mode 9) force
// sums on the drifted planet, every step, into the clock
template <typename RT>
__global__ void __launch_bounds__(1024) k_reduce_forces(Tables T, const RT *R, DevClock *clk, int mode,
                                                        double p_alpha, int ndim, double *ring_part,
                                                        unsigned int *counter) {
  reduce_body<RT>(T, R, Body{}, clk, 0.0, mode, 1, p_alpha, ndim, ring_part, counter,
                  mode == 8 ? &clk->f8 : &clk->f9, nullptr, blockIdx.x, gridDim.x, gridDim.x, true);
}

// append a diagnostics row when this step prints (main.cu:414-428)
__device__ __forceinline__ void record_body(DevClock *clk) {
  DevClock &c = *clk;
  if (!c.prin) return;
  if (c.hist && c.hist_count < c.hist_cap) {
    double *h = c.hist + (size_t)HIST_COLS * c.hist_count;
    Body &p = c.planet;
    double vy = p.vy + c.frrot;
    double L = vy * p.x * p.x;                                        // get_L planet.cu:11-15
    double E = (p.vx * p.vx + vy * vy * p.x * p.x) / 2.0 - 1.0 / p.x; // get_E planet.cu:17-21
    h[0] = c.simtime;
    h[1] = c.mass;
    h[2] = c.torque / c.hist_norm;
    h[3] = p.x; h[4] = p.y; h[5] = p.vx; h[6] = p.vy; h[7] = p.fx; h[8] = p.fy;
    h[9] = sqrt(1.0 + (2.0 * E * L * L));
    h[10] = -1.0 / (2.0 * E);
    c.hist_count += 1;
  }
  c.prin = 0;
}

__global__ void k_record(DevClock *clk) { record_body(clk); }

// ---------------------------------------------------------------------------
// planet (planet.cu:28-93), device copies of the host arithmetic
__device__ double d_set_M_p(const DevClock &c, double t) {
  if (t < c.t_growth) return fmax(c.M_p * sin(3.1415926535897932384626433832795 * t / (2.0 * c.t_growth)), 0.01 * 0.000003);
  return c.M_p;
}
__device__ void d_kick(Body &pl, double &FrRot, double dt, int frflag) {
  pl.vx += dt * pl.fx;
  pl.vy += FrRot + dt * pl.fy / pl.x / pl.x;
  FrRot = (frflag == 1) ? pl.vy : 0.0;
  pl.vy -= FrRot;
}
// The planet's arithmetic is host code in the reference (planet.cu), whose
// compiler folds pow with the constant exponents 0, 1, -1 and 2 into 1, x,
// 1/x and x*x; the device copies below use the same forms (other exponents
// stay pow calls), and round products that feed a sum on their own, as the
// host does.
__device__ __forceinline__ double pow_host_form(double x, double y) {
  if (y == 0.0) return 1.0;
  if (y == 1.0) return x;
  if (y == -1.0) return 1.0 / x;
  if (y == 2.0) return __dmul_rn(x, x);
  return pow(x, y);
}
__device__ void d_drift(Body &pl, double FrRot, double dt, const DevClock &c) {
  double old_rad = pl.x;
  pl.x += dt * pl.vx;
  pl.y += dt * pl.vy;
  pl.vy = ((pl.vy + FrRot) * old_rad * old_rad / pl.x / pl.x) - FrRot;
  if (pl.y < 0.0) pl.y += 6.283185307179586476925286766559;
  if (pl.y >= 6.283185307179586476925286766559) pl.y -= 6.283185307179586476925286766559;
  // rs = rs_fac*get_h(x), get_h = sqrt(cs2(x) x^3); cs2 = sc2 * x^-p_beta is
  // evaluated on the host for the fixed-orbit case and never changes there
  (void)c;
}
// moving planet: the drift moves x, and the softening follows it as
// kick_drift_kick does on the host, rs = rs_fac h(x), h = sqrt(cs2(x) x^3)
// with cs2 = sc_h^2 x^-p_beta (disk_profile.cu:39-52)
__device__ void d_drift_moving(Body &pl, double FrRot, double dt, const DevClock &c) {
  d_drift(pl, FrRot, dt, c);
  pl.rs = c.rs_fac * sqrt(c.sc2 * pow_host_form(pl.x, -c.p_beta) * pl.x * pl.x * pl.x);
}
__device__ void d_forces_fixed(Body &pl, double FrRot) {
  pl.fx = -1.0 / pl.x / pl.x + __dmul_rn(pl.x, pow_host_form(pl.vy + FrRot, 2.0));
  pl.fy = 0.0;
}

// get_dt host part + dt clipping + Index_Shift + half kick (main.cu:345-370)
__device__ __forceinline__ void prestep_body(DevClock *clk, const Tables &T, int fargo) {
  __shared__ double s_dt, s_frrot;
  __shared__ int s_run;
  if (threadIdx.x == 0) {
    DevClock &c = *clk;
    int run = !(c.halted || c.done);
    if (run && c.status != 0) { c.halted = 1; run = 0; }
    if (run) {
      double rate = __longlong_as_double((long long)c.cfl_bits);
      double hdt = c.courant / rate;               // dt_lv3 timestep.cu:105
      double dt = 1.1 * c.dt;                      // timestep.cu:135-141
      dt = (hdt < dt) ? hdt : dt;
      if (dt / c.endtime < 1.0e-12 || !(dt > 0.0)) { c.status = 4; c.halted = 1; run = 0; }
      else {
        c.prin = 0;
        if (c.ncycle == c.ncycend) { c.prin = 1; c.done = 1; }
        if (c.simtime + dt >= c.endtime) {
          c.old_dt = dt; dt = c.endtime - c.simtime; c.prin = 1; c.make_pict = 1; c.done = 1;
        }
        if (c.timem + dt >= c.tmovie) { c.old_dt = dt; dt = c.tmovie - c.timem; c.make_pict = 1; }
        c.dt = dt;
        c.dt_step = dt;
        s_dt = dt;
        s_frrot = c.frrot;   // Index_Shift sees FrRot before the kick
        // kick_drift_kick(planet, FrRot, ..., 0.5*dt, true) main.cu:370
        if (c.plnt_flag > 0) d_kick(c.planet, c.frrot, 0.5 * dt, c.frrot_flag);
        // FrRot at the next get_dt, for the fused CFL: replay drift, forces
        // and kick on copies (fixed planet: forces are analytic)
        Body b = c.planet;
        double fr = c.frrot;
        if (c.plnt_flag > 0) {
          d_drift(b, fr, dt, c);
          d_forces_fixed(b, fr);
          d_kick(b, fr, 0.5 * dt, c.frrot_flag);
        }
        c.frrot_next = fr;
        c.cfl_bits = 0ull;
      }
    }
    s_run = run;
  }
  __syncthreads();
  if (!s_run) return;
  for (int t = threadIdx.x; t < T.nr * T.nk; t += blockDim.x) index_shift_ring(T, t, s_dt, s_frrot, fargo);
}

__global__ void k_prestep(DevClock *clk, Tables T, int fargo) { prestep_body(clk, T, fargo); }

// simtime/drift/forces/kick/dump bookkeeping (main.cu:378-412)
// phase 0: the whole end of a step; with a moving planet phase 1 (rotation,
// time, drift, mass) and phase 2 (forces from the disk reductions f8, f9
// made between the two, kick, bookkeeping; planet.cu:54-93, main.cu:378-412)
__device__ __forceinline__ void poststep_body(DevClock *clk, const Tables &T, int phase = 0) {
  int t = threadIdx.x;
  DevClock &c = *clk;
  int halted = c.halted;
  __syncthreads();
  if (halted) return;
  // rotate_rings ppm.cu:309-322
  for (int q = t; phase != 2 && q < T.nr * T.nk; q += blockDim.x) {
    int k = q / T.nr, i = q % T.nr;
    int rk = k * T.nrg + i + NPAD;
    T.rot_j[rk] = wrap1(T.rot_j[rk] + T.inc_j[rk], T.nphi);
  }
  if (t != 0) return;
  double dt = c.dt_step;
  if (phase != 2) {
    c.simtime += dt;
    c.timem += dt;
    c.ncycle += 1;
    c.ncycp += 1;
  }
  if (phase == 0) {
    if (c.plnt_flag > 0) {
      d_drift(c.planet, c.frrot, dt, c);
      c.planet.m = d_set_M_p(c, c.simtime);
      d_forces_fixed(c.planet, c.frrot);
      d_kick(c.planet, c.frrot, 0.5 * dt, c.frrot_flag);
    }
  } else if (phase == 1) {
    d_drift_moving(c.planet, c.frrot, dt, c);
    c.planet.m = d_set_M_p(c, c.simtime);
    return;
  } else {
    // planet_forces planet.cu:58-59 with the disk sums of this state
    Body &p = c.planet;
    p.fx = c.Sigma_0 * c.f8 / p.m - 1.0 / p.x / p.x + __dmul_rn(p.x, pow_host_form(p.vy + c.frrot, 2.0));
    p.fy = c.Sigma_0 * c.f9 / p.m;
    d_kick(p, c.frrot, 0.5 * dt, c.frrot_flag);
    c.frrot_next = c.frrot;      // the CFL of the next get_dt runs after this kernel
  }
  if (c.ncycp == c.nprin) { c.ncycp = 0; c.prin = 1; }
  if (c.make_pict) {
    c.timem = 0.0;
    c.make_pict = 0;
    c.dt = c.old_dt;
    c.halted = 1;   // the host dumps before continuing
  }
  if (c.done) c.halted = 1;
}

__global__ void k_poststep(DevClock *clk, Tables T) { poststep_body(clk, T); }
__global__ void k_poststep_drift(DevClock *clk, Tables T) { poststep_body(clk, T, 1); }
__global__ void k_poststep_kick(DevClock *clk, Tables T) { poststep_body(clk, T, 2); }

// ---------------------------------------------------------------------------
// Dump <-> planes.  The dump holds each ring's field arrays in storage order
// (j_store = j_phys - rot_j, init.cpp:241, output.cu:48-55); the planes hold
// physical order.  Thread (j, ring i, layer k) moves one cell.
__global__ void k_unpack_dump(Tables T, const double *stage, DumpPlanes D, int ndim, int fp32, int *err) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y, k = blockIdx.z;
  const int nphi = T.nphi;
  if (j >= nphi) return;
  const int rk = k * T.nrg + i + NPAD;
  int jp = j + T.rot_j[rk];
  if (jp >= nphi) jp -= nphi;
  const double *f = stage + ((size_t)i + (size_t)T.nr * k) * 5 * nphi;
  const double r = f[j], p = f[nphi + j], u = f[2 * nphi + j], v = f[3 * nphi + j], w = f[4 * nphi + j];
  if (!(r > 0.0) || !isfinite(r)) atomicOr(err, 1);
  if (ndim == 2 && w != 0.0) atomicOr(err, 2);
  const size_t o = (size_t)rk * nphi + jp;
  if (fp32) {
    D.fr[o] = (float)(r - T.sbg[rk]);
    D.fu[o] = (float)u;
    D.fv[o] = (float)(v - T.vbg[rk]);
    if (ndim == 3) D.fw[o] = (float)w;
  } else {
    D.r[o] = r; D.u[o] = u; D.v[o] = v; D.p0[o] = p;
    if (ndim == 3) D.w[o] = w;
  }
}

// the fixed radial ghost rings (init_bound, init.cpp:253-413): phi-uniform
// r, u, v, p per ghost row, w = 0
__global__ void k_fill_ghost_rows(Tables T, const double *ghosts, DumpPlanes D, int ndim, int fp32) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, gi = blockIdx.y, k = blockIdx.z;
  if (j >= T.nphi) return;
  const int row = gi < NPAD ? gi : T.nr + gi;
  const int rk = k * T.nrg + row;
  const double *g = ghosts + ((size_t)k * 2 * NPAD + gi) * 4;
  const size_t o = (size_t)rk * T.nphi + j;
  if (fp32) {
    D.fr[o] = (float)(g[0] - T.sbg[rk]);
    D.fu[o] = (float)g[1];
    D.fv[o] = (float)(g[2] - T.vbg[rk]);
    if (ndim == 3) D.fw[o] = 0.f;
  } else {
    D.r[o] = g[0]; D.u[o] = g[1]; D.v[o] = g[2]; D.p0[o] = g[3];
    if (ndim == 3) D.w[o] = 0.0;
  }
}

// whole ring records (72*nphi + 96 bytes) in the dump layout
__global__ void k_pack_dump(Tables T, DumpPlanes D, Phys ph, int ndim, int fp32, int p0_live, unsigned char *out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y, k = blockIdx.z;
  const int nphi = T.nphi, row = i + NPAD, rk = k * T.nrg + row, kz = k + NPAD;
  if (j >= nphi) return;
  unsigned char *base = out + ((size_t)i + (size_t)T.nr * k) * ((size_t)72 * nphi + 96);
  int jp = j + T.rot_j[rk];
  if (jp >= nphi) jp -= nphi;
  const size_t o = (size_t)rk * nphi + jp;
  double *f = (double *)base;
  double r, u, v, w;
  if (fp32) {
    r = T.sbg[rk] + (double)D.fr[o];
    u = D.fu[o];
    v = T.vbg[rk] + (double)D.fv[o];
    w = (ndim == 3) ? (double)D.fw[o] : 0.0;
  } else {
    r = D.r[o]; u = D.u[o]; v = D.v[o];
    w = (ndim == 3) ? D.w[o] : 0.0;
  }
  f[j] = r;
  f[nphi + j] = p0_live ? D.p0[o] : eos_p_rt(r, T.cs2[rk], ph);   // the store's p, ppm.cu:138-143
  f[2 * nphi + j] = u;
  f[3 * nphi + j] = v;
  f[4 * nphi + j] = w;
  double *col = (double *)(base + (size_t)40 * nphi + 32);
  col[j] = T.y[j]; col[nphi + j] = T.dy[j]; col[2 * nphi + j] = T.yvol[j]; col[3 * nphi + j] = T.yc[j];
  if (j == 0) {
    double *sc = (double *)(base + (size_t)40 * nphi);
    sc[0] = T.rx[row]; sc[1] = T.rdx[row]; sc[2] = T.rxvol[row]; sc[3] = T.rxc[row];
    double *zs = (double *)(base + (size_t)72 * nphi + 32);
    zs[0] = T.z[kz]; zs[1] = T.dz[kz]; zs[2] = T.zvol[kz]; zs[3] = T.zc[kz];
    int *ik = (int *)(base + (size_t)72 * nphi + 64);
    ik[0] = i; ik[1] = k;
    double *rot = (double *)(base + (size_t)72 * nphi + 72);
    rot[0] = T.rot_v[rk]; rot[1] = T.res_v[rk];
    int *rj = (int *)(base + (size_t)72 * nphi + 88);
    rj[0] = T.rot_j[rk]; rj[1] = T.inc_j[rk];
  }
}

// ---------------------------------------------------------------------------
// Post-processing of a state (the reference's read/ tools, on the device).
// Both work on the physical-order planes, which is what read/p_init.cpp:108-133
// (update_grid) builds from a dump by undoing each ring's rot_j.
__device__ __forceinline__ double block_sum(double v, double *red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  __syncthreads();
  if (lane == 0) red[wid] = v;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += red[w];
  return t;
}

// write_har_file, read/p_output.cpp:35-55: per ring of layer 0,
// a = sum_j sin(m yc_j) Sigma_j and b = sum_j cos(m yc_j) Sigma_j
template <typename RT>
__global__ void k_post_harmonic(Tables T, const RT *R, double m, double *ab) {
  __shared__ double red[32];
  const int i = blockIdx.x, rk = i + NPAD;
  const size_t base = (size_t)rk * T.nphi;
  const double off = (sizeof(RT) == 4) ? T.sbg[rk] : 0.0;   // FP32 planes hold Sigma - S_bg
  double a = 0.0, b = 0.0;
  for (int j = threadIdx.x; j < T.nphi; j += blockDim.x) {
    double sig = off + (double)R[base + j];
    a += sin(m * T.yc[j]) * sig;
    b += cos(m * T.yc[j]) * sig;
  }
  a = block_sum(a, red);
  b = block_sum(b, red);
  if (threadIdx.x == 0) { ab[2 * i] = a; ab[2 * i + 1] = b; }
}

// get_torque, read/transform.cpp:386-420: torque of the disk on a planet of
// mass ratio M_p at r = 1, azimuth pi, in the barycentric frame (star at
// distance M_p/(1+M_p) opposite), softening 3e-6 in Rp^2; one sum per ring
template <typename RT>
__global__ void k_post_torque(Tables T, const RT *R, double M_p, double *ring_out) {
  __shared__ double red[32];
  const int i = blockIdx.x, k = blockIdx.y;
  const int row = i + NPAD, rk = k * T.nrg + row, kz = k + NPAD;
  const size_t base = (size_t)rk * T.nphi;
  const double off = (sizeof(RT) == 4) ? T.sbg[rk] : 0.0;
  const double stm = 1.0 / (1.0 + M_p), plm = M_p * stm, plx = 1.0 * stm, stx = 1.0 * plm;
  const double rad = T.rxc[row], z = T.zc[kz], dxz = T.rdx[row] * T.dz[kz];
  double t = 0.0;
  for (int j = threadIdx.x; j < T.nphi; j += blockDim.x) {
    double azi = T.yc[j];
    double cosfac = cos(azi - 3.1415926535897932384626433832795);
    double sinfac = sin(azi - 3.1415926535897932384626433832795);
    double Rp = rad * rad + plx * plx - 2.0 * plx * rad * cosfac + z * z;
    Rp = sqrt(Rp + 0.000003);
    double Rs = sqrt(rad * rad + stx * stx + 2.0 * stx * rad * cosfac + z * z);
    double rho = off + (double)R[base + j];
    t += rho * (plm * plx * sinfac / (Rp * Rp * Rp) - stm * stx * sinfac / (Rs * Rs * Rs)) * rad * T.dy[j] * dxz;
  }
  t = block_sum(t, red);
  if (threadIdx.x == 0) ring_out[k * T.nr + i] = t;
}

// ---------------------------------------------------------------------------
// Batched 2D steps: the clock kernels and the ring reductions of every run of
// a group in one launch each (the sweeps are in pg_sweep.cu).
__global__ void kb_prestep(const BatchRun *runs) {
  const BatchRun &b = runs[blockIdx.x];
  prestep_body(b.clk, b.T, b.fargo);
}
__global__ void kb_poststep(const BatchRun *runs) {
  const BatchRun &b = runs[blockIdx.x];
  poststep_body(b.clk, b.T);
}
__global__ void kb_record(const BatchRun *runs) { record_body(runs[blockIdx.x].clk); }

template <typename RT>
__global__ void __launch_bounds__(1024) kb_reduce(BatchQueue q, int mode) {
  const int r = batch_find(q, blockIdx.x);
  const BatchRun &b = q.runs[r];
  if (mode == 9 && !b.plnt) return;
  const RT *R;
  if constexpr (sizeof(RT) == 4) R = (const RT *)b.QX.r;   // a 2D step ends in its first planes
  else R = (const RT *)b.PX.r;
  double *out = (mode == 0) ? &b.clk->mass : &b.clk->torque;
  reduce_body<RT>(b.T, R, Body{}, b.clk, 0.0, mode, mode == 9 ? 1 : b.plnt, b.p_alpha, 2, b.ring_part, b.counter,
                  out, nullptr, blockIdx.x - q.start[r], b.T.nr, (unsigned)b.T.nr);
}

}  // namespace pgd

// ---------------------------------------------------------------------------
namespace pgk {
using namespace pgd;

template <class RT>
void cfl(const Tables &T, const RT *r, const RT *u, const RT *v, const RT *w, const double *p0, const Phys &ph,
         double frrot, int ndim, unsigned long long *out, DevClock *clk, int rot_pending, cudaStream_t s) {
  dim3 grid(T.nr, T.nk);
  k_cfl<RT><<<grid, 256, 0, s>>>(T, r, u, v, w, p0, ph, frrot, ndim, out, clk, rot_pending);
}

template <class RT>
void damp(const Tables &T, RT *r, RT *u, RT *v, RT *w, double dt, const DevClock *clk, int ndim, cudaStream_t s) {
  dim3 grid(T.nr, T.nk);
  k_damp<RT><<<grid, 256, 0, s>>>(T, r, u, v, w, dt, clk, ndim);
}
#define PG_AROUND(RT)                                                                                                   \
  template void cfl<RT>(const Tables &, const RT *, const RT *, const RT *, const RT *, const double *, const Phys &,   \
                        double, int, unsigned long long *, DevClock *, int, cudaStream_t);                              \
  template void damp<RT>(const Tables &, RT *, RT *, RT *, RT *, double, const DevClock *, int, cudaStream_t);
PG_AROUND(double)
PG_AROUND(float)

void index_shift(const Tables &T, double dt, double frrot, int fargo, const DevClock *clk, cudaStream_t s) {
  int n = T.nr * T.nk;
  k_index<<<(n + 127) / 128, 128, 0, s>>>(T, dt, frrot, fargo, clk);
}

void rotate(const Tables &T, const DevClock *clk, cudaStream_t s) {
  int n = T.nr * T.nk;
  k_rotate<<<(n + 127) / 128, 128, 0, s>>>(T, clk);
}

// The ring sums run on two 1024-thread CTAs per SM, each taking every
// grid-th ring: most steps print nothing and every CTA returns at once, so
// a grid of one CTA per ring would only pay for starting them.
static int reduce_grid(const Tables &T) {
  static int nsm = 0;
  if (nsm == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (nsm <= 0) nsm = 148;
  }
  const int rings = T.nr * T.nk;
  return rings < 2 * nsm ? rings : 2 * nsm;
}

// The mass sums of a run with at least 1024 rings go one warp per ring
// (k_reduce_mass_w): on the 128x1024x32 disk 4096 rings in one wave of
// warps instead of 14 rings in turn per 1024-thread CTA.
static bool mass_warp(const Tables &T) { return T.nr * T.nk >= 1024; }
static int mass_grid(const Tables &T) { return (T.nr * T.nk + RW - 1) / RW; }

void reduce(const Tables &T, const double *r, const Body &pl, const DevClock *clk, double exclude,
            int mode, int plnt, double p_alpha, int ndim, double *ring_part, unsigned int *counter,
            double *out, double *hist_row, cudaStream_t s) {
  if ((mode == 0 || !plnt) && mass_warp(T)) {
    k_reduce_mass_w<double><<<mass_grid(T), 32 * RW, 0, s>>>(T, r, clk, ndim, ring_part, counter, out);
    return;
  }
  k_reduce<double><<<reduce_grid(T), 1024, 0, s>>>(T, r, pl, clk, exclude, mode, plnt, p_alpha, ndim, ring_part, counter,
                                         out, hist_row);
}

void reduce32(const Tables &T, const float *r, const Body &pl, const DevClock *clk, double exclude, int mode,
              int plnt, double p_alpha, int ndim, double *ring_part, unsigned int *counter, double *out,
              cudaStream_t s) {
  if ((mode == 0 || !plnt) && mass_warp(T)) {
    k_reduce_mass_w<float><<<mass_grid(T), 32 * RW, 0, s>>>(T, r, clk, ndim, ring_part, counter, out);
    return;
  }
  k_reduce<float><<<reduce_grid(T), 1024, 0, s>>>(T, r, pl, clk, exclude, mode, plnt, p_alpha, ndim, ring_part, counter,
                                        out, nullptr);
}

void prestep(DevClock *clk, const Tables &T, int fargo, cudaStream_t s) {
  k_prestep<<<1, 256, 0, s>>>(clk, T, fargo);
}

void poststep_drift(DevClock *clk, const Tables &T, cudaStream_t s) {
  k_poststep_drift<<<1, 256, 0, s>>>(clk, T);
}
void poststep_kick(DevClock *clk, cudaStream_t s) {
  Tables T{};
  k_poststep_kick<<<1, 1, 0, s>>>(clk, T);
}
void reduce_forces(const Tables &T, const void *r, int fp32, DevClock *clk, double p_alpha, int ndim,
                   double *ring_part, unsigned int *counter, cudaStream_t s) {
  const int grid = reduce_grid(T);
  for (int mode : {8, 9}) {
    if (fp32)
      k_reduce_forces<float><<<grid, 1024, 0, s>>>(T, (const float *)r, clk, mode, p_alpha, ndim, ring_part, counter);
    else
      k_reduce_forces<double><<<grid, 1024, 0, s>>>(T, (const double *)r, clk, mode, p_alpha, ndim, ring_part, counter);
  }
}
void post_harmonic(const Tables &T, const void *r, int fp32, double m, double *ab, cudaStream_t s) {
  if (fp32) k_post_harmonic<float><<<T.nr, 256, 0, s>>>(T, (const float *)r, m, ab);
  else k_post_harmonic<double><<<T.nr, 256, 0, s>>>(T, (const double *)r, m, ab);
}
void post_torque(const Tables &T, const void *r, int fp32, double M_p, double *ring_out, cudaStream_t s) {
  dim3 grid(T.nr, T.nk);
  if (fp32) k_post_torque<float><<<grid, 256, 0, s>>>(T, (const float *)r, M_p, ring_out);
  else k_post_torque<double><<<grid, 256, 0, s>>>(T, (const double *)r, M_p, ring_out);
}

void unpack_dump(const Tables &T, const double *stage, const DumpPlanes &D, int ndim, int fp32, int *err,
                 cudaStream_t s) {
  dim3 grid((T.nphi + 255) / 256, T.nr, T.nk);
  k_unpack_dump<<<grid, 256, 0, s>>>(T, stage, D, ndim, fp32, err);
}
void fill_ghost_rows(const Tables &T, const double *ghosts, const DumpPlanes &D, int ndim, int fp32,
                     cudaStream_t s) {
  dim3 grid((T.nphi + 255) / 256, 2 * NPAD, T.nk);
  k_fill_ghost_rows<<<grid, 256, 0, s>>>(T, ghosts, D, ndim, fp32);
}
void pack_dump(const Tables &T, const DumpPlanes &D, const Phys &ph, int ndim, int fp32, int p0_live, unsigned char *out,
               cudaStream_t s) {
  dim3 grid((T.nphi + 255) / 256, T.nr, T.nk);
  k_pack_dump<<<grid, 256, 0, s>>>(T, D, ph, ndim, fp32, p0_live, out);
}

void poststep(DevClock *clk, const Tables &T, cudaStream_t s) {
  k_poststep<<<1, 256, 0, s>>>(clk, T);
}

void record(DevClock *clk, cudaStream_t s) {
  k_record<<<1, 1, 0, s>>>(clk);
}

void tables(const Tables &T, const Phys &ph, int ndim, double kill_rin, double kill_rout, double xmin,
            double xmax, cudaStream_t s) {
  int n = T.nk * T.nrg;
  if (2 * NPAD * T.nr > n) n = 2 * NPAD * T.nr;         // the polar ghost-layer nu table
  if (T.nk + 2 * NPAD > n) n = T.nk + 2 * NPAD;
  if (T.nphi > n) n = T.nphi;
  k_tables<<<(n + 127) / 128, 128, 0, s>>>(T, ph, ndim, kill_rin, kill_rout, xmin, xmax);
  axis_tables(T, ndim, s);
}


void batch_prestep(const BatchRun *runs, int nruns, cudaStream_t s) {
  if (nruns > 0) kb_prestep<<<nruns, 256, 0, s>>>(runs);
}
void batch_poststep(const BatchRun *runs, int nruns, cudaStream_t s) {
  if (nruns > 0) kb_poststep<<<nruns, 256, 0, s>>>(runs);
}
void batch_record(const BatchRun *runs, int nruns, cudaStream_t s) {
  if (nruns > 0) kb_record<<<nruns, 1, 0, s>>>(runs);
}
void batch_reduce(const BatchQueue &rings, int fp32, int mode, cudaStream_t s) {
  if (rings.total <= 0) return;
  if (fp32) kb_reduce<float><<<rings.total, 1024, 0, s>>>(rings, mode);
  else kb_reduce<double><<<rings.total, 1024, 0, s>>>(rings, mode);
}
}  // namespace pgk
