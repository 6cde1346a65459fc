// pg_kernels.cu -- sm_100a kernels around the sweeps (pg_sweep.cu) and
// the step (pg_step.cu).
//
//   k_tables    per-ring, per-column and per-layer tables
//   k_cfl       CFL rate max (dt_lv1, timestep.cu:12-73)
//   k_damp      wave damping
//   k_pack_dump, k_unpack_dump  dump records <-> planes
//   k_post_*    the reference's read/ tools
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
    const_cast<double *>(T.rpa)[t] = pow(T.rxc[t], -ph.p_alpha);
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
  set_shift(T, t, T.inc_j[t], T.rot_j[t]);
  cs2[t] = ph.sc2 * pow(rc, -ph.p_beta);          // get_cs2 disk_profile.cu:39-42
  const_cast<double *>(T.irc)[t] = 1.0 / rc;
  const_cast<double *>(T.snd)[t] = sqrt(ph.gam * cs2[t]);
  RingOut &o = T.ro[t];
  o.f = o.off = 0.0;
  o.cs = T.snd[t]; o.irc = T.irc[t]; o.rc = rc;
  o.irdx = 1.0 / T.rdx[row];
  o.iwz = ndim == 3 ? __dmul_rn(1.0 / T.dz[k + NPAD], 1.0 / T.rxc[row]) : 0.0;
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
// are checked, and rot_j may still lack the step's shift (rot_pending).  With
// hout (get_dt) the last CTA to finish hands the maximum to the host's memory
// and clears *out for the next call.
template <class RT>
__global__ void k_cfl(Tables T, const RT *R, const RT *U, const RT *V, const RT *W, const double *P0, Phys ph,
                      double frrot, int ndim, unsigned long long *out, DevClock *clk, int rot_pending, unsigned *counter,
                      unsigned long long *hout) {
  after_previous();
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
    if (hout) {
      __threadfence();
      if (atomicAdd(counter, 1u) == gridDim.x * gridDim.y - 1) {
        *counter = 0u;
        *hout = atomicExch(out, 0ull);
      }
    }
  }
}

// wave damping by dt, or by the clock's step: the rule and the bits of the
// last sweep's epilogue
template <class RT>
__global__ void k_damp(Tables T, RT *R, RT *U, RT *V, RT *W, double dt, const DevClock *clk, int ndim) {
  after_previous();
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

}  // namespace pgd

// ---------------------------------------------------------------------------
namespace pgk {
using namespace pgd;

template <class RT>
void cfl(const Tables &T, const RT *r, const RT *u, const RT *v, const RT *w, const double *p0, const Phys &ph,
         double frrot, int ndim, unsigned long long *out, DevClock *clk, int rot_pending, unsigned *counter,
         unsigned long long *hout, cudaStream_t s) {
  dim3 grid(T.nr, T.nk);
  launch(k_cfl<RT>, grid, 256, 0, s, T, r, u, v, w, p0, ph, frrot, ndim, out, clk, rot_pending, counter, hout);
}

template <class RT>
void damp(const Tables &T, RT *r, RT *u, RT *v, RT *w, double dt, const DevClock *clk, int ndim, cudaStream_t s) {
  dim3 grid(T.nr, T.nk);
  launch(k_damp<RT>, grid, 256, 0, s, T, r, u, v, w, dt, clk, ndim);
}
#define PG_AROUND(RT)                                                                                                   \
  template void cfl<RT>(const Tables &, const RT *, const RT *, const RT *, const RT *, const double *, const Phys &,   \
                        double, int, unsigned long long *, DevClock *, int, unsigned *, unsigned long long *,           \
                        cudaStream_t);                                                                                  \
  template void damp<RT>(const Tables &, RT *, RT *, RT *, RT *, double, const DevClock *, int, cudaStream_t);
PG_AROUND(double)
PG_AROUND(float)

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

void tables(const Tables &T, const Phys &ph, int ndim, double kill_rin, double kill_rout, double xmin,
            double xmax, cudaStream_t s) {
  int n = T.nk * T.nrg;
  if (2 * NPAD * T.nr > n) n = 2 * NPAD * T.nr;         // the polar ghost-layer nu table
  if (T.nk + 2 * NPAD > n) n = T.nk + 2 * NPAD;
  if (T.nphi > n) n = T.nphi;
  k_tables<<<(n + 127) / 128, 128, 0, s>>>(T, ph, ndim, kill_rin, kill_rout, xmin, xmax);
  axis_tables(T, ndim, s);
}

}  // namespace pgk
