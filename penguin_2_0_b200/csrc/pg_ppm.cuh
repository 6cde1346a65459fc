// pg_ppm.cuh -- constants, pressure relation and planet gravity shared by the
// sweeps (pg_warp.cuh, pg_sweep.cu) and the kernels around them.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace pgd {

constexpr int NPAD = 6;
constexpr int ARR = 128;
constexpr int REAL = ARR - 2 * NPAD;   // 116

constexpr double kTwoPi = 6.283185307179586476925286766559;
constexpr double kThird = 0.3333333333333333333333333;
constexpr double kFourthd = 1.3333333333333333333333333;
constexpr double kSmallp = 1.0e-15;
constexpr double kSmallr = 1.0e-15;

struct Body { double m, x, y, vx, vy, fx, fy, rs; };

// Physics constants of the run (global.h), passed by value to kernels.
struct Phys {
  double gam, sc2, vis_nu, p_alpha, p_beta;
  double gamfac1, gamfac2;  // (gam + 1)/gam/2 and gam + 1 (global.h:54-55)
  int plnt;       // plnt_flag > 0
  int flat;       // flat_flag
  int visc;       // visc_flag
  int eos;        // EOS: 0 isothermal, 1 isentropic (global.h:18)
};

// Pressure of a cell from its density by the sweep store's relation
// (ppm.cu:138-143): EOS 0 p = rho cs2, EOS 1 p = cs2 rho^gam / gam.  The
// planes hold no pressure; every reader of p derives it here.  The sweeps
// take EOS as a template argument (the EOS-0 kernels carry no pow); the
// small kernels around them (CFL, dump packing) branch at run time.
template <int EOS>
__device__ __forceinline__ double eos_p(double r, double cs2, const Phys &ph) {
  if (EOS == 0) return r * cs2;
  return cs2 * pow(r, ph.gam) / ph.gam;
}
__device__ __forceinline__ double eos_p_rt(double r, double cs2, const Phys &ph) {
  return ph.eos ? eos_p<1>(r, cs2, ph) : eos_p<0>(r, cs2, ph);
}

// ---- star + planet gravity, forces.cu:23-182 (non-barycentric frame) ------
// as pg_noalloc.cu's sums take it; the sweeps' form is in pg_warp.cuh
__device__ __forceinline__ double planet_cosfac(double azi, const Body &p, double dt) {
  return cos(azi - (p.y + dt * p.vy));
}
// cos and sin of the planet's angle in one out-of-line copy
static __device__ __noinline__ double2 pg_cossin(double x) { return make_double2(cos(x), sin(x)); }
__device__ __forceinline__ double grav_rad_cyl_cf(double rad, double cosfac, double z, const Body &p) {
  double plm = p.m;
  double plx = p.x;
  double Rp = sqrt(rad * rad + plx * plx - 2.0 * plx * rad * cosfac + z * z + p.rs * p.rs);
  return -plm * (rad - plx * cosfac) / (Rp * Rp * Rp) - plm * cosfac / (plx * plx);
}
__device__ __forceinline__ double grav_rad_cyl(double rad, double azi, double z, const Body &p, double dt) {
  return grav_rad_cyl_cf(rad, planet_cosfac(azi, p, dt), z, p);
}
__device__ __forceinline__ double grav_azi_cyl(double rad, double azi, double z, const Body &p, double dt) {
  const double2 cs = pg_cossin(azi - (p.y + dt * p.vy));
  double cosfac = cs.x;
  double sinfac = cs.y;
  double plm = p.m;
  double plx = p.x;
  double Rp = sqrt(rad * rad + plx * plx - 2.0 * plx * rad * cosfac + z * z + p.rs * p.rs);
  return -plm * plx * sinfac / (Rp * Rp * Rp) + plm * sinfac / plx / plx;
}
__device__ __forceinline__ double max3(double A, double B, double C) {   // simple_func.cu:16-28
  if (A > B) { if (C > A) return C; else return A; }
  else       { if (C > B) return C; else return B; }
}

}  // namespace pgd
