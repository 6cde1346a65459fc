// pg_kernels.cuh -- device-side data of a run and the kernel launchers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "pg_ppm.cuh"

namespace pgd {

// Chunking of one pencil direction (ppm.cu:34, 48, 169, 196).
struct Chunking {
  int loop;      // number of 116-cell chunks
  int lim_last;  // lim of the last chunk: n % 116 + 12
  int stuck;     // n % 116 == 0: the reference never updates the last chunk
};

__host__ __device__ inline Chunking make_chunking(int n) {
  Chunking c;
  c.loop = n / REAL + (n % REAL != 0);
  c.lim_last = (n % REAL) + 2 * NPAD;
  c.stuck = (n % REAL == 0);
  return c;
}

// How a sweep lays a chunk of lim cells on warps: G lanes per pencil, P
// pencils per warp, cols pencils per CTA, step rows per pass of a CTA's loads
// and stores, ng groups of cols pencils across the grid.  mG, mP, mC: 2^16 / d
// rounded up, for quotients of small numbers (quot16); mng: 2^40 / ng.
struct Tile {
  int lim, G, P, cols, step, ng;
  unsigned mG, mP, mC;
  unsigned long long mng;
};

// The planet of a step as the sweeps' forces use it (forces.cu:23-182):
// mass (3D with a planet: the reference's reduced mass), distance, 1/x^2,
// x^2 + rs^2, the star's share of the mass, azimuth and its rate, cos and sin
// of the azimuth
struct PlanetC {
  double m, x, ix2, b2, star, y, vy, cy, sy;
  double2 turn;              // 3D: turn_of a ring with no residual velocity (fixed layers)
};

// What the last sweep of a step needs of a ring at its store, in one place: four
// 16-byte loads where an array each took nine and their addresses.
struct __align__(16) RingOut {
  double f, off;             // this step's damping factor and CFL frame offset (pg_step.cu)
  double cs, irc, rc;        // sound speed (EOS 0), 1/r_cyl, r_cyl
  double irdx, iwz;          // 1/dr, 1/(r dtheta)
  int2 shift;                // inc_j and rot_j + inc_j modulo nphi
};

// Geometry and per-ring tables, all device pointers.  A "row" counts radial
// rings including the 6 fixed ghost rings on each side (row = i + 6); a
// "ring" index rk = k*nrg + row.
struct Tables {
  int nr, nphi, nk, nrg;
  int odd;                                      // ghost cells without a state: 1 of the radial sweep, 2 of the polar one
  Chunking cx, cy, cz;
  Tile tx[2], ty[2], tz[2];                     // per axis: full chunks, last chunk (pgk::tiles)
  unsigned long long mnr;                       // 2^40 / nr rounded up
  const double *rx, *rdx, *rxvol, *rxc;         // [nrg]
  const double *irdx, *irxc, *rpa;              // [nrg]: 1/rdx, 1/rxc, rxc^-p_alpha (k_tables)
  const double *radc, *cs2, *nu;                // [nk*nrg]
  const double *irc, *snd;                      // [nk*nrg]: 1/radc, sqrt(gam cs2) (k_tables)
  const double *y, *dy, *yvol, *yc;             // [nphi]
  const double *idy, *cyc, *syc;                // [nphi]: 1/dy, cos(yc), sin(yc) (k_tables)
  const double *z, *dz, *zvol, *zc;             // [nk + 12]: 6 ghost layers each side
  const double *szc, *idz;                      // [nk + 12]: sin(zc), 1/dz (k_tables)
  const double *csg;                            // [12 nr]: cs2 of the fixed polar ghost layers (as nug)
  const double *ax[3];                          // per axis: what a chunk's cells need of the grid (pg_warp.cuh)
  const double *nug;                            // [12 nr]: nu of the polar ghost layers (6 below, 6 above) per ring
  const double *val_r, *val_u, *val_v;          // [nk*nrg] damping / FARGO targets
  const double *damp_g, *damp_pw;               // [nk*nrg] zone factor, r^-1.5
  const double *tg;                             // [6*nr*4] theta ghost state (udr): r,p,u,v
  const double *vbg;                            // [nk*nrg] FP32 runs: v_phi background (val.v / ghost v)
  const double *sbg;                            // [nk*nrg] FP32 runs: Sigma background (val.r / ghost r)
  double *res_v, *rot_v;                        // [nk*nrg]
  int *inc_j, *rot_j;                           // [nk*nrg]
  double2 *turn;                                // [nk*nrg], 3D: cos and sin of the planet's angle's change in dt/2 (turn_of)
  RingOut *ro;                                  // [nk*nrg]
};

// State planes a sweep reads and writes: FP64 Sigma, v_r, v_phi, v_theta, or
// FP32 dS = Sigma - S_bg, v_r, dv = v_phi - v_bg, v_theta
template <class RT>
struct PlanesT {
  const RT *r = nullptr, *u = nullptr, *v = nullptr, *w = nullptr;
  RT *ro = nullptr, *uo = nullptr, *vo = nullptr, *wo = nullptr;
  const double *p0 = nullptr;   // non-null: pressure of a freshly loaded dump (first sweep only, FP64)
};
using Planes = PlanesT<double>;
using Planes32 = PlanesT<float>;

// The device-resident clock of the fused loop (main.cu:270-441).
struct DevClock {
  double simtime, timem, dt, old_dt, dt_step, frrot, frrot_next;
  double endtime, tmovie, courant;
  Body planet;
  PlanetC pc;                    // of planet, for the step's sweeps
  long long ncycle, ncycp, ncycend;
  int make_pict, prin, done, halted, status, pad;
  unsigned long long cfl_bits;   // max CFL rate as ordered bits (non-negative)
  int nprin, plnt_flag, frrot_flag, ndim;
  double M_p, t_growth, rs_fac, sc2, R_p, Sigma_0, p_beta;
  double f8, f9;                 // moving planet: disk forces of the step (reductions 8, 9)
  double hist_norm;
  double mass, torque;           // last diagnostics reductions
  double *hist;                  // device history rows (HIST_COLS each)
  int hist_count, hist_cap;
};
constexpr int HIST_COLS = 11;

struct SweepCtl {
  double dt;
  double frrot;
  Body planet;
  DevClock *clk;      // non-null: read dt/planet/frrot from the clock, honour halt
  int fuse;           // sweepy epilogue: damping + CFL + finiteness check
  int shift;          // store at (j + inc_j) mod jmax: the last sweep of a step
  int nocfl;          // with fuse: no CFL rate (a moving planet's FrRot is known only after the step)
};

// parts of what happens between two steps (pg_step.cu): the end of one with a
// fixed planet, its diagnostics, the start of the next
constexpr int BETWEEN_POST = 1, BETWEEN_DIAG = 2, BETWEEN_PRE = 4;

// Planes a dump is unpacked into / packed from (pg_load_rings, pg_save_rings).
struct DumpPlanes {
  double *r, *u, *v, *w, *p0;    // FP64 run, p0: the dump's pressure
  float *fr, *fu, *fv, *fw;      // FP32 run (residual Sigma and v_phi)
};

// One run of a batch (pg_batch.cu): what its kernels read, in device memory.
struct BatchRun {
  Tables T;
  Phys ph;
  DevClock *clk;
  Planes PX, PY;          // FP64 runs: planes of the radial and of the azimuthal sweep
  Planes32 QX, QY;        // FP32 runs
  const double *p0;       // FP64 run with a freshly loaded dump: its pressure plane,
  long long p0_cycle;     //   read by the radial sweep of the step with ncycle == p0_cycle
  double *ring_part;
  unsigned int *counter;
  int fargo, plnt;
};

// A group of runs walked by one launch: tile t belongs to run r when
// start[r] <= t < start[r + 1].
struct BatchQueue {
  const BatchRun *runs;
  const int *start;       // [nruns + 1] device prefix sums
  int nruns;
  int total;
};

// ---- small device functions the sweeps and the kernels around them share ----
// Operations are written out, so that a value has the same bits wherever it
// is formed (the fused epilogue and the separate kernels must agree).
__device__ __forceinline__ int wrap1(int j, int n) {
  if (j < 0) j += n;
  if (j >= n) j -= n;
  return j;
}
__device__ __forceinline__ int wrapm(int j, int n) {
  j %= n;
  return j < 0 ? j + n : j;
}
// a density or azimuthal velocity from and to its plane (FP32: less the ring's background)
template <class RT>
__device__ __forceinline__ double load_r(RT x, double bg) {
  return sizeof(RT) == 4 ? bg + (double)x : (double)x;
}
template <class RT>
__device__ __forceinline__ RT store_r(double x, double bg) {
  return sizeof(RT) == 4 ? (RT)(x - bg) : (RT)x;
}
__device__ __forceinline__ double damped(double x, double target, double f) { return __fma_rn(f, __dsub_rn(target, x), x); }
__device__ __forceinline__ double sound_speed(double r, double p, const Phys &ph) { return sqrt(__dmul_rn(ph.gam, p) / r); }
// dt_lv1's rate of a cell (timestep.cu:36-57): 1/dr, azimuthal velocity less
// the ring's frame, 1/(r dphi), 1/(r dtheta)
template <bool THREED>
__device__ __forceinline__ double cfl_rate(double cs, double u, double irdx, double v, double iwy, double w, double iwz) {
  const double t0 = __dmul_rn(__dadd_rn(fabs(u), cs), irdx), t1 = __dmul_rn(__dadd_rn(fabs(v), cs), iwy);
  if (!THREED) return fmax(t0, t1);
  return max3(t0, t1, __dmul_rn(__dadd_rn(fabs(w), cs), iwz));
}
// A step's kernels are launched so that each is set up while the one before it
// still runs (pgk::launch); each waits here, before it reads or writes memory,
// until that one is complete and its writes are visible.  Of a small grid's
// step a third is launches: 136x203 launched call by call 34 -> 27.7 us, moving
// planet 251x767 59 -> 47, graph replay 128x384 33.0 -> 31.7, 80x240x24 149 ->
// 147.  No kernel lets the next one start earlier than its own end: with
// launch_dependents at the top of each the 128x384 replay took 39.3 us, before
// the sweeps' last stores 32.1.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
// a / d for small a (a d < 2^16) from m = 2^16 / d rounded up
__device__ __forceinline__ int quot16(int a, unsigned m) { return (int)((unsigned)a * m >> 16); }
// a / d (a d < 2^40) from m = 2^40 / d rounded up
__device__ __forceinline__ int quot40(int a, int d, unsigned long long m) {
  const int q = (int)((unsigned long long)(unsigned)a * m >> 40);
  return q * d > a ? q - 1 : q;
}
// the sweeps' copy of a ring's shift
__device__ __forceinline__ void set_shift(const Tables &T, int rk, int inc, int rot) {
  T.ro[rk].shift = make_int2(wrapm(inc, T.nphi), wrapm(rot + inc, T.nphi));
}
// the run of tile t of a batch queue, by bisection in its prefix sums
__device__ __forceinline__ int batch_find(const BatchQueue &q, int t) {
  int lo = 0, hi = q.nruns;   // q.start[lo] <= t < q.start[hi]
  while (hi - lo > 1) {
    int mid = (lo + hi) >> 1;
    if (q.start[mid] <= t) lo = mid; else hi = mid;
  }
  return lo;
}

}  // namespace pgd

// launchers (pg_kernels.cu; the sweeps in pg_sweep.cu)
namespace pgk {
// Launches a kernel that calls after_previous() first thing: it may be set up
// while the kernel before it in the stream still runs.
template <class... K, class... A>
inline void launch(void (*f)(K...), dim3 grid, int block, size_t shm, cudaStream_t s, A &&...a) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3(block);
  c.dynamicSmemBytes = shm;
  c.stream = s;
  c.attrs = &at;
  c.numAttrs = 1;
  cudaLaunchKernelEx(&c, f, K(a)...);
}
using namespace pgd;
void tables(const Tables &T, const Phys &ph, int ndim, double kill_rin, double kill_rout, double xmin,
            double xmax, cudaStream_t s);
template <class RT>
void sweep_x(const Tables &T, const PlanesT<RT> &P, const Phys &ph, const SweepCtl &c, int ndim, cudaStream_t s);
template <class RT>
void sweep_y(const Tables &T, const PlanesT<RT> &P, const Phys &ph, const SweepCtl &c, int ndim, cudaStream_t s);
template <class RT>
void sweep_z(const Tables &T, const PlanesT<RT> &P, const Phys &ph, const SweepCtl &c, int ntop, cudaStream_t s);
// per-device kernel attributes (dynamic shared memory limits); 0 on success
int setup_device();
// the grid's tiles (Tables::tx, ty, tz, mnr)
void make_tiles(Tables &T);
// CTAs of a run's radial and azimuthal sweep (batch queues)
int tiles_x(const Tables &T);
int tiles_y(const Tables &T);
// the grid's axis tables (Tables::ax), and the doubles one takes
void axis_tables(const Tables &T, int ndim, cudaStream_t s);
size_t axis_table_elems(const Chunking &ch);
// CFL rate max of the planes (p0: the pressure of a freshly loaded dump, or
// null) into *out; with clk, the device loop's: FrRot, target and halt flag
// from the clock, the step's shift still pending when rot_pending; with hout,
// *out goes to *hout (host memory) and is cleared (counter: 0 between launches)
template <class RT>
void cfl(const Tables &T, const RT *r, const RT *u, const RT *v, const RT *w, const double *p0, const Phys &ph,
         double frrot, int ndim, unsigned long long *out, DevClock *clk, int rot_pending, unsigned *counter,
         unsigned long long *hout, cudaStream_t s);
// damping by dt, or by the clock's step
template <class RT>
void damp(const Tables &T, RT *r, RT *u, RT *v, RT *w, double dt, const DevClock *clk, int ndim, cudaStream_t s);
// the step around the sweeps (pg_step.cu)
void index_shift(const Tables &T, double dt, double frrot, int fargo, cudaStream_t s);
void rotate(const Tables &T, cudaStream_t s);
// disk mass (mode 0), radial force (8) or torque (9) on the planet into *out;
// part: 2 nr nk doubles, counter: 0 between launches
template <class RT>
void reduce(const Tables &T, const RT *r, const Body &pl, double exclude, int mode, int plnt, int ndim,
            double *part, unsigned *counter, double *out, cudaStream_t s);
// between two steps: any of the parts BETWEEN_*
template <class RT>
void between(const Tables &T, const RT *r, DevClock *clk, double *part, unsigned *counter, int fargo,
             int plnt, int ndim, int fl, cudaStream_t s);
// moving planet (plnt_flag 2): a step's end up to the kick
template <class RT>
void moving(const Tables &T, const RT *r, DevClock *clk, double *part, unsigned *counter, int ndim,
            cudaStream_t s);
// between() of every member of a batch; CTAs of a member
template <class RT>
void batch_between(const BatchQueue &q, int fl, cudaStream_t s);
int between_ctas(int rings);
// batched 2D sweeps over many runs
template <class RT>
void batch_sweep_x(const BatchQueue &q, int grid, cudaStream_t s);
template <class RT>
void batch_sweep_y(const BatchQueue &q, int grid, cudaStream_t s);
// dump <-> planes: stage holds the dump's field arrays ring by ring ([nr*nk][5][nphi]
// for unpack, whole 72*nphi+96-byte ring records for pack); err bit 1: a density
// that is not finite and positive, bit 2: nonzero w in a 2D dump
void unpack_dump(const Tables &T, const double *stage, const DumpPlanes &D, int ndim, int fp32, int *err,
                 cudaStream_t s);
void fill_ghost_rows(const Tables &T, const double *ghosts, const DumpPlanes &D, int ndim, int fp32,
                     cudaStream_t s);
void pack_dump(const Tables &T, const DumpPlanes &D, const Phys &ph, int ndim, int fp32, int p0_live, unsigned char *out,
               cudaStream_t s);
// post-processing (read/ tools): azimuthal harmonic m per ring of layer 0
// (ab[2i], ab[2i+1]), torque on a planet at r = 1 per ring (ring_out[k*nr+i])
void post_harmonic(const Tables &T, const void *r, int fp32, double m, double *ab, cudaStream_t s);
void post_torque(const Tables &T, const void *r, int fp32, double M_p, double *ring_out, cudaStream_t s);
}  // namespace pgk
