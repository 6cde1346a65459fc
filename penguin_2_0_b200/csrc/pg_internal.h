// pg_internal.h -- what the batch and serving code (pg_batch.cu, pg_serve.cpp)
// use of a run object.  Not part of the C ABI.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/penguin_b200.h"
#include "pg_kernels.cuh"

namespace pgi {

struct RunShape {
  int dev, ndim, fp32, loaded, clock_ready, p0_live;
  int moving;              // plnt_flag 2: the planet feels the disk (own step sequence)
  int eos;                 // EOS 1: isentropic sweeps (own step sequence)
  int odd;                 // ghost rings without a state (own step sequence)
  int nr, nphi, nk;
  int tiles_x, tiles_y;    // CTAs of the radial and azimuthal sweeps
  int ctas_b;              // CTAs between two steps
};
int run_shape(const pg_run *run, RunShape *out);

// Device descriptor of a 2D run whose clock is set (pg_clock_reset).
int run_batch_desc(pg_run *run, pgd::BatchRun *d);
// The batch enqueued steps of this run: the p0 plane is used up.
void run_batched(pg_run *run);
// The batch is about to step this run: its step count is the device's to tell.
void run_stepped(pg_run *run);
// One step of the device-resident loop of this run, enqueued on stream s
// (first, last: of the sequence being queued).
int run_enqueue_on(pg_run *run, cudaStream_t s, bool first, bool last, int64_t *launches);
// cudaMalloc that gives the dumps' idle block back where memory is short.
cudaError_t device_malloc(int dev, void **p, size_t bytes);
// Device clock of the run.
pgd::DevClock *run_clock(pg_run *run);
// which of the two plane copies is current (3D steps flip it)
int run_cur(const pg_run *run);
void run_set_cur(pg_run *run, int cur);
// The batch a run is in (null: none), which is told when the run is destroyed.
void run_set_batch(pg_run *run, pg_batch *b);
void batch_forget(pg_batch *b, pg_run *run);
cudaStream_t run_stream(pg_run *run);

}  // namespace pgi
