// Ensemble mean of a projected trajectory in blocks of steps, and its adjoint
// (rk4_mean.cu).
#pragma once
#include "qsx_common.cuh"

namespace qsx {

bool rk4_mean_supported(int m, int64_t nsave);
int rk4_mean_grid(int64_t batch, int* grid);
// partial [grid][nsave], the sums over each CTA's samples; *flag nonzero
// afterwards (on the device) when a value was not finite and the stepped loop
// has to run.  The same flag for the adjoint.
int rk4_mean_run(const qsx_rk4_args* a, int grid, double2* partial, int* flag, cudaStream_t s);

// The stepped loop of FP64 arguments with out_state, run only when the device
// word *only_if is nonzero (null: always).
int rk4_stepped_states(const qsx_rk4_args* a, const int* only_if, cudaStream_t s);

bool rk4_mean_adjoint_supported(int m, int nsteps);
int rk4_mean_adjoint_run(const double2* D, int m, int64_t batch, int nsteps, const double2* y0,
                         int64_t y0_stride, const double2* c, const double2* g, double scale,
                         double2* gradD, int* flag, cudaStream_t s);

}  // namespace qsx
