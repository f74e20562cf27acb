// Doubling form of the RK4 loop for few samples (rk4_traj.cu).
#pragma once
#include "qsx_common.cuh"

namespace qsx {

enum TrajForm { TRAJ_NONE = 0, TRAJ_CTA = 1, TRAJ_SPREAD = 2 };

struct TrajPlan {
  TrajForm form;
  int64_t mats;   // distinct propagators
  int stop;       // TRAJ_SPREAD: steps of the last power
  int sms;
  size_t bytes;   // workspace: an int flag (16 bytes), then the powers
};

// The form for these arguments: TRAJ_NONE where the stepped loop is sooner
// done, or where it is the only one (projections, stages, m > 512).
int rk4_traj_plan(const qsx_rk4_args* a, TrajPlan* pl);
// Runs it in a->workspace; the int at its start is nonzero afterwards (on the
// device) when a value was not finite and the stepped loop has to run.
int rk4_traj_run(const qsx_rk4_args* a, const TrajPlan& pl, cudaStream_t s);
// D = P - I of few samples in FP64, a CTA per row.
int propagator_rows_run(const double2* L, int m, int64_t batch, double h, double2* D,
                        cudaStream_t s);

}  // namespace qsx
