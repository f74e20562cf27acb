// FP64 ensemble mean of the populations and coherences of a Hermitian block,
// in its real form (hermitian coordinates, see hermitian_propagator_kernel):
// x_{n+1} = x_n + D x_n with D real m x m, m = nb^2, mean over samples of the
// selected coordinates at every step (simulate_dynamics with ensemble_size,
// qspectra/simulate/eom.py:11-74, decorators.py:40-64).
//
// A quarter of the complex loop's multiply-adds, and the FP64 pipe (2 a clock
// and SM, a warp instruction every 16 clocks) is what bounds it, so the layout
// is chosen to keep its lanes full: a thread owns one row of D, in registers,
// and the rows of G samples are packed side by side (49 rows alone would pay
// for 64 lanes).  The state goes round through shared memory, read as 16-byte
// broadcasts; one barrier a step.  The first lanes add the CTA's samples and
// write one partial row a step, a fixed-order reduction follows.
//
// simulate_dynamics of 300 7-site samples, 499 steps: 5.66 ms with the complex
// loop (a CTA per sample, two barriers a step) and its propagators, 2.36 ms
// with the real ones (1.89 ms as the call is now, the loop 1.04 of it).
#include <algorithm>

#include "qsx_common.cuh"

namespace qsx {

namespace {

constexpr int R64_THREADS = 256;

struct Real64P {
  const double *D, *x0;
  const int* sel;
  double* partial;          // [grid][nsteps + 1][nsel]
  int* status;
  int nsteps, nsel, G;
  int64_t batch, ngroups;
};

template <int M>
__global__ void __launch_bounds__(R64_THREADS) real64_kernel(Real64P p) {
  constexpr int LD = (M + 1) & ~1;       // 16-byte rows
  extern __shared__ __align__(16) double xs[];   // [2][G][LD]
  const int tid = threadIdx.x, G = p.G;
  const int g = min(tid / M, G - 1), r = tid % M;
  const bool active = tid < G * M;
  double* dst = p.partial + (int64_t)blockIdx.x * (p.nsteps + 1) * p.nsel;
  int si = -1;
  if (tid < p.nsel) {
    si = p.sel[tid];
    if (si < 0 || si >= M) {   // bad index table: record it, touch nothing
      if (p.status) atomicOr(p.status, QSX_ERR_INVALID_ARG);
      si = -1;
    }
  }
  for (int e = tid; e < 2 * G * LD; e += blockDim.x) xs[e] = 0.0;
  __syncthreads();
  bool first = true;
  for (int64_t grp = blockIdx.x; grp < p.ngroups; grp += gridDim.x, first = false) {
    const int64_t s = grp * G + g;
    const bool valid = active && s < p.batch;
    double row[LD], x = 0.0;
    const double* d = p.D + (valid ? s * M * M + (int64_t)r * M : 0);
#pragma unroll
    for (int j = 0; j < LD; ++j) row[j] = valid && j < M ? d[j] : 0.0;
    if (valid) x = p.x0[r];
    if (active) xs[g * LD + r] = x;   // samples past the batch stay zero
    __syncthreads();
    const int live = (int)min((int64_t)G, p.batch - grp * G);
    for (int n = 0; n <= p.nsteps; ++n) {
      const double* cur = xs + (n & 1) * G * LD;
      if (si >= 0) {
        double sum = cur[si];
        for (int q = 1; q < live; ++q) sum += cur[q * LD + si];
        double* o = dst + (int64_t)n * p.nsel + tid;
        *o = first ? sum : *o + sum;
      }
      if (n == p.nsteps) break;
      const double2* v = reinterpret_cast<const double2*>(cur + g * LD);
      double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
#pragma unroll
      for (int j = 0; j < LD / 2; ++j) {
        const double2 w = v[j];
        if (j & 1) {
          a2 = fma(row[2 * j], w.x, a2);
          if (2 * j + 1 < M) a3 = fma(row[2 * j + 1], w.y, a3);
        } else {
          a0 = fma(row[2 * j], w.x, a0);
          if (2 * j + 1 < M) a1 = fma(row[2 * j + 1], w.y, a1);
        }
      }
      x += (a0 + a1) + (a2 + a3);
      if (active) xs[((n + 1) & 1) * G * LD + g * LD + r] = x;
      __syncthreads();
    }
    if (valid && p.status && !isfinite(x)) atomicOr(p.status, QSX_ERR_NONFINITE);
    __syncthreads();
  }
}

// out[e] = scale * sum over the slots, 32 outputs a CTA, slots over 8 warps
__global__ void __launch_bounds__(256)
    real64_reduce_kernel(const double* __restrict__ partial, int64_t nslots, int64_t per,
                         double scale, double* __restrict__ out) {
  __shared__ double red[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t e = (int64_t)blockIdx.x * 32 + lane;
  double acc = 0.0;
  if (e < per)
    for (int64_t sl = w; sl < nslots; sl += 8) acc += partial[sl * per + e];
  red[w][lane] = acc;
  __syncthreads();
  if (w == 0 && e < per) {
    double t = red[0][lane];
#pragma unroll
    for (int i = 1; i < 8; ++i) t += red[i][lane];
    out[e] = t * scale;
  }
}

bool real64_size(int m) {
  return m == 4 || m == 9 || m == 16 || m == 25 || m == 36 || m == 49 || m == 64;
}

// Samples a CTA: the G whose busiest SM runs the fewest warps a step (each
// pays 16 clocks an element whether its lanes have rows or not), then the
// smallest.
int real64_plan(int m, int64_t batch, int* G, int64_t* ngroups, int64_t* grid) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return cuda_status(e, "qsx_rk4_real_mean_f64 plan");
  int64_t best = INT64_MAX;
  for (int g = 1; g * m <= R64_THREADS; ++g) {
    const int64_t groups = (batch + g - 1) / g;
    const int64_t cost = (groups + sms - 1) / sms * ((g * m + 31) / 32);
    if (cost < best) {
      best = cost;
      *G = g;
    }
  }
  *ngroups = (batch + *G - 1) / *G;
  // two CTAs an SM at most, then further groups in turn
  *grid = std::min<int64_t>(*ngroups, 2 * (int64_t)sms);
  return QSX_OK;
}

}  // namespace

}  // namespace qsx

using namespace qsx;

extern "C" size_t qsx_rk4_real_mean_f64_workspace_bytes(int m, int64_t batch, int nsteps,
                                                        int nsel) {
  int G;
  int64_t groups, grid;
  if (!real64_size(m) || batch < 1 || nsteps < 0 || nsel < 1 ||
      real64_plan(m, batch, &G, &groups, &grid) != QSX_OK)
    return 0;
  return (size_t)grid * ((size_t)nsteps + 1) * nsel * sizeof(double);
}

extern "C" int qsx_rk4_real_mean_f64(const double* D, int m, int64_t batch, int nsteps,
                                     const double* x0, const int32_t* select, int nsel,
                                     double* out, void* workspace, size_t workspace_bytes,
                                     int32_t* status, void* stream) {
  QSX_CHECK_ARG(real64_size(m), "qsx_rk4_real_mean_f64: m = %d is not 2^2 .. 8^2", m);
  QSX_CHECK_ARG(batch >= 0 && batch <= 0x7fffffffLL && nsteps >= 0 && nsel >= 1 && nsel <= m,
                "qsx_rk4_real_mean_f64: bad sizes");
  if (batch == 0) return QSX_OK;
  QSX_CHECK_ARG(D && x0 && select && out && workspace, "qsx_rk4_real_mean_f64: null pointer");
  Real64P p;
  int64_t grid;
  int st = real64_plan(m, batch, &p.G, &p.ngroups, &grid);
  if (st) return st;
  const int64_t per = ((int64_t)nsteps + 1) * nsel;
  QSX_CHECK_ARG(workspace_bytes >= (size_t)grid * per * sizeof(double),
                "qsx_rk4_real_mean_f64: workspace of %zu bytes needed (got %zu)",
                (size_t)grid * per * sizeof(double), workspace_bytes);
  p.D = D;
  p.x0 = x0;
  p.sel = select;
  p.partial = (double*)workspace;
  p.status = status;
  p.nsteps = nsteps;
  p.nsel = nsel;
  p.batch = batch;
  cudaStream_t s = (cudaStream_t)stream;
  const int threads = std::max((p.G * m + 31) / 32 * 32, (nsel + 31) / 32 * 32);
  const size_t smem = 2 * (size_t)p.G * ((m + 1) & ~1) * sizeof(double);
  switch (m) {
#define R(MM) case MM: real64_kernel<MM><<<(unsigned)grid, threads, smem, s>>>(p); break;
    R(4) R(9) R(16) R(25) R(36) R(49) R(64)
#undef R
  }
  QSX_LAUNCH_CHECK("qsx_rk4_real_mean_f64");
  real64_reduce_kernel<<<(unsigned)((per + 31) / 32), 256, 0, s>>>(
      (const double*)workspace, grid, per, 1.0 / (double)batch, out);
  QSX_LAUNCH_CHECK("qsx_rk4_real_mean_f64 reduce");
  return QSX_OK;
}
