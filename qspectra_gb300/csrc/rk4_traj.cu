// Trajectories of a constant propagator by doubling, for few samples.
//
// The fixed-step RK4 loop of integrate() (qspectra/simulate/utils.py:16-109)
// is y_{n+1} = y_n + D y_n.  Run step by step it is one dependent chain per
// sample: with one 49-element state, 8 us a step on one SM, the others idle.
// With D_n = P^n - I the states come in doubling blocks instead,
//   y_{n + j} = y_j + D_n y_j   (j < n),    D_{2n} = 2 D_n + D_n D_n,
// log2 T dependent phases whose T m^2 + log2(T) m^3 multiply-adds are
// independent within a phase and spread over every SM.  Large blocks stop
// squaring early and go on in blocks of that many states: a square of 252
// elements costs as much as 250 states.  All of it runs in FP64, for
// single-precision propagators too.
//
// The powers are kept transposed, DT[c][r] = D[r][c]: then a square and a
// block of states are the same operation on rows x (of DT, or of states),
//   out[j][r] = x[j][r] (+ add[j][r]) + sum_k DT[k][r] x[j][k],
// with coalesced loads of DT and broadcast loads of x.
//
// Bound: FP64 issue (2 multiply-adds per clock and SM) once a phase fills the
// chip, launch latency before that.  Whole calls in FP64, with the stepped loop
// and as they are now: a 7-site trajectory (49 elements, 1000 states) 8.52 and
// 0.42 ms, a 7-site spectrum (7 elements, 2048 states) 5.11 and 0.82 ms, a dimer
// trajectory (4 elements, 120 states) 0.51 and 0.32 ms, a trimer hierarchy
// through its dense propagator (252 elements, 500 states) 12.6 and 1.64 ms.
// Rounding: a few ulp more than the steps leave (error against 64-bit formulas
// 9e-16 and 1.5e-15 for the 7 sites, 2e-16 and 7e-16 for the trimer), as the
// powers' own rounding is shared by the states of a block.
//
// A power can overflow, or meet a non-finite generator, where the stepped
// loop would not (an unstable mode that the state does not excite).  Every
// value is tested (states of a single-precision run against that range: the
// stepped loop keeps them in FP32); the caller runs the stepped loop instead when one is not
// finite (rk4_traj_run returns the device flag to guard it).
#include <math.h>

#include <algorithm>

#include "qsx_common.cuh"
#include "rk4_traj.cuh"

namespace qsx {

namespace {

template <bool SINGLE>
__device__ __forceinline__ bool state_finite(double2 v) {
  return SINGLE ? isfinite((float)v.x) && isfinite((float)v.y) : finite2(v);
}

constexpr int TRAJ_THREADS = 128;
constexpr int TRAJ_CTA_THREADS = 256;

struct TrajJob {
  const double2* x;
  const double2* add;   // or null
  double2* out;
  int64_t x_stride, add_stride, out_stride;  // elements between samples
  int rows, batch;
};

// sum over k = k0, k0 + step, .. < m of DT[k][r] x[k], eight independent
// chains of multiply-adds: a dependent one takes 140 clocks, an issue 16
__device__ __forceinline__ double2 traj_dot(const double2* dt, const double2* x, int m, int k0 = 0,
                                            int step = 1) {
  double a[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  int k = k0;
#pragma unroll 2
  for (; k + step < m; k += 2 * step) {
    const double2 d0 = dt[(int64_t)k * m], v0 = x[k];
    const double2 d1 = dt[(int64_t)(k + step) * m], v1 = x[k + step];
    a[0] = fma(d0.x, v0.x, a[0]);
    a[1] = fma(-d0.y, v0.y, a[1]);
    a[2] = fma(d0.x, v0.y, a[2]);
    a[3] = fma(d0.y, v0.x, a[3]);
    a[4] = fma(d1.x, v1.x, a[4]);
    a[5] = fma(-d1.y, v1.y, a[5]);
    a[6] = fma(d1.x, v1.y, a[6]);
    a[7] = fma(d1.y, v1.x, a[7]);
  }
  if (k < m) {
    const double2 d0 = dt[(int64_t)k * m], v0 = x[k];
    a[0] = fma(d0.x, v0.x, a[0]);
    a[1] = fma(-d0.y, v0.y, a[1]);
    a[2] = fma(d0.x, v0.y, a[2]);
    a[3] = fma(d0.y, v0.x, a[3]);
  }
  return make_double2((a[0] + a[1]) + (a[4] + a[5]), (a[2] + a[3]) + (a[6] + a[7]));
}

// output e of the job by `parts` neighbouring lanes, this one's share k = part, ..
template <bool SINGLE>
__device__ __forceinline__ void traj_output(const TrajJob& job, const double2* dt_all,
                                            int64_t dt_stride, int m, unsigned e, bool live,
                                            int parts, int part, int* flag) {
  const unsigned r = e % m, row = e / m, j = row % job.rows, b = row / job.rows;
  const double2* x = job.x + b * job.x_stride + (int64_t)j * m;
  double2 z = make_double2(0.0, 0.0);
  if (live) z = traj_dot(dt_all + b * dt_stride + r, x, m, part, parts);
  for (int o = 16; o >= 32 / parts; o >>= 1) {
    z.x += __shfl_xor_sync(0xffffffffu, z.x, o);
    z.y += __shfl_xor_sync(0xffffffffu, z.y, o);
  }
  if (!live || part) return;
  double2 v = x[r];
  if (job.add) v = cadd(v, job.add[b * job.add_stride + (int64_t)j * m + r]);
  v = cadd(v, z);
  job.out[b * job.out_stride + (int64_t)j * m + r] = v;
  if (!state_finite<SINGLE>(v)) atomicOr(flag, 1);
}

template <typename C>
__global__ void __launch_bounds__(256)
    traj_init_kernel(const C* __restrict__ D, int64_t d_stride, int m, int mat_batch,
                     const double2* __restrict__ y0, int64_t y0_stride, int batch, int64_t nsave,
                     double2* __restrict__ DT, double2* __restrict__ state,
                     int* __restrict__ flag) {
  const int64_t mm = (int64_t)m * m, nmat = mm * mat_batch;
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < nmat) {
    const int64_t b = e / mm, c = e % mm / m, r = e % m;
    const C v = D[b * d_stride + r * m + c];
    DT[e] = make_double2((double)v.x, (double)v.y);
  } else if (e < nmat + (int64_t)batch * m) {
    const int64_t q = e - nmat, b = q / m, r = q % m;
    state[b * nsave * m + r] = y0[b * y0_stride + r];
  }
  if (e == 0) *flag = 0;
}

// A warp takes 32 / parts consecutive outputs of one job: lane l the output
// l % (32 / parts), its share l / (32 / parts) of the sum.
template <bool SINGLE>
__global__ void __launch_bounds__(TRAJ_THREADS)
    traj_phase_kernel(TrajJob rows, TrajJob power, const double2* DT, int64_t dt_stride, int m,
                      int parts, int* flag) {
  const unsigned per = 32 / parts, lane = threadIdx.x & 31;
  const unsigned nr = (unsigned)rows.rows * rows.batch * m;
  const unsigned np = (unsigned)power.rows * power.batch * m;
  const unsigned wr = (nr + per - 1) / per;   // warps of the first job
  const unsigned w = blockIdx.x * (TRAJ_THREADS / 32) + threadIdx.x / 32;
  const int part = lane / per;
  if (w < wr) {
    const unsigned e = w * per + lane % per;
    traj_output<SINGLE>(rows, DT, dt_stride, m, min(e, nr - 1), e < nr, parts, part, flag);
  } else {
    const unsigned e = (w - wr) * per + lane % per;
    if ((w - wr) * per >= np) return;   // whole warps
    traj_output<false>(power, DT, power.x_stride, m, min(e, np - 1), e < np, parts, part, flag);
  }
}

// Every phase in one launch, one CTA per sample, the powers in shared memory:
// for work that one SM finishes sooner than the phases' launches take.
template <typename C>
__global__ void __launch_bounds__(TRAJ_CTA_THREADS)
    traj_cta_kernel(const C* __restrict__ D, int64_t d_stride, int m,
                    const double2* __restrict__ y0, int64_t y0_stride, int nsave, double2* state,
                    int* flag) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* dt = reinterpret_cast<double2*>(smraw);
  double2* next = dt + m * m;
  const int64_t b = blockIdx.x;
  double2* ys = state + b * (int64_t)nsave * m;
  bool bad = false;
  for (int e = threadIdx.x; e < m * m; e += TRAJ_CTA_THREADS) {
    const C v = D[b * d_stride + (int64_t)(e % m) * m + e / m];
    dt[e] = make_double2((double)v.x, (double)v.y);
  }
  for (int e = threadIdx.x; e < m; e += TRAJ_CTA_THREADS) {
    const double2 v = y0[b * y0_stride + e];
    bad |= !finite2(v);
    ys[e] = v;
  }
  __syncthreads();
  for (int n = 1; n < nsave; n *= 2) {
    const int cnt = min(n, nsave - n);
    const int nr = cnt * m, total = nr + (2 * n < nsave ? m * m : 0);
    for (int e = threadIdx.x; e < total; e += TRAJ_CTA_THREADS) {
      const bool st = e < nr;
      const int q = st ? e : e - nr, j = q / m, r = q % m;
      const double2* x = (st ? ys : dt) + (int64_t)j * m;
      const double2 z = traj_dot(dt + r, x, m);
      double2 v = cadd(x[r], z);
      if (!st) v = cadd(x[r], v);
      (st ? ys + (int64_t)n * m : next)[q] = v;
      bad |= !(st ? state_finite<sizeof(C) == 8>(v) : finite2(v));
    }
    __syncthreads();   // this CTA's states in global memory are visible to it
    double2* t = dt;
    dt = next;
    next = t;
  }
  if (bad) atomicOr(flag, 1);
}

// --------------------------------------------------------------- propagator
// D = P - I of few samples, one CTA per row: with A = h L the row of
// A + A^2/2 + A^3/6 + A^4/24 needs row r alone, r A (I + A/2 (I + A/3 (I + A/4)))
// evaluated left to right, so m CTAs a sample share nothing.  Three products
// where the two-product form of the batched kernel needs the whole of A^2 in
// one CTA: 256 us for one 49 x 49 block, on one SM, where this takes 24.
__global__ void __launch_bounds__(64)
    propagator_rows_kernel(const double2* __restrict__ L, int m, double h,
                           double2* __restrict__ D) {
  __shared__ double2 row[2][64];
  const int r = blockIdx.x, c = threadIdx.x;
  const int64_t base = (int64_t)blockIdx.y * m * m;
  const double2* l = L + base;
  double2 sum = make_double2(0.0, 0.0);
  if (c < m) {
    sum = cscale(l[(int64_t)r * m + c], h);
    row[0][c] = sum;
  }
  __syncthreads();
  const double fac[3] = {0.5, 1.0 / 3.0, 0.25};
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (c < m) {
      const double2 v = cscale(traj_dot(l + c, row[q & 1], m), h * fac[q]);
      row[(q + 1) & 1][c] = v;
      sum = cadd(sum, v);
    }
    __syncthreads();
  }
  if (c < m) D[base + (int64_t)r * m + c] = sum;
}

}  // namespace

int propagator_rows_run(const double2* L, int m, int64_t batch, double h, double2* D,
                        cudaStream_t s) {
  propagator_rows_kernel<<<dim3((unsigned)m, (unsigned)batch), 64, 0, s>>>(L, m, h, D);
  QSX_LAUNCH_CHECK("qsx_rk4_propagator_batched rows");
  return QSX_OK;
}

// --------------------------------------------------------------------- plan
int rk4_traj_plan(const qsx_rk4_args* a, TrajPlan* pl) {
  pl->form = TRAJ_NONE;
  const int64_t m = a->m, B = a->batch, nsave = a->nsteps / a->save_every + 1;
  if (a->form != 0 || !a->out_state || a->nproj || a->nselect || a->block_k > 1 || m > 512 ||
      a->variant || nsave < 8 || B < 1 || B * nsave * m >= (int64_t)1 << 31 ||
      (a->matrix_stride != 0 && B * m * m >= (int64_t)1 << 31))
    return QSX_OK;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return cuda_status(e, "qsx_rk4 trajectory plan");
  const int64_t mats = a->matrix_stride ? B : 1;
  int phases = 0, power = 0;
  for (int64_t n = 1; n < nsave; n *= 2) ++phases;
  for (int k = a->save_every; k > 1; k >>= 1) power += 1 + (k & 1);
  // Times in us, from the rates measured on GB300 (152 SMs, 1.92 GHz, 3840
  // FP64 multiply-adds per us and SM).
  const double rows = 4.0 * nsave * m * m, sq = 4.0 * m * m * m, sm_rate = 3840.0;
  // stepped loop: FP64 0.9 + 0.145 m a step while the chip is not full, then
  // its FP64 issue (a warp's 32 lanes pay for every row of a 32-row group);
  // FP32 0.25 a step, then its issue
  const double per_sm = (double)B / sms;
  const double chain =
      a->precision == QSX_FP64
          ? a->nsteps * std::max(0.9 + 0.145 * m, per_sm * 4.0 * m * ((m + 31) / 32 * 32) / sm_rate)
          : a->nsteps * std::max(0.25, per_sm * 4.0 * m * m / (16.0 * sm_rate));
  // one launch, a CTA per sample
  const double waves = std::ceil(per_sm);
  const double cta = a->save_every == 1 && m <= 64
                         ? 4.0 + waves * (0.6 * phases + (rows + phases * sq) / sm_rate)
                         : 1e30;
  // a launch a phase, outputs spread over all SMs: squares up to D_stop, then
  // blocks of `stop` states
  const double rate = 0.7 * sm_rate * sms;
  double spread = 1e30;
  double squares = 0.0;
  const double phase = 3.0 + 0.01 * m;   // launch, and a shared sum's latency
  for (int64_t stop = 1, q = 0; ; stop *= 2, ++q) {
    const double blocks = (double)((nsave - stop + stop - 1) / stop);
    const double t = 4.0 + (power + q + blocks) * phase + mats * power * sq / rate + squares +
                     B * rows / rate;
    if (t < spread) {
      spread = t;
      pl->stop = (int)stop;
    }
    if (stop >= nsave || stop >= (int64_t)1 << 30) break;
    squares += mats * sq / rate;   // D_{2 stop}
  }
  if (std::min(cta, spread) >= chain) return QSX_OK;
  pl->form = cta < spread ? TRAJ_CTA : TRAJ_SPREAD;
  pl->mats = mats;
  pl->sms = sms;
  const int bufs = pl->form == TRAJ_CTA ? 0 : a->save_every > 1 ? 4 : 2;
  pl->bytes = 16 + (size_t)bufs * mats * m * m * sizeof(double2);
  return QSX_OK;
}

template <typename C>
static int traj_run(const qsx_rk4_args* a, const TrajPlan& pl, cudaStream_t s) {
  const int m = a->m;
  const int64_t mm = (int64_t)m * m, nsave = a->nsteps / a->save_every + 1;
  int* flag = (int*)a->workspace;
  double2* state = (double2*)a->out_state;
  const double2* y0 = (const double2*)a->y0;
  if (pl.form == TRAJ_CTA) {
    const size_t smem = 2 * mm * sizeof(double2);
    cudaError_t e = cudaFuncSetAttribute(traj_cta_kernel<C>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) e = cudaMemsetAsync(flag, 0, sizeof(int), s);
    if (e != cudaSuccess) return cuda_status(e, "qsx_rk4_batched trajectory");
    traj_cta_kernel<C><<<(unsigned)a->batch, TRAJ_CTA_THREADS, smem, s>>>(
        (const C*)a->matrix, a->matrix_stride, m, y0, a->y0_stride, (int)nsave, state, flag);
    QSX_LAUNCH_CHECK("qsx_rk4_batched trajectory");
    return QSX_OK;
  }
  double2* buf = (double2*)((char*)a->workspace + 16);
  const int64_t per = pl.mats * mm;
  double2 *cur = buf, *spare = buf + per;
  const int64_t init = per + a->batch * m;
  traj_init_kernel<C><<<(unsigned)((init + 255) / 256), 256, 0, s>>>(
      (const C*)a->matrix, a->matrix_stride, m, (int)pl.mats, y0, a->y0_stride, (int)a->batch,
      nsave, cur, state, flag);
  QSX_LAUNCH_CHECK("qsx_rk4_batched trajectory init");
  const int64_t ms = pl.mats > 1 ? mm : 0;   // powers shared by all samples, or one each
  auto launch = [&](const TrajJob& rows, const TrajJob& power, const double2* dt) {
    // few outputs: lanes share each one's sum until every SM has four warps
    // (or a share is down to eight terms)
    const int64_t nr = (int64_t)rows.rows * rows.batch * m;
    const int64_t np = (int64_t)power.rows * power.batch * m;
    int parts = 1;
    while (parts < 16 && (nr + np) * parts < (int64_t)pl.sms * 128 && m >= 16 * parts) parts *= 2;
    const int64_t per = 32 / parts, warps = (nr + per - 1) / per + (np + per - 1) / per;
    const int64_t wpc = TRAJ_THREADS / 32;
    traj_phase_kernel<sizeof(C) == 8><<<(unsigned)((warps + wpc - 1) / wpc), TRAJ_THREADS, 0, s>>>(
        rows, power, dt, ms, m, parts, flag);
  };
  const TrajJob none = {nullptr, nullptr, nullptr, 0, 0, 0, 0, 0};
  auto square = [&](const double2* dt, double2* out) {
    return TrajJob{dt, dt, out, mm, mm, mm, m, (int)pl.mats};
  };
  if (a->save_every > 1) {   // D of save_every steps, by binary powering
    double2 *res = nullptr, *free1 = buf + 2 * per, *free2 = buf + 3 * per;
    for (int k = a->save_every; k > 0; k >>= 1) {
      if (k & 1) {
        if (!res) {
          cudaError_t e = cudaMemcpyAsync(free1, cur, per * sizeof(double2),
                                          cudaMemcpyDeviceToDevice, s);
          if (e != cudaSuccess) return cuda_status(e, "qsx_rk4_batched trajectory power");
          res = free1;
        } else {   // (I + X)(I + Y) - I = X + Y + X Y
          double2* o = res == free1 ? free2 : free1;
          launch(none, TrajJob{res, cur, o, mm, mm, mm, m, (int)pl.mats}, cur);
          res = o;
        }
      }
      if (k > 1) {
        launch(none, square(cur, spare), cur);
        std::swap(cur, spare);
      }
    }
    spare = cur;
    cur = res;
  }
  for (int64_t n = 1; n < nsave;) {
    // states n .. from the `block` before them
    const int64_t block = std::min<int64_t>(n, pl.stop);
    const int cnt = (int)std::min(block, nsave - n);
    const TrajJob rows = {state + (n - block) * m, nullptr, state + n * m, nsave * m, 0,
                          nsave * m, cnt, (int)a->batch};
    const bool more = n < pl.stop && 2 * n < nsave;
    launch(rows, more ? square(cur, spare) : none, cur);
    if (more) std::swap(cur, spare);
    n += cnt;
  }
  QSX_LAUNCH_CHECK("qsx_rk4_batched trajectory");
  return QSX_OK;
}

int rk4_traj_run(const qsx_rk4_args* a, const TrajPlan& pl, cudaStream_t s) {
  return a->precision == QSX_FP32 ? traj_run<float2>(a, pl, s) : traj_run<double2>(a, pl, s);
}

}  // namespace qsx
