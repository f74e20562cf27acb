// Direct DFT of uniformly sampled signals at arbitrary frequencies (FP64),
// replacing fourier_transform (qspectra/simulate/utils.py:154-219).
//
// The reference zero-pads to a symmetric time grid and runs an FFT; padded
// zeros contribute nothing, so on the FFT frequency grid the result equals
//   X(f) = dt * sum_n x_n exp(i * sign * (f - rw) * uc * t_n)
// which these kernels evaluate directly (any grid, e.g. 1024 points in a
// window), sums of 32 samples at a time by Horner's rule in z = e^{i Delta}
// (four multiply-adds a sample; a twiddle advanced by rotation takes eight, and
// the FP64 pipe is the bound), the sums by Horner's rule in z^32, the phase of
// the first sample from sincos.
#include "qsx_common.cuh"

namespace qsx {

struct DftPhase {
  double2 z, z32;   // e^{i w dt}, e^{i 32 w dt}
};

__device__ __forceinline__ double2 dft_cis(double a) {
  double2 r;
  sincos(a, &r.y, &r.x);
  return r;
}
__device__ __forceinline__ DftPhase dft_phase(double wdt) {
  return {dft_cis(wdt), dft_cis(32.0 * wdt)};
}
__device__ __forceinline__ double2 dft_cmul(double2 a, double2 b) {
  return make_double2(fma(a.x, b.x, -(a.y * b.y)), fma(a.x, b.y, a.y * b.x));
}
// a z + x
__device__ __forceinline__ double2 dft_step(double2 a, double2 z, double2 x) {
  return make_double2(fma(a.x, z.x, fma(-a.y, z.y, x.x)), fma(a.x, z.y, fma(a.y, z.x, x.y)));
}

// sum over n < count of x[n stride] z^n
__device__ __forceinline__ double2 dft_sum(const double2* x, int64_t stride, int count,
                                           const DftPhase& p) {
  double2 total = make_double2(0.0, 0.0);
  for (int b = (count - 1) & ~31; b >= 0; b -= 32) {
    double2 acc = make_double2(0.0, 0.0);
#pragma unroll 4
    for (int n = min(count, b + 32) - 1; n >= b; --n) acc = dft_step(acc, p.z, x[n * stride]);
    total = dft_step(total, p.z32, acc);
  }
  return total;
}

// grid (ceil(nf / 8), batch), 128 threads: 8 frequencies per CTA, each summed
// over 16 time slices (lane / 8 and the warp pick the slice) that meet in shared
// memory in a fixed order.  A thread's three sincos cost as much as 60 samples,
// so 16 slices and not more; 2048 samples at 4095 frequencies took 163 us with
// rotated twiddles and 32 slices, 86 now.
constexpr int DFT_SLICES = 16;

__global__ void __launch_bounds__(8 * DFT_SLICES)
    dft_kernel(const double2* __restrict__ x, int nt, double t0, double dt,
               const double* __restrict__ freqs, int nf, double rw, double uc, int sign,
               double2* __restrict__ X) {
  __shared__ double2 part[DFT_SLICES][8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int kl = lane & 7, slice = w * 4 + (lane >> 3);
  const int64_t b = blockIdx.y;
  const int k = blockIdx.x * 8 + kl;
  const double wk = k < nf ? (double)sign * (freqs[k] - rw) * uc : 0.0;
  const DftPhase p = dft_phase(wk * dt);
  const int chunk = (nt + DFT_SLICES - 1) / DFT_SLICES;
  const int n0 = slice * chunk, n1 = min(nt, n0 + chunk);
  double2 acc = make_double2(0.0, 0.0);
  if (n0 < n1)
    acc = dft_cmul(dft_sum(x + b * nt + n0, 1, n1 - n0, p), dft_cis(wk * (t0 + (double)n0 * dt)));
  part[slice][kl] = acc;
  __syncthreads();
  if (threadIdx.x < 8 && k < nf) {
    double2 t = part[0][kl];
#pragma unroll
    for (int i = 1; i < DFT_SLICES; ++i) t = cadd(t, part[i][kl]);
    X[b * nf + k] = cscale(t, dt);
  }
}

// The same sum for signals that come from FP32 propagation: the phase is
// anchored in FP64 at the start of each time slice (one sincos a thread),
// then rotated and accumulated in FP32 over the slice (at most 128 samples,
// a relative drift of order 1e-5 at worst), with the slices added in FP64.
// The signal is read once per CTA and converted to FP32 in shared memory, so
// the inner loop issues no FP64 work.
__global__ void __launch_bounds__(256)
    dft_f32_kernel(const double2* __restrict__ x, int nt, double t0, double dt,
                   const double* __restrict__ freqs, int nf, double rw, double uc, int sign,
                   double2* __restrict__ X) {
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* sx = reinterpret_cast<float2*>(smraw);   // [nt]
  __shared__ double2 part[32][8];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int kl = lane & 7, slice = w * 4 + (lane >> 3);
  const int64_t b = blockIdx.y;
  const int k = blockIdx.x * 8 + kl;
  const double2* xb = x + b * nt;
  for (int n = threadIdx.x; n < nt; n += blockDim.x) {
    const double2 v = xb[n];
    sx[n] = make_float2((float)v.x, (float)v.y);
  }
  __syncthreads();
  const double wk = k < nf ? (double)sign * (freqs[k] - rw) * uc : 0.0;
  double sd, cd;
  sincos(wk * dt, &sd, &cd);
  const float sdf = (float)sd, cdf = (float)cd;
  const int chunk = (nt + 31) / 32;
  const int n0 = slice * chunk, n1 = min(nt, n0 + chunk);
  double2 acc = make_double2(0.0, 0.0);
  float2 ph = make_float2(1.f, 0.f), a32 = make_float2(0.f, 0.f);
  for (int n = n0; n < n1; ++n) {
    if (((n - n0) & 127) == 0) {   // FP64 anchor (at most every 128 samples)
      acc.x += (double)a32.x;
      acc.y += (double)a32.y;
      a32 = make_float2(0.f, 0.f);
      double s, c;
      sincos(wk * (t0 + (double)n * dt), &s, &c);
      ph = make_float2((float)c, (float)s);
    }
    const float2 v = sx[n];
    a32.x = fmaf(v.x, ph.x, fmaf(-v.y, ph.y, a32.x));
    a32.y = fmaf(v.x, ph.y, fmaf(v.y, ph.x, a32.y));
    ph = make_float2(ph.x * cdf - ph.y * sdf, ph.x * sdf + ph.y * cdf);
  }
  acc.x += (double)a32.x;
  acc.y += (double)a32.y;
  part[slice][kl] = acc;
  __syncthreads();
  if (threadIdx.x < 8 && k < nf) {
    double2 t = part[0][kl];
#pragma unroll
    for (int i = 1; i < 32; ++i) t = cadd(t, part[i][kl]);
    X[b * nf + k] = cscale(t, dt);
  }
}

// Two-dimensional transform of a third-order signal x[n1][b][n3] (t1, t2,
// t3; any strides) over t1 and t3 in one launch (FP64):
//   X[k1][b][k3] = dt1 dt3 sum_{n1, n3} x[n1][b][n3]
//                  exp(i s1 (f1_k1 - rw) uc t1_n1) exp(i s3 (f3_k3 - rw) uc t3_n3),
// t_n = t0 + n dt on each axis.  CTA (chunk of F3 t3 frequencies, b): first the
// t3 transform of every t1 row for those frequencies, into shared memory
// (Y[n1][F3]); then the t1 transform of Y for every t1 frequency.  The bound is
// each SM's FP64 pipe: a CTA costs as F3 (n1 = n3 = 100: 85, 160 and 310 us for
// 2, 4 and 8), and those on one SM share it, so F3 is the one of 8, 4, 2 whose
// busiest SM has the least to do (the largest of equals, which repeats the fewest
// loads).  us with F3 = 8, 4, 2 on 152 SMs: 64 x 5 x 64 140, 143, 118; 100 x 3 x
// 100 321, 175, 173 (652 with rotated twiddles); 100 x 4 x 100 320, 315, 252; 128 x
// 5 x 128 908, 691, 593; 60 x 3 x 200 195, 205, 224.
template <int F3>
__global__ void __launch_bounds__(256)
    dft2_kernel(const double2* __restrict__ x, int n1, int n3, int64_t s1, int64_t sb,
                int64_t s3, double t01, double dt1, const double* __restrict__ f1, int nf1,
                int sign1, double t03, double dt3, const double* __restrict__ f3, int nf3,
                int sign3, double rw, double uc, double2* __restrict__ X) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* Y = reinterpret_cast<double2*>(smraw);   // [n1][F3]
  const int kl = threadIdx.x % F3, k = blockIdx.x * F3 + kl;
  const int64_t b = blockIdx.y;
  const int64_t nb = gridDim.y;
  const double2* xb = x + b * sb;
  // t3 transform: one (n1, k3) sum a thread, the thread's k3 the same in all
  if (k < nf3) {
    const double wk = (double)sign3 * (f3[k] - rw) * uc;
    const DftPhase p = dft_phase(wk * dt3);
    const double2 first = dft_cis(wk * t03);
    for (int r = threadIdx.x / F3; r < n1; r += 256 / F3)
      Y[r * F3 + kl] =
          cscale(dft_cmul(dft_sum(xb + (int64_t)r * s1, s3, n3, p), first), dt3);
  }
  __syncthreads();
  // t1 transform: one (k1, k3) sum a thread
  if (k >= nf3) return;
  for (int k1 = threadIdx.x / F3; k1 < nf1; k1 += 256 / F3) {
    const double wk = (double)sign1 * (f1[k1] - rw) * uc;
    const double2 sum = dft_sum(Y + kl, F3, n1, dft_phase(wk * dt1));
    X[((int64_t)k1 * nb + b) * nf3 + k] = cscale(dft_cmul(sum, dft_cis(wk * t01)), dt1);
  }
}

}  // namespace qsx

extern "C" int qsx_dft_batched_f32(const double* x, int nt, int64_t batch, double t0, double dt,
                                   const double* freqs, int nf, double rw_freq,
                                   double unit_convert, int sign, double* X, void* stream) {
  QSX_CHECK_ARG(nt >= 1 && nt <= 24576 && nf >= 1 && batch >= 0 && batch <= 65535,
                "qsx_dft_batched_f32: bad sizes nt=%d nf=%d (nt <= 24576)", nt, nf);
  QSX_CHECK_ARG(sign == 1 || sign == -1, "qsx_dft_batched_f32: sign must be +1 or -1");
  if (batch == 0) return QSX_OK;
  QSX_CHECK_ARG(x && freqs && X, "qsx_dft_batched_f32: null pointer");
  const size_t smem = (size_t)nt * sizeof(float2);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(qsx::dft_f32_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return qsx::cuda_status(e, "qsx_dft_batched_f32");
  }
  dim3 grid((unsigned)((nf + 7) / 8), (unsigned)batch);
  qsx::dft_f32_kernel<<<grid, 256, smem, (cudaStream_t)stream>>>(
      (const double2*)x, nt, t0, dt, freqs, nf, rw_freq, unit_convert, sign, (double2*)X);
  QSX_LAUNCH_CHECK("qsx_dft_batched_f32");
  return QSX_OK;
}

extern "C" int qsx_dft_batched(const double* x, int nt, int64_t batch, double t0, double dt,
                               const double* freqs, int nf, double rw_freq,
                               double unit_convert, int sign, double* X, void* stream) {
  QSX_CHECK_ARG(nt >= 1 && nf >= 1 && batch >= 0 && batch <= 65535,
                "qsx_dft_batched: bad sizes nt=%d nf=%d", nt, nf);
  QSX_CHECK_ARG(sign == 1 || sign == -1, "qsx_dft_batched: sign must be +1 or -1");
  if (batch == 0) return QSX_OK;
  QSX_CHECK_ARG(x && freqs && X, "qsx_dft_batched: null pointer");
  dim3 grid((unsigned)((nf + 7) / 8), (unsigned)batch);
  qsx::dft_kernel<<<grid, 8 * qsx::DFT_SLICES, 0, (cudaStream_t)stream>>>(
      (const double2*)x, nt, t0, dt, freqs, nf, rw_freq, unit_convert, sign, (double2*)X);
  QSX_LAUNCH_CHECK("qsx_dft_batched");
  return QSX_OK;
}

extern "C" int qsx_dft2_batched(const double* x, int n1, int64_t batch, int n3, int64_t s1,
                                int64_t sb, int64_t s3, double t01, double dt1,
                                const double* f1, int nf1, int sign1, double t03, double dt3,
                                const double* f3, int nf3, int sign3, double rw_freq,
                                double unit_convert, double* X, void* stream) {
  QSX_CHECK_ARG(n1 >= 1 && n3 >= 1 && nf1 >= 1 && nf3 >= 1 && batch >= 0 && batch <= 65535,
                "qsx_dft2_batched: bad sizes n1=%d n3=%d nf1=%d nf3=%d", n1, n3, nf1, nf3);
  QSX_CHECK_ARG((sign1 == 1 || sign1 == -1) && (sign3 == 1 || sign3 == -1),
                "qsx_dft2_batched: signs must be +1 or -1");
  if (batch == 0) return QSX_OK;
  QSX_CHECK_ARG(x && f1 && f3 && X, "qsx_dft2_batched: null pointer");
  QSX_CHECK_ARG((size_t)n1 * 8 * sizeof(double2) <= 200 * 1024,
                "qsx_dft2_batched: n1 = %d too long (at most %d)", n1,
                (int)(200 * 1024 / (8 * sizeof(double2))));
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return qsx::cuda_status(e, "qsx_dft2_batched");
  auto run = [&](auto kern, int chunk) -> int {
    const size_t smem = (size_t)n1 * chunk * sizeof(double2);
    if (smem > 48 * 1024) {
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return qsx::cuda_status(e, "qsx_dft2_batched");
    }
    const dim3 grid((unsigned)((nf3 + chunk - 1) / chunk), (unsigned)batch);
    kern<<<grid, 256, smem, (cudaStream_t)stream>>>(
        (const double2*)x, n1, n3, s1, sb, s3, t01, dt1, f1, nf1, sign1, t03, dt3, f3, nf3, sign3,
        rw_freq, unit_convert, (double2*)X);
    QSX_LAUNCH_CHECK("qsx_dft2_batched");
    return QSX_OK;
  };
  // the busiest SM's frequencies
  auto load = [&](int chunk) {
    return ((int64_t)((nf3 + chunk - 1) / chunk) * batch + sms - 1) / sms * chunk;
  };
  const int64_t l8 = load(8), l4 = load(4), l2 = load(2);
  if (l8 <= l4 && l8 <= l2) return run(qsx::dft2_kernel<8>, 8);
  return l4 <= l2 ? run(qsx::dft2_kernel<4>, 4) : run(qsx::dft2_kernel<2>, 2);
}
