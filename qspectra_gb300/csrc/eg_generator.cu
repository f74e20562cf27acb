// The differentiable 'eg' Redfield generator of absorption fits and the RK4
// step of small blocks, forward and backward (no reference counterpart: the
// reference has no gradients; the formulas are those of redfield.py:41-104
// and bath.py:84-102 of qspectra).
//
// Per sample, with E, U the eigenpairs of the rotating-frame H:
//   C[c][d] = lam c0(E_d - E_c),  W[a][d] = sum_c U[a][c]^2 C[c][d],
//   G[a][b] = uc sum_d W[a][d] U[a][d] U[b][d],  L = -(G + i uc H)^T.
// One warp per sample, everything in its own shared memory, forward and
// backward one launch each: as array operations this was 300 launches and most
// of a fit step, above all the 999-term Matsubara sums written out as
// [element][term] arrays.  Misfit and gradient over 1024 7-site samples:
// 10.35 ms with the array operations, 2.33 ms with these kernels (2.06 as the
// call is now).
//
// The sums: with k in units of 2 pi T, a = gamma / 2 pi T and y = x / 2 pi T,
// the terms k^2/((k^2 - a^2)(k^2 + y^2)) and k/(..) are added directly below
// k = 24, and the rest as the series in (a/k)^2 and (y/k)^2 over the partial
// zeta sums Z(s) = sum_{24 <= k < K} k^-s, which only depend on K.  Every
// part is as well conditioned as the direct sum, so it keeps that sum's
// accuracy (the digamma form of the builds loses a digit and a half to the
// cancellation of its logarithms).  Beyond a, |y| = 6, where 16 terms of the
// series no longer reach 1e-17, all terms are added directly.
//
// Bound: FP64 issue, about 25k instructions a sample.
#include <algorithm>

#include "qsx_common.cuh"

namespace qsx {

namespace {

constexpr int FW = 4;          // warps (samples) per CTA
constexpr int FIT_NMAX = 16;
constexpr int SUM_DIRECT = 24, SUM_SERIES = 16;
constexpr double SUM_MAX = 36.0;   // largest a^2, y^2 of the series

struct MatsubaraSums {
  double a2, c, gamma, cot, zero_re, four_t, freq_t;  // freq_t = 2 T / gamma
  int K, series;                  // terms k = 1 .. K - 1; series usable for a
  double w[SUM_DIRECT];           // k / (k^2 - a^2)
  double z[2 * SUM_SERIES + 4];   // Z(s)
};

// k / (k^2 - a^2) from the frequency itself, nu / (nu^2 - gamma^2): near a
// pole its rounding then is the reference sum's
__host__ __device__ __forceinline__ double matsubara_weight(double c, double gamma, double k) {
  const double nu = c * k;
  return c * (nu / (nu * nu - gamma * gamma));
}

// c0(x) and dc0/dx, and the same at -x (bath.py:84-102 without lam; at x = 0
// the value is the reference's limit)
__device__ __forceinline__ void unit_corr_pair(const MatsubaraSums& p, double x, double2& cp,
                                               double2& dp, double2& cm, double2& dm) {
  const double y = x / p.c, y2 = y * y;
  double f1 = 0.0, f2 = 0.0, q1 = 0.0, q2 = 0.0;
  int top = p.K;
  if (p.K > SUM_DIRECT && p.series && y2 <= SUM_MAX) {
    top = SUM_DIRECT;
    double pj = 1.0, sj = 1.0, t = 1.0;
#pragma unroll
    for (int j = 0; j < SUM_SERIES; ++j) {
      f1 = fma(pj, p.z[2 + 2 * j], f1);
      f2 = fma(pj, p.z[3 + 2 * j], f2);
      q1 = fma(sj, p.z[4 + 2 * j], q1);
      q2 = fma(sj, p.z[5 + 2 * j], q2);
      t *= -y2;
      pj = fma(p.a2, pj, t);
      sj = fma(p.a2, sj, (j + 2) * t);
    }
  }
  for (int k = top - 1; k >= 1; --k) {
    const double kk = (double)k, q = 1.0 / fma(kk, kk, y2);
    const double w = k < SUM_DIRECT ? p.w[k] : matsubara_weight(p.c, p.gamma, kk);
    const double wq = w * q, wqq = wq * q;
    f1 = fma(kk, wq, f1);
    f2 += wq;
    q1 = fma(kk, wqq, q1);
    q2 += wqq;
  }
  const double c2 = 1.0 / (p.c * p.c);
  // sum w r = F1 + i x F2 and its derivative F1' + i (F2 + x F2')
  const double F1 = f1 * c2, xF2 = y * f2 * c2;
  const double dF1 = -2.0 * y * q1 * c2 / p.c, dxF2 = (f2 - 2.0 * y2 * q2) * c2 / p.c;
  const double2 a = cmk(p.cot, -1.0);
  auto value = [&](double s) {
    const double2 base = crecip(cmk(p.gamma, -s * x));
    const double2 v = cmul(a, base);
    return cscale(cmk(fma(p.four_t, F1, v.x), fma(p.four_t, s * xF2, v.y)), p.gamma);
  };
  auto deriv = [&](double s) {
    const double2 base = crecip(cmk(p.gamma, -s * x));
    const double2 v = cmul(a, cmul(base, base));   // times i below
    return cscale(cmk(fma(p.four_t, s * dF1, -v.y), fma(p.four_t, dxF2, v.x)), p.gamma);
  };
  cp = value(1.0);
  cm = value(-1.0);
  dp = deriv(1.0);
  dm = deriv(-1.0);
  if (x == 0.0) cp = cm = cmk(p.freq_t, -1.0);
}

__global__ void __launch_bounds__(256)
    unit_corr_kernel(const double* __restrict__ x, int64_t n, MatsubaraSums p,
                     double2* __restrict__ val, double2* __restrict__ der) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= n) return;
  double2 cp, dp, cm, dm;
  unit_corr_pair(p, x[e], cp, dp, cm, dm);
  val[e] = cp;
  der[e] = dp;
}

// lanes over the n x n entries of one sample
#define FIT_EACH(e) for (int e = lane; e < nn; e += 32)

struct GenP {
  const double *H, *E, *U, *lam;
  double2 *L, *c0, *d0;      // forward outputs, backward inputs
  const double2* gL;
  double *gH, *glam;         // glam per sample
  int n;
  int64_t batch;
  double uc;
};

__device__ __forceinline__ void gen_w(int nn, int n, int lane, const double* U, const double2* C,
                                      double2* W) {
  FIT_EACH(e) {
    const int a = e / n, d = e % n;
    double2 w = cmk(0.0, 0.0);
    for (int c = 0; c < n; ++c) {
      const double u = U[a * n + c], s = u * u;
      w.x = fma(s, C[c * n + d].x, w.x);
      w.y = fma(s, C[c * n + d].y, w.y);
    }
    W[e] = w;
  }
  __syncwarp();
}

__global__ void __launch_bounds__(32 * FW) gen_forward_kernel(GenP p, MatsubaraSums sums) {
  extern __shared__ __align__(16) double2 sm[];
  const int lane = threadIdx.x & 31, n = p.n, nn = n * n;
  const int64_t s = (int64_t)blockIdx.x * FW + (threadIdx.x >> 5);
  if (s >= p.batch) return;   // whole warps: no CTA barrier below
  double2* C = sm + (size_t)(threadIdx.x >> 5) * 3 * nn;
  double2* W = C + nn;
  double* U = (double*)(W + nn);
  const double* E = p.E + s * n;
  FIT_EACH(e) U[e] = p.U[s * nn + e];
  const double lam = *p.lam;
  for (int t = lane; t < n * (n + 1) / 2; t += 32) {   // pairs c <= d
    int c = 0, left = t;
    while (left >= n - c) left -= n - c++;
    const int d = c + left, f = c * n + d, b = d * n + c;
    double2 cp, dp, cm, dm;
    unit_corr_pair(sums, E[d] - E[c], cp, dp, cm, dm);
    C[f] = cscale(cp, lam);
    C[b] = cscale(cm, lam);
    p.c0[s * nn + f] = cp;
    p.c0[s * nn + b] = cm;
    p.d0[s * nn + f] = dp;
    p.d0[s * nn + b] = dm;
  }
  __syncwarp();
  gen_w(nn, n, lane, U, C, W);
  FIT_EACH(e) W[e] = cscale(W[e], U[e]);
  __syncwarp();
  FIT_EACH(e) {   // L[b][a] = -(G + i uc H)[a][b]
    const int b = e / n, a = e % n;
    double2 g = cmk(0.0, 0.0);
    for (int d = 0; d < n; ++d) {
      const double u = U[b * n + d];
      g.x = fma(W[a * n + d].x, u, g.x);
      g.y = fma(W[a * n + d].y, u, g.y);
    }
    p.L[s * nn + e] = cmk(-p.uc * g.x, -p.uc * (g.y + p.H[s * nn + a * n + b]));
  }
}

__global__ void __launch_bounds__(32 * FW) gen_backward_kernel(GenP p) {
  extern __shared__ __align__(16) double2 sm[];
  const int lane = threadIdx.x & 31, n = p.n, nn = n * n;
  const int64_t s = (int64_t)blockIdx.x * FW + (threadIdx.x >> 5);
  if (s >= p.batch) return;   // whole warps: no CTA barrier below
  double2* gG = sm + (size_t)(threadIdx.x >> 5) * 8 * nn;
  double2 *C = gG + nn, *W = C + nn, *gW = W + nn, *T = gW + nn, *gC = T + nn;
  double* U = (double*)(gC + nn);
  double *gU = U + nn, *in = gU + nn, *tmp = in + nn;
  const double *E = p.E + s * n, lam = *p.lam;
  FIT_EACH(e) {
    U[e] = p.U[s * nn + e];
    C[e] = cscale(p.c0[s * nn + e], lam);
    const double2 g = p.gL[s * nn + (e % n) * n + e / n];
    gG[e] = cmk(-g.x, -g.y);
  }
  __syncwarp();
  gen_w(nn, n, lane, U, C, W);
  FIT_EACH(e) {   // V = gG U, gW = uc U o V, T = W o U
    const int a = e / n, d = e % n;
    double2 v = cmk(0.0, 0.0);
    for (int b = 0; b < n; ++b) {
      const double u = U[b * n + d];
      v.x = fma(gG[a * n + b].x, u, v.x);
      v.y = fma(gG[a * n + b].y, u, v.y);
    }
    gU[e] = p.uc * (W[e].x * v.x + W[e].y * v.y);
    gW[e] = cscale(v, p.uc * U[e]);
    T[e] = cscale(W[e], U[e]);
  }
  __syncwarp();
  double glam = 0.0;
  FIT_EACH(e) {
    const int r = e / n, k = e % n;
    double sum = 0.0, gs = 0.0;
    double2 gc = cmk(0.0, 0.0);
    for (int j = 0; j < n; ++j) {
      // gU[b][d] += uc Re sum_a conj(T[a][d]) gG[a][b]
      const double2 t = T[j * n + k], g = gG[j * n + r];
      sum = fma(t.x, g.x, fma(t.y, g.y, sum));
      // gS[a][c] = Re sum_d conj(C[c][d]) gW[a][d]
      const double2 c = C[k * n + j], w = gW[r * n + j];
      gs = fma(c.x, w.x, fma(c.y, w.y, gs));
      // gC[c][d] = sum_a U[a][c]^2 gW[a][d]
      const double u = U[j * n + r], u2 = u * u;
      gc.x = fma(u2, gW[j * n + k].x, gc.x);
      gc.y = fma(u2, gW[j * n + k].y, gc.y);
    }
    gU[e] += p.uc * sum + 2.0 * U[e] * gs;
    const double2 c0 = p.c0[s * nn + e], d0 = p.d0[s * nn + e];
    glam += c0.x * gc.x + c0.y * gc.y;
    tmp[e] = lam * (d0.x * gc.x + d0.y * gc.y);   // cotangent of E_d - E_c
  }
  for (int o = 16; o > 0; o >>= 1) glam += __shfl_xor_sync(0xffffffffu, glam, o);
  if (lane == 0) p.glam[s] = glam;
  __syncwarp();
  FIT_EACH(e) {   // eigenpairs: diag(gE) + F o (U^T gU), F_ij = 1 / (E_j - E_i)
    const int i = e / n, j = e % n;
    double v = 0.0;
    if (i == j) {
      for (int c = 0; c < n; ++c) v += tmp[c * n + i] - tmp[i * n + c];
    } else {
      const double gap = E[j] - E[i];
      for (int a = 0; a < n; ++a) v = fma(U[a * n + i], gU[a * n + j], v);
      v = gap != 0.0 ? v / gap : 0.0;
    }
    in[e] = v;
  }
  __syncwarp();
  FIT_EACH(e) {   // tmp = in U^T
    const int i = e / n, b = e % n;
    double v = 0.0;
    for (int j = 0; j < n; ++j) v = fma(in[i * n + j], U[b * n + j], v);
    tmp[e] = v;
  }
  __syncwarp();
  FIT_EACH(e) {
    const int a = e / n, b = e % n;
    double v = 0.0, w = 0.0;
    for (int i = 0; i < n; ++i) {
      v = fma(U[a * n + i], tmp[i * n + b], v);
      w = fma(U[b * n + i], tmp[i * n + a], w);
    }
    p.gH[s * nn + e] = fma(p.uc, gG[e].y, 0.5 * (v + w));
  }
}

// ----------------------------------------------------------------- RK4 step
// D = P - I = A + A^2/2 + A^2 (A/6 + A^2/24), A = h L, and its transpose map.
__device__ __forceinline__ void step_product(int nn, int n, int lane, const double2* X,
                                             const double2* Y, double2* Z) {
  FIT_EACH(e) {
    double2 z = cmk(0.0, 0.0);
    for (int k = 0; k < n; ++k) cfma(z, X[e / n * n + k], Y[k * n + e % n]);
    Z[e] = z;
  }
  __syncwarp();
}

__global__ void __launch_bounds__(32 * FW)
    step_forward_kernel(const double2* __restrict__ L, int n, int64_t batch, double h,
                        double2* __restrict__ D) {
  extern __shared__ __align__(16) double2 sm[];
  const int lane = threadIdx.x & 31, nn = n * n;
  const int64_t s = (int64_t)blockIdx.x * FW + (threadIdx.x >> 5);
  if (s >= batch) return;   // whole warps: no CTA barrier below
  double2* A = sm + (size_t)(threadIdx.x >> 5) * 4 * nn;
  double2 *A2 = A + nn, *B = A2 + nn, *Z = B + nn;
  FIT_EACH(e) A[e] = cscale(L[s * nn + e], h);
  __syncwarp();
  step_product(nn, n, lane, A, A, A2);
  FIT_EACH(e) B[e] = cadd(cscale(A[e], 1.0 / 6.0), cscale(A2[e], 1.0 / 24.0));
  __syncwarp();
  step_product(nn, n, lane, A2, B, Z);
  FIT_EACH(e) D[s * nn + e] = cadd(cadd(A[e], cscale(A2[e], 0.5)), Z[e]);
}

// X Y^H and X^H Y, element e
__device__ __forceinline__ double2 step_xyh(int n, int e, const double2* X, const double2* Y) {
  double2 z = cmk(0.0, 0.0);
  for (int k = 0; k < n; ++k) cfma(z, X[e / n * n + k], cconj(Y[e % n * n + k]));
  return z;
}
__device__ __forceinline__ double2 step_xhy(int n, int e, const double2* X, const double2* Y) {
  double2 z = cmk(0.0, 0.0);
  for (int k = 0; k < n; ++k) cfma(z, cconj(X[k * n + e / n]), Y[k * n + e % n]);
  return z;
}

__global__ void __launch_bounds__(32 * FW)
    step_backward_kernel(const double2* __restrict__ L, const double2* __restrict__ gD, int n,
                         int64_t batch, double h, double2* __restrict__ gL) {
  extern __shared__ __align__(16) double2 sm[];
  const int lane = threadIdx.x & 31, nn = n * n;
  const int64_t s = (int64_t)blockIdx.x * FW + (threadIdx.x >> 5);
  if (s >= batch) return;   // whole warps: no CTA barrier below
  double2* A = sm + (size_t)(threadIdx.x >> 5) * 6 * nn;
  double2 *A2 = A + nn, *B = A2 + nn, *g = B + nn, *gB = g + nn, *gA2 = gB + nn;
  FIT_EACH(e) {
    A[e] = cscale(L[s * nn + e], h);
    g[e] = gD[s * nn + e];
  }
  __syncwarp();
  step_product(nn, n, lane, A, A, A2);
  FIT_EACH(e) {
    B[e] = cadd(cscale(A[e], 1.0 / 6.0), cscale(A2[e], 1.0 / 24.0));
    gB[e] = step_xhy(n, e, A2, g);
  }
  __syncwarp();
  FIT_EACH(e)
    gA2[e] = cadd(cadd(cscale(g[e], 0.5), cscale(gB[e], 1.0 / 24.0)), step_xyh(n, e, g, B));
  __syncwarp();
  FIT_EACH(e) {
    double2 v = cadd(g[e], cscale(gB[e], 1.0 / 6.0));
    v = cadd(v, cadd(step_xyh(n, e, gA2, A), step_xhy(n, e, A, gA2)));
    gL[s * nn + e] = cscale(v, h);
  }
}

#undef FIT_EACH

MatsubaraSums make_sums(double T, double gamma, int K) {
  // the partial zeta sums depend on K alone and take 30k operations
  static thread_local int last_K = -1;
  static thread_local double last_z[2 * SUM_SERIES + 4];
  MatsubaraSums p = {};
  if (last_K != K) {
    for (double& z : last_z) z = 0.0;
    for (int k = K - 1; k >= SUM_DIRECT; --k) {   // small terms first
      const double inv = 1.0 / k;
      double t = inv;
      for (int s = 2; s < 2 * SUM_SERIES + 4; ++s) last_z[s] += t *= inv;
    }
    last_K = K;
  }
  for (int s = 0; s < 2 * SUM_SERIES + 4; ++s) p.z[s] = last_z[s];
  p.c = 2.0 * M_PI * T;
  const double a = gamma / p.c;
  p.a2 = a * a;
  p.series = p.a2 <= SUM_MAX;
  for (int k = 1; k < SUM_DIRECT; ++k) p.w[k] = matsubara_weight(p.c, gamma, k);
  p.gamma = gamma;
  p.cot = 1.0 / tan(gamma / (2.0 * T));
  p.four_t = 4.0 * T;
  p.freq_t = 2.0 * T / gamma;
  p.K = K;
  return p;
}

template <typename F>
int fit_launch(F fn, size_t per_warp, cudaError_t* e) {
  *e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(FW * per_warp));
  return *e == cudaSuccess;
}

}  // namespace

}  // namespace qsx

using namespace qsx;

#define FIT_CHECK(name)                                                                       \
  QSX_CHECK_ARG(n >= 1 && n <= FIT_NMAX && batch >= 0 && batch <= 0x7fffffffLL,               \
                name ": need 1 <= n <= %d (got %d) and a batch", FIT_NMAX, n);                \
  if (batch == 0) return QSX_OK;                                                              \
  const size_t nn = (size_t)n * n;                                                            \
  const unsigned grid = (unsigned)((batch + FW - 1) / FW);                                    \
  cudaStream_t s = (cudaStream_t)stream;                                                      \
  cudaError_t e

extern "C" int qsx_debye_unit(const double* x, int64_t count, double temperature,
                              double cutoff_freq, int matsubara_cutoff, double* value,
                              double* derivative, void* stream) {
  QSX_CHECK_ARG(count >= 0 && (count == 0 || (x && value && derivative)) && matsubara_cutoff >= 1,
                "qsx_debye_unit: bad arguments");
  if (count == 0) return QSX_OK;
  unit_corr_kernel<<<(unsigned)((count + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      x, count, make_sums(temperature, cutoff_freq, matsubara_cutoff), (double2*)value,
      (double2*)derivative);
  QSX_LAUNCH_CHECK("qsx_debye_unit");
  return QSX_OK;
}

extern "C" int qsx_eg_generator(const double* H, const double* E, const double* U, int n,
                                int64_t batch, const double* lam, double temperature,
                                double cutoff_freq, int matsubara_cutoff, double unit_convert,
                                double* L, double* c0, double* d0, void* stream) {
  FIT_CHECK("qsx_eg_generator");
  QSX_CHECK_ARG(H && E && U && lam && L && c0 && d0 && matsubara_cutoff >= 1,
                "qsx_eg_generator: bad arguments");
  GenP p = {H, E, U, lam, (double2*)L, (double2*)c0, (double2*)d0, nullptr, nullptr, nullptr, n,
            batch, unit_convert};
  const size_t per = 3 * nn * sizeof(double2);
  if (fit_launch(gen_forward_kernel, per, &e))
    gen_forward_kernel<<<grid, 32 * FW, FW * per, s>>>(
        p, make_sums(temperature, cutoff_freq, matsubara_cutoff));
  if (e != cudaSuccess) return cuda_status(e, "qsx_eg_generator");
  QSX_LAUNCH_CHECK("qsx_eg_generator");
  return QSX_OK;
}

extern "C" int qsx_eg_generator_adjoint(const double* E, const double* U, int n, int64_t batch,
                                        const double* lam, double unit_convert, const double* c0,
                                        const double* d0, const double* gL, double* gH,
                                        double* glam, void* stream) {
  FIT_CHECK("qsx_eg_generator_adjoint");
  QSX_CHECK_ARG(E && U && lam && c0 && d0 && gL && gH && glam,
                "qsx_eg_generator_adjoint: null pointer");
  GenP p = {nullptr, E, U, lam, nullptr, (double2*)c0, (double2*)d0, (const double2*)gL, gH, glam,
            n, batch, unit_convert};
  const size_t per = 8 * nn * sizeof(double2);
  if (fit_launch(gen_backward_kernel, per, &e))
    gen_backward_kernel<<<grid, 32 * FW, FW * per, s>>>(p);
  if (e != cudaSuccess) return cuda_status(e, "qsx_eg_generator_adjoint");
  QSX_LAUNCH_CHECK("qsx_eg_generator_adjoint");
  return QSX_OK;
}

extern "C" int qsx_rk4_step(const double* L, int n, int64_t batch, double h, double* D,
                            void* stream) {
  FIT_CHECK("qsx_rk4_step");
  QSX_CHECK_ARG(L && D, "qsx_rk4_step: null pointer");
  const size_t per = 4 * nn * sizeof(double2);
  if (fit_launch(step_forward_kernel, per, &e))
    step_forward_kernel<<<grid, 32 * FW, FW * per, s>>>((const double2*)L, n, batch, h,
                                                        (double2*)D);
  if (e != cudaSuccess) return cuda_status(e, "qsx_rk4_step");
  QSX_LAUNCH_CHECK("qsx_rk4_step");
  return QSX_OK;
}

extern "C" int qsx_rk4_step_adjoint(const double* L, const double* gD, int n, int64_t batch,
                                    double h, double* gL, void* stream) {
  FIT_CHECK("qsx_rk4_step_adjoint");
  QSX_CHECK_ARG(L && gD && gL, "qsx_rk4_step_adjoint: null pointer");
  const size_t per = 6 * nn * sizeof(double2);
  if (fit_launch(step_backward_kernel, per, &e))
    step_backward_kernel<<<grid, 32 * FW, FW * per, s>>>((const double2*)L, (const double2*)gD, n,
                                                         batch, h, (double2*)gL);
  if (e != cudaSuccess) return cuda_status(e, "qsx_rk4_step_adjoint");
  QSX_LAUNCH_CHECK("qsx_rk4_step_adjoint");
  return QSX_OK;
}
