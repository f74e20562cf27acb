// Ensemble mean of one projected trajectory of small blocks (m <= 16), in
// FP64 and in blocks of 32 steps, and its adjoint.
//
// x_n = scale sum_s c^T P_s^n y0_s (linear_response averaged over disorder,
// qspectra/simulate/response.py:15-43, decorators.py:40-64).  Split at
// n = 32 i + j the term of one sample is a product of a row and a state,
//   r_j . Y_i,   r_j = c^T P^j (j < 32),   Y_i = P^{32 i} y0,
// so only 32 + T/32 vectors are propagated (by doubling: r_{j+n} = r_j P^n,
// Y_{i+n} = P^{32 n} Y_i, with D_{2n} = 2 D_n + D_n D_n for P^n = I + D_n) and
// each x_n costs m multiply-adds in place of m^2 + m.
//
// Forward: a persistent CTA runs one sample after another.  Its doubling
// phases spread their outputs over all 256 threads, then warp w and lane j
// own the outputs (i = w, w + 8, ..; j): the row elements come from shared
// memory once per i-loop, the states are broadcasts, and the sums over the
// CTA's samples stay in registers, so nothing of [sample][step] is stored.
//
// Adjoint: the doubling run backwards.  With the cotangents
//   gY_i = sum_j conj(r_j) g_{32 i + j},  gr_j = sum_i conj(Y_i) g_{32 i + j},
// each phase gives back gY_j += P_n^H gY_{n+j}, gD_n += sum_j gY_{n+j} Y_j^H
// and each square gD_n += gD_{2n} P_n^H + P_n^H gD_{2n}: twice the forward's
// multiply-adds, all of a phase independent, against the stepped adjoint's
// 3 m^2 a step on one lane a row.
//
// Bound: FP64 issue (2 multiply-adds per clock and SM), of which the forward
// needs 83k a sample and the adjoint 190k at m = 7 and 2048 steps.
#include <algorithm>

#include "qsx_common.cuh"
#include "rk4_mean.cuh"

namespace qsx {

namespace {

constexpr int MT = 256;   // threads
constexpr int KB = 32;    // steps in a block: one lane each

// acc += conj(a) b
__device__ __forceinline__ void cfma_conj(double2& acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(-a.y, b.x, acc.y);
}

// One doubling phase over the CTA.  Rows x of length m, row stride ld;
// RIGHT: x_{n+j} = x_j + x_j D (rows), else x_{n+j} = x_j + D x_j (states);
// then next = 2 D + D D when `square`.  ld is odd, so that lanes on
// consecutive rows of D hit different banks.
template <bool RIGHT>
__device__ __forceinline__ bool mean_phase(double2* x, int n, int cnt, const double2* D,
                                           double2* next, bool square, int m, int ld) {
  bool bad = false;
  const int nr = cnt * m, total = nr + (square ? m * m : 0);
  for (int e = threadIdx.x; e < total; e += MT) {
    const bool row = e < nr;
    const int q = row ? e : e - nr, j = q / m, r = q % m;
    const double2* v = (row ? x : D) + j * ld;          // the row that is multiplied
    const bool right = RIGHT || !row;
    const double2* d = right ? D + r : D + r * ld;
    const int step = right ? ld : 1;
    double2 a0 = make_double2(0.0, 0.0), a1 = a0;
    int k = 0;
#pragma unroll 4
    for (; k + 1 < m; k += 2) {
      cfma(a0, v[k], d[k * step]);
      cfma(a1, v[k + 1], d[(k + 1) * step]);
    }
    if (k < m) cfma(a0, v[k], d[k * step]);
    double2 o = cadd(v[r], cadd(a0, a1));
    if (!row) o = cadd(v[r], o);
    (row ? x + (n + j) * ld : next + j * ld)[r] = o;
    bad |= !finite2(o);
  }
  __syncthreads();
  return bad;
}

struct MeanP {
  const void* D;
  int64_t d_stride, y0_stride, c_stride, batch;
  const double2 *y0, *c;
  int m, nsave, nblk;       // nblk = ceil(nsave / 32)
  double2* partial;         // [grid][nsave]
  int* flag;
};

template <typename C, int NI>
__global__ void __launch_bounds__(MT) mean_forward_kernel(MeanP p) {
  extern __shared__ __align__(16) double2 sm[];
  const int m = p.m, ld = m | 1;
  double2* D = sm;                      // [2][m][ld]
  double2* R = D + 2 * m * ld;          // [32][ld]
  double2* Y = R + KB * ld;             // [nblk + 1][ld]
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  double2 acc[NI];
#pragma unroll
  for (int k = 0; k < NI; ++k) acc[k] = make_double2(0.0, 0.0);
  bool bad = false;
  for (int64_t s = blockIdx.x; s < p.batch; s += gridDim.x) {
    const C* d = (const C*)p.D + s * p.d_stride;
    for (int e = threadIdx.x; e < m * m; e += MT)
      D[e / m * ld + e % m] = make_double2((double)d[e].x, (double)d[e].y);
    for (int e = threadIdx.x; e < m; e += MT) {
      R[e] = p.c[s * p.c_stride + e];
      Y[e] = p.y0[s * p.y0_stride + e];
      bad |= !finite2(R[e]) || !finite2(Y[e]);
    }
    __syncthreads();
    double2 *cur = D, *next = D + m * ld;
    auto swap = [&] { double2* t = cur; cur = next; next = t; };
    for (int n = 1; n < KB; n *= 2, swap())
      bad |= mean_phase<true>(R, n, n, cur, next, true, m, ld);
    // one state past the last block: growth up to the last step shows there
    for (int n = 1; n < p.nblk + 1; n *= 2, swap()) {
      const bool more = 2 * n < p.nblk + 1;
      bad |= mean_phase<false>(Y, n, min(n, p.nblk + 1 - n), cur, next, more, m, ld);
      if (sizeof(C) == sizeof(float2))   // the range of the FP32 stepped loop
        for (int e = threadIdx.x; e < min(n, p.nblk + 1 - n) * m; e += MT) {
          const double2 v = Y[(n + e / m) * ld + e % m];
          bad |= !isfinite((float)v.x) || !isfinite((float)v.y);
        }
    }
    for (int a = 0; a < m; ++a) {
      const double2 r = R[lane * ld + a];
#pragma unroll
      for (int k = 0; k < NI; ++k)
        if (w + 8 * k < p.nblk) cfma(acc[k], r, Y[(w + 8 * k) * ld + a]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k < NI; ++k) {
    const int n = (w + 8 * k) * KB + lane;
    if (n < p.nsave) {
      p.partial[(int64_t)blockIdx.x * p.nsave + n] = acc[k];
      bad |= !finite2(acc[k]);
    }
  }
  if (bad) atomicOr(p.flag, 1);
}

struct MeanAdjP {
  const double2 *D, *y0, *c, *g;
  int64_t y0_stride;
  int m, nsteps, nblk;
  double scale;
  double2* gradD;
  int* flag;
};

__global__ void __launch_bounds__(MT) mean_adjoint_kernel(MeanAdjP p) {
  extern __shared__ __align__(16) double2 sm[];
  const int m = p.m, ld = m | 1, mm = m * ld, nblk = p.nblk;
  const int tid = threadIdx.x;
  int py = 0;                              // state phases
  while ((1 << py) < nblk) ++py;
  const int np = 5 + max(py, 1);           // powers D_1, D_2, .., kept for the way back
  double2* D = sm;                         // [np][m][ld]
  double2* R = D + np * mm;                // [32][ld]
  double2* gR = R + KB * ld;
  double2* Y = gR + KB * ld;               // [nblk][ld]
  double2* gY = Y + nblk * ld;
  double2* gD = gY + nblk * ld;            // [2][m][ld]
  const int64_t s = blockIdx.x;
  bool bad = false;
  const double2* d = p.D + s * m * m;
  for (int e = tid; e < m * m; e += MT) D[e / m * ld + e % m] = d[e];
  for (int e = tid; e < m; e += MT) {
    R[e] = p.c[e];
    Y[e] = p.y0[s * p.y0_stride + e];
  }
  __syncthreads();
  for (int q = 0; q < 5; ++q)
    bad |= mean_phase<true>(R, 1 << q, 1 << q, D + q * mm, D + (q + 1) * mm, true, m, ld);
  for (int q = 0; q < py; ++q)
    bad |= mean_phase<false>(Y, 1 << q, min(1 << q, nblk - (1 << q)), D + (5 + q) * mm,
                             D + (6 + q) * mm, q + 1 < py, m, ld);
  // cotangents of the states and rows (g past the last step is zero)
  for (int e = tid; e < (nblk + KB) * m; e += MT) {
    const bool st = e < nblk * m;
    const int q = st ? e : e - nblk * m, i = q / m, a = q % m;
    const double2* v = (st ? R : Y) + a;
    const int n0 = st ? i * KB : i, dn = st ? 1 : KB;
    const int cnt = st ? min(KB, p.nsteps + 1 - n0)
                       : (n0 <= p.nsteps ? (p.nsteps - n0) / KB + 1 : 0);
    double2 a0 = make_double2(0.0, 0.0), a1 = a0;
    int k = 0;
#pragma unroll 4
    for (; k + 1 < cnt; k += 2) {
      cfma_conj(a0, v[k * ld], p.g[n0 + k * dn]);
      cfma_conj(a1, v[(k + 1) * ld], p.g[n0 + (k + 1) * dn]);
    }
    if (k < cnt) cfma_conj(a0, v[k * ld], p.g[n0 + k * dn]);
    (st ? gY : gR)[i * ld + a] = cadd(a0, a1);
  }
  __syncthreads();
  // back through the phases, the last power first; gh is the cotangent of the
  // power above (none above the last one used)
  double2 *gh = nullptr, *gd = gD;
  for (int q = 4 + py; q >= 0; --q) {
    const bool st = q >= 5;
    const int n = 1 << (st ? q - 5 : q), cnt = st ? min(n, nblk - n) : n;
    const double2* Dq = D + q * mm;
    double2* x = st ? Y : R;
    double2* gx = st ? gY : gR;
    const int nr = cnt * m;
    for (int e = tid; e < nr + m * m; e += MT) {
      if (e < nr) {   // gx_j += P^H gx_{n+j}, or its row form gx_{n+j} P^H
        const int j = e / m, k = e % m;
        const double2* up = gx + (n + j) * ld;
        const double2* col = st ? Dq + k : Dq + k * ld;
        const int step = st ? ld : 1;
        double2 a0 = up[k], a1 = make_double2(0.0, 0.0);
        int r = 0;
        for (; r + 1 < m; r += 2) {
          cfma_conj(a0, col[r * step], up[r]);
          cfma_conj(a1, col[(r + 1) * step], up[r + 1]);
        }
        if (r < m) cfma_conj(a0, col[r * step], up[r]);
        gx[j * ld + k] = cadd(gx[j * ld + k], cadd(a0, a1));
      } else {        // gD[r][k]: rows of this phase, then the square above
        const int f = e - nr, r = f / m, k = f % m;
        double2 a0 = make_double2(0.0, 0.0), a1 = a0;
        const double2* u = st ? gx + n * ld + r : gx + n * ld + k;
        const double2* v = st ? x + k : x + r;
        int j = 0;
        for (; j + 1 < cnt; j += 2) {
          cfma_conj(a0, v[j * ld], u[j * ld]);
          cfma_conj(a1, v[(j + 1) * ld], u[(j + 1) * ld]);
        }
        if (j < cnt) cfma_conj(a0, v[j * ld], u[j * ld]);
        if (gh) {
          a0 = cadd(a0, cscale(gh[r * ld + k], 2.0));
          for (int l = 0; l < m; ++l) {
            cfma_conj(a0, Dq[k * ld + l], gh[r * ld + l]);
            cfma_conj(a1, Dq[l * ld + r], gh[l * ld + k]);
          }
        }
        gd[r * ld + k] = cadd(a0, a1);
      }
    }
    __syncthreads();
    gh = gd;
    gd = gd == gD ? gD + mm : gD;
  }
  double2* out = p.gradD + s * m * m;
  for (int e = tid; e < m * m; e += MT) {
    const double2 v = cscale(gh[e / m * ld + e % m], p.scale);
    bad |= !finite2(v);
    out[e] = v;
  }
  if (bad) atomicOr(p.flag, 1);
}

int adjoint_nblk(int nsteps) { return nsteps / KB + 1; }

size_t adjoint_smem(int m, int nsteps) {
  const int nblk = adjoint_nblk(nsteps), ld = m | 1;
  int py = 0;
  while ((1 << py) < nblk) ++py;
  const size_t np = 5 + std::max(py, 1);
  return ((np + 2) * m * ld + 2 * (size_t)(KB + nblk) * ld) * sizeof(double2);
}

}  // namespace

// Blocks pay from a few of them on: below 64 outputs the stepped loop is as
// short as the doubling's phases.  16 rows and 4096 outputs keep the states
// and the register sums of a CTA in place.
bool rk4_mean_supported(int m, int64_t nsave) { return m <= 16 && nsave >= 64 && nsave <= 4096; }

int rk4_mean_grid(int64_t batch, int* grid) {
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return cuda_status(e, "qsx_rk4 mean plan");
  // two CTAs an SM: one's phases (barriers) beside the other's contraction
  *grid = (int)std::max<int64_t>(1, std::min<int64_t>(batch, 2 * (int64_t)sms));
  return QSX_OK;
}

int rk4_mean_run(const qsx_rk4_args* a, int grid, double2* partial, int* flag, cudaStream_t s) {
  const int64_t nsave = a->nsteps / a->save_every + 1;
  MeanP p;
  p.D = a->matrix;
  p.d_stride = a->matrix_stride;
  p.y0 = (const double2*)a->y0;
  p.y0_stride = a->y0_stride;
  p.c = (const double2*)a->proj;
  p.c_stride = a->proj_stride;
  p.batch = a->batch;
  p.m = a->m;
  p.nsave = (int)nsave;
  p.nblk = (int)((nsave + KB - 1) / KB);
  p.partial = partial;
  p.flag = flag;
  const int ld = a->m | 1;
  const size_t smem = (2 * (size_t)a->m * ld + (size_t)(KB + p.nblk + 1) * ld) * sizeof(double2);
  cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), s);
  auto launch = [&](void (*fn)(MeanP)) {
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) fn<<<(unsigned)grid, MT, smem, s>>>(p);
  };
  const bool f32 = a->precision == QSX_FP32;
  if (p.nblk <= 32)
    launch(f32 ? mean_forward_kernel<float2, 4> : mean_forward_kernel<double2, 4>);
  else if (p.nblk <= 64)
    launch(f32 ? mean_forward_kernel<float2, 8> : mean_forward_kernel<double2, 8>);
  else
    launch(f32 ? mean_forward_kernel<float2, 16> : mean_forward_kernel<double2, 16>);
  if (e != cudaSuccess) return cuda_status(e, "qsx_rk4_batched mean");
  QSX_LAUNCH_CHECK("qsx_rk4_batched mean");
  return QSX_OK;
}

bool rk4_mean_adjoint_supported(int m, int nsteps) {
  return nsteps >= 1 && rk4_mean_supported(m, (int64_t)nsteps + 1) &&
         adjoint_smem(m, nsteps) <= 200 * 1024;
}

int rk4_mean_adjoint_run(const double2* D, int m, int64_t batch, int nsteps, const double2* y0,
                         int64_t y0_stride, const double2* c, const double2* g, double scale,
                         double2* gradD, int* flag, cudaStream_t s) {
  MeanAdjP p = {D, y0, c, g, y0_stride, m, nsteps, adjoint_nblk(nsteps), scale, gradD, flag};
  const size_t smem = adjoint_smem(m, nsteps);
  cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), s);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(mean_adjoint_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem);
  if (e != cudaSuccess) return cuda_status(e, "qsx_rk4_mean_adjoint");
  mean_adjoint_kernel<<<(unsigned)batch, MT, smem, s>>>(p);
  QSX_LAUNCH_CHECK("qsx_rk4_mean_adjoint");
  return QSX_OK;
}

}  // namespace qsx
