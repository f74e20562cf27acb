// Batched FP64 symmetric eigensolver for matrices too large for the
// register Jacobi kernels (the two-exciton block: 276 states at 24 sites).
// The reference diagonalises each sample's Hamiltonian with scipy.linalg.eigh
// (qspectra/hamiltonian.py:310-328).
//
// Four kernels over a global-memory workspace:
//   1. Householder reduction to tridiagonal form, A = Q T Q^T: for each
//      column k, v with (I - tau v v^T) x = alpha e_1 and the two-sided
//      update B <- B - v w^T - w v^T, w = p - (tau/2)(v^T p) v, p = tau B v.
//      A cluster of CTAs per matrix, each with every c-th column in shared
//      memory; v and p cross through distributed shared memory.  (One CTA per
//      matrix on a copy in global memory where a cluster cannot hold it.)
//   2. Eigenvalues of T by bisection on Sturm counts (one thread per
//      eigenvalue of every matrix; O(n) per count, about 50 counts), the
//      counts from the scaled polynomial recurrence: three FP64 instructions
//      a step where the pivot recurrence's reciprocal alone takes a dozen.
//   3. Eigenvectors of T by inverse iteration (one thread per eigenvalue of
//      every matrix): LU with partial pivoting of
//      T - lambda I, three solves from a vector of ones; eigenvalues closer
//      than 1e-5 |T| form a cluster handled by one thread with modified
//      Gram-Schmidt against the cluster's earlier vectors, wider ones are
//      orthogonalised in a pass of their own.  The threads' scratch vectors
//      are interleaved, so a warp's accesses are one line.
//   4. Back-transform by the Householder reflectors, U = H_0 ... H_{n-3} Z:
//      columns are independent, so a tile of them per CTA, in shared memory.
// 32 matrices of 276 states: tridiagonal form 8.9 ms and back-transform 9.7 ms
// with one CTA per matrix (32 of 152 SMs), now 2.8 and 1.8; bisection 6.6 ms
// with the pivot recurrence one point at a time, now 1.9; inverse iteration
// 6.3 ms with a scratch of its own per thread, now 1.1.
// This keeps the FP64 work near 2 n^3 multiply-adds per matrix (no Givens
// rotations accumulated into Q).  Eigenvalues are returned ascending with
// U[:, k] the k-th eigenvector.  Every loop is bounded (bisection stops after
// 128 halvings, inverse iteration runs three solves).
#include <algorithm>
#include <cfloat>

#include "qsx_common.cuh"

namespace qsx {

__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  __syncthreads();
  if (lane == 0) red[warp] = v;
  __syncthreads();
  double t = 0.0;
  const int nw = blockDim.x >> 5;
  for (int i = 0; i < nw; ++i) t += red[i];
  return t;
}

// sum_j x[j * ld] v[j]: four independent chains, eight loads in flight
__device__ __forceinline__ double col_dot(const double* __restrict__ x, int ld,
                                          const double* __restrict__ v, int m) {
  double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
  int j = 0;
  for (; j + 7 < m; j += 8) {
    double t[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) t[q] = x[(int64_t)(j + q) * ld];
    a0 = fma(t[0], v[j], a0);
    a1 = fma(t[1], v[j + 1], a1);
    a2 = fma(t[2], v[j + 2], a2);
    a3 = fma(t[3], v[j + 3], a3);
    a0 = fma(t[4], v[j + 4], a0);
    a1 = fma(t[5], v[j + 5], a1);
    a2 = fma(t[6], v[j + 6], a2);
    a3 = fma(t[7], v[j + 7], a3);
  }
  for (; j < m; ++j) a0 = fma(x[(int64_t)j * ld], v[j], a0);
  return (a0 + a1) + (a2 + a3);
}

// x[i * ld] -= a[i] * bc + b[i] * ac for i < m, eight rows loaded before
// any is stored (the shared vectors a, b cannot alias x)
__device__ __forceinline__ void col_rank2(double* __restrict__ x, int ld,
                                          const double* __restrict__ a,
                                          const double* __restrict__ b, double bc, double ac,
                                          int m) {
  int i = 0;
  for (; i + 7 < m; i += 8) {
    double t[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) t[q] = x[(int64_t)(i + q) * ld];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      x[(int64_t)(i + q) * ld] = fma(-a[i + q], bc, fma(-b[i + q], ac, t[q]));
  }
  for (; i < m; ++i) x[(int64_t)i * ld] = fma(-a[i], bc, fma(-b[i], ac, x[(int64_t)i * ld]));
}

constexpr int TQ_THREADS = 320;

// The exponent of a matrix's largest element, which the reduction divides out:
// the square of no element that matters then leaves the range.  0 for a matrix
// of zeros and for one that is not finite (the eigenvalues report that).
__device__ __forceinline__ int scale_of(double top) {
  return top > 0.0 && isfinite(top) ? ilogb(top) : 0;
}
__device__ __forceinline__ double larger(double top, double v) {
  return isfinite(v) ? fmax(top, fabs(v)) : INFINITY;
}

// The reflector of a column (x0, rest), rest the sum of the squares below x0:
// summed by itself, since |x|^2 - x0^2 loses what lies 1e-8 below x0.
struct Reflector {
  double alpha, v0, tau;   // tau = 0: the column is done as it is
};
__device__ __forceinline__ Reflector reflector(double x0, double rest) {
  if (rest == 0.0) return {x0, x0, 0.0};   // (NaN goes on and is reported)
  const double alpha = -copysign(sqrt(fma(x0, x0, rest)), x0), v0 = x0 - alpha;
  return {alpha, v0, 2.0 / fma(v0, v0, rest)};
}

// ---- A. Householder tridiagonalisation: one CTA per matrix.  Writes the
// diagonal and sub-diagonal of A / 2^ex to de[b] = {d[0..n), e[0..n)}, ex to
// expo[b], and keeps, in the work matrix W, each reflector v_k in row k right of
// the diagonal with tau_k on the diagonal.
__global__ void __launch_bounds__(TQ_THREADS, 2)
    eigh_tridiag_kernel(const double* __restrict__ A, int n, double* W, double* de,
                        double* expo) {
  extern __shared__ __align__(16) double sm[];
  double* v = sm;          // [n] Householder vector
  double* w = v + n;       // [n]
  double* red = w + n;     // [32]
  const int tid = threadIdx.x, bd = blockDim.x;
  const int64_t b = blockIdx.x;
  const int64_t nn = (int64_t)n * n;
  const double* a = A + b * nn;
  double* Wm = W + b * nn;
  double* d = de + b * 2 * (int64_t)n;
  double* e = d + n;
  double top = 0.0;
  for (int64_t i = tid; i < nn; i += bd) top = larger(top, a[i]);
  for (int o = 16; o; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
  if ((tid & 31) == 0) red[tid >> 5] = top;
  __syncthreads();
  for (int i = 0; i < bd >> 5; ++i) top = fmax(top, red[i]);
  const int ex = scale_of(top);
  if (tid == 0) expo[b] = (double)ex;
  for (int64_t i = tid; i < nn; i += bd) Wm[i] = scalbn(a[i], -ex);
  __syncthreads();
  for (int k = 0; k < n - 2; ++k) {
    const int m = n - k - 1;
    const double* rowk = Wm + (int64_t)k * n + k + 1;
    double part = 0.0;
    for (int i = tid; i < m; i += bd) {
      const double x = rowk[i];
      v[i] = x;
      if (i) part += x * x;
    }
    const double rest = block_sum(part, red);
    const Reflector f = reflector(v[0], rest);
    const double tau = f.tau;
    if (tid == 0) {
      d[k] = Wm[(int64_t)k * n + k];
      e[k] = f.alpha;
    }
    if (tau != 0.0) {
      __syncthreads();
      if (tid == 0) v[0] = f.v0;
      __syncthreads();
      double* B = Wm + (int64_t)(k + 1) * n + k + 1;
      // p = tau B v (B symmetric: column r read across threads)
      double vp = 0.0;
      for (int r = tid; r < m; r += bd) {
        const double wr = tau * col_dot(B + r, n, v, m);
        w[r] = wr;
        vp += v[r] * wr;
      }
      const double K = 0.5 * tau * block_sum(vp, red);
      for (int r = tid; r < m; r += bd) w[r] -= K * v[r];
      __syncthreads();
      for (int c = tid; c < m; c += bd) col_rank2(B + c, n, v, w, w[c], v[c], m);
    }
    __syncthreads();
    for (int i = tid; i < m; i += bd) Wm[(int64_t)k * n + k + 1 + i] = tau != 0.0 ? v[i] : 0.0;
    if (tid == 0) Wm[(int64_t)k * n + k] = tau;
    __syncthreads();
  }
  if (tid == 0) {
    if (n >= 2) {
      d[n - 2] = Wm[(int64_t)(n - 2) * n + n - 2];
      e[n - 2] = Wm[(int64_t)(n - 1) * n + n - 2];
    }
    d[n - 1] = Wm[(int64_t)(n - 1) * n + n - 1];
    e[n - 1] = 0.0;
    if (n >= 2) Wm[(int64_t)(n - 2) * n + n - 2] = 0.0;  // no reflector for k = n-2
  }
}

// ---- A'. the same reduction by a cluster per matrix.  CTA `rank` of c keeps
// the columns rank, rank + c, .. in shared memory (cyclic, so that the
// trailing matrix stays spread out as it shrinks).  Step k: the owner of
// column k forms v and writes it to every CTA; each forms p = tau B v for its
// columns and writes that to every CTA; each then updates its columns.  Two cluster barriers a step.  A column is shared by
// `parts` neighbouring lanes, more of them as the active columns get fewer.
constexpr int TC_THREADS = 512;
constexpr int TC_MAX_CLUSTER = 8;

__host__ __device__ constexpr int tri_ld(int n) { return (n + 11) / 16 * 16 + 4; }  // 4 mod 16

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;"
               ::: "memory");
}
// store to the same shared-memory place of CTA `rank`
__device__ __forceinline__ void store_remote(double* p, unsigned rank, double v) {
  unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(r), "d"(v) : "memory");
}

// sum over i = i0, i0 + 32, .. < n of a warp's lanes (i0 = first + lane)
__device__ __forceinline__ double warp_dot(const double* x, const double* y, int i0, int n) {
  double a0 = 0.0, a1 = 0.0;
  int i = i0;
  for (; i + 32 < n; i += 64) {
    a0 = fma(x[i], y[i], a0);
    a1 = fma(x[i + 32], y[i + 32], a1);
  }
  if (i < n) a0 = fma(x[i], y[i], a0);
  double s = a0 + a1;
  for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

__global__ void __launch_bounds__(TC_THREADS)
    eigh_tridiag_cluster_kernel(const double* __restrict__ A, int n, int c, double* W, double* de,
                                double* expo) {
  extern __shared__ __align__(16) double sm[];
  const int ld = tri_ld(n), cols = (n + c - 1) / c;
  double* B = sm;                        // [cols][ld], column lc is matrix column lc c + rank
  // v and tau of step k at parity k & 1: the next owner may write its own
  // while a slower CTA still updates with these
  double* vbuf = B + (size_t)cols * ld;  // [2][n] row i of the matrix at v[i]
  double* w = vbuf + 2 * n;              // [n] p
  double* head = w + n;                  // [2]
  double* sv = head + 2;                 // [3] v_0, tau and K of this step
  __shared__ double tops[TC_THREADS / 32], ctop[TC_MAX_CLUSTER];
  const int tid = threadIdx.x;
  const int rank = (int)cluster_rank();
  const int64_t b = blockIdx.x / c, nn = (int64_t)n * n;
  const double* a = A + b * nn;
  double* Wm = W + b * nn;
  double* d = de + b * 2 * (int64_t)n;
  double* e = d + n;
  double top = 0.0;
  for (int64_t i = tid; i < (int64_t)cols * n; i += TC_THREADS) {
    // symmetric: row j of A is column j, read along the row
    const int lc = (int)(i / n), r = (int)(i % n), j = lc * c + rank;
    if (j >= n) continue;
    const double v = a[(int64_t)j * n + r];
    B[(size_t)lc * ld + r] = v;
    top = larger(top, v);
  }
  for (int o = 16; o; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
  if ((tid & 31) == 0) tops[tid >> 5] = top;
  __syncthreads();
  cluster_barrier();   // every CTA of the cluster runs before remote stores
  if (tid < c) {
    for (int i = 0; i < TC_THREADS / 32; ++i) top = fmax(top, tops[i]);
    store_remote(ctop + rank, tid, top);
  }
  cluster_barrier();
  top = ctop[0];
  for (int i = 1; i < c; ++i) top = fmax(top, ctop[i]);
  const int ex = scale_of(top);
  if (rank == 0 && tid == 0) expo[b] = (double)ex;
  for (int64_t i = tid; i < (int64_t)cols * n; i += TC_THREADS) {
    const int lc = (int)(i / n), r = (int)(i % n);
    if (lc * c + rank < n) B[(size_t)lc * ld + r] = scalbn(B[(size_t)lc * ld + r], -ex);
  }
  __syncthreads();
  for (int k = 0; k < n - 2; ++k) {
    double* v = vbuf + (k & 1) * n;
    if (rank == k % c) {
      // one warp: more of them would only queue for the FP64 pipe
      const double* x = B + (size_t)(k / c) * ld;
      if (tid < 32) {
        const Reflector f = reflector(x[k + 1], warp_dot(x, x, k + 2 + tid, n));
        if (tid < c) store_remote(head + (k & 1), tid, f.tau);
        if (tid == 0) {
          sv[0] = f.v0;
          sv[1] = f.tau;
          d[k] = x[k];
          e[k] = f.alpha;
          Wm[(int64_t)k * n + k] = f.tau;
        }
      }
      __syncthreads();
      for (int i = tid; i < (n - k - 1) * c; i += TC_THREADS) {
        const int r = k + 1 + i / c;
        const double vi = sv[1] == 0.0 ? 0.0 : r == k + 1 ? sv[0] : x[r];
        store_remote(v + r, i % c, vi);
        if (i % c == 0) Wm[(int64_t)k * n + r] = vi;
      }
    }
    cluster_barrier();
    const double tau = head[k & 1];
    if (tau != 0.0) {   // the same in every CTA
      const int lc0 = k >= rank ? (k - rank) / c + 1 : 0;      // first column past k
      const int nact = max(0, (n - rank + c - 1) / c - lc0);
      int parts = 4;
      while (parts < 32 && 2 * parts * nact <= TC_THREADS) parts *= 2;
      const int pt = tid % parts;
      for (int q0 = 0; q0 < nact; q0 += TC_THREADS / parts) {
        const int q = q0 + tid / parts, lc = lc0 + q;
        double a0 = 0.0, a1 = 0.0;
        if (q < nact) {
          const double* x = B + (size_t)lc * ld;
          int i = k + 1 + pt;
          for (; i + parts < n; i += 2 * parts) {
            a0 = fma(x[i], v[i], a0);
            a1 = fma(x[i + parts], v[i + parts], a1);
          }
          if (i < n) a0 = fma(x[i], v[i], a0);
        }
        double s = a0 + a1;
        for (int o = parts / 2; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (q < nact) {
          const int j = lc * c + rank;
          const double wr = tau * s;
          for (int t = pt; t < c; t += parts) store_remote(w + j, t, wr);
        }
      }
      cluster_barrier();
      if (tid < 32) {
        const double vp = warp_dot(v, w, k + 1 + tid, n);
        if (tid == 0) sv[2] = 0.5 * tau * vp;
      }
      __syncthreads();
      const double K = sv[2];
      for (int q = tid / parts; q < nact; q += TC_THREADS / parts) {
        const int lc = lc0 + q, j = lc * c + rank;
        double* x = B + (size_t)lc * ld;
        const double vj = v[j], wj = w[j] - K * vj;
        // w_i = p_i - K v_i folded: x -= v_i (w_j - K v_j) + p_i v_j
        const double vc = wj - K * vj;
        for (int i = k + 1 + pt; i < n; i += parts) x[i] = fma(-v[i], vc, fma(-w[i], vj, x[i]));
      }
      __syncthreads();
    }
  }
  // the last two columns
  for (int j = max(0, n - 2); j < n; ++j)
    if (rank == j % c && tid == 0) {
      const double* x = B + (size_t)(j / c) * ld;
      d[j] = x[j];
      if (j == n - 2) {
        e[j] = x[n - 1];
        Wm[(int64_t)j * n + j] = 0.0;  // no reflector for k = n-2
      } else {
        e[j] = 0.0;
      }
    }
  cluster_barrier();   // no CTA leaves while others may still write to it
}

// ---- B. eigenvalues by bisection on Sturm counts, one thread per
// eigenvalue of every matrix (FP64 instructions of a serial recurrence are
// slow on this part; these threads fill whole warps).  Eigenvalue j is the
// point where the count of eigenvalues below x steps from j to j + 1: the
// sign changes of p_i = (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2} (leading minors).
// Three points at a time quarter the interval, FP32 first.  A step's rounding is
// a perturbation of d_i - x and e^2 by a few ulp, so a count is exact for a
// matrix within eps |T|, like the pivot recurrence's.  Every four steps both
// p are rescaled through their exponent fields.  Results land sorted in ws.

// Per matrix, one warp: Gershgorin interval and |T|, and T scaled by a power of
// two to |T| about 1 (so that the minors grow by a known factor a step):
// diagonal in tri[b][0..n), squared sub-diagonal in tri[b][n..2n), the same in
// FP32 in trif, and in lim[b] the interval, the smallest pivot and the scale.
// Squared sub-diagonals get a floor far below their rounding: a minor that is
// exactly zero then always has a successor of the sign opposite to its
// predecessor's, and its own sign does not matter to the count.
__global__ void __launch_bounds__(128)
    eigh_scale_kernel(const double* __restrict__ de, int n, int64_t batch, double* tri,
                      float* trif, double* lim) {
  const int64_t b = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (b >= batch) return;
  const int lane = threadIdx.x & 31;
  const double* d = de + b * 2 * (int64_t)n;
  const double* e = d + n;
  double lo = d[0], hi = d[0], tnorm = 0.0;
  bool bad = false;
  for (int i = lane; i < n; i += 32) {
    const double r = (i ? fabs(e[i - 1]) : 0.0) + fabs(e[i]);
    lo = fmin(lo, d[i] - r);
    hi = fmax(hi, d[i] + r);
    tnorm = fmax(tnorm, fabs(d[i]) + r);
    bad |= !isfinite(d[i]) || !isfinite(e[i]);
  }
  for (int o = 16; o; o >>= 1) {
    lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
    hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    tnorm = fmax(tnorm, __shfl_xor_sync(0xffffffffu, tnorm, o));
  }
  if (__any_sync(0xffffffffu, bad)) tnorm = nan("");   // (fmax drops a NaN)
  int ex = 0;
  if (tnorm > 0.0 && isfinite(tnorm)) ex = max(-1000, min(1000, ilogb(tnorm)));
  for (int i = lane; i < n; i += 32) {
    const double f = scalbn(e[i], -ex), di = scalbn(d[i], -ex), ff = fmax(f * f, 1e-60);
    tri[b * 2 * n + i] = di;
    tri[b * 2 * n + n + i] = ff;
    trif[b * 2 * n + i] = (float)di;
    trif[b * 2 * n + n + i] = fmaxf((float)ff, 1e-20f);
  }
  if (lane == 0) {
    const double pivmin = DBL_EPSILON * fmax(scalbn(tnorm, -ex), DBL_MIN);
    lim[4 * b] = scalbn(lo, -ex) - 2.0 * pivmin;
    lim[4 * b + 1] = scalbn(hi, -ex) + 2.0 * pivmin;
    lim[4 * b + 2] = isnan(tnorm) ? tnorm : pivmin;
    lim[4 * b + 3] = (double)ex;
  }
}

// 2^k x by its exponent field; what falls below the normal range stays the
// smallest normal number of its sign
__device__ __forceinline__ double scale_exp(double x, int k) {
  const int hi = __double2hiint(x), ex = (hi >> 20) & 0x7ff;
  const bool low = ex == 0 || ex + k <= 0;
  return __hiloint2double(low ? (hi & 0x80000000) | 0x00100000 : hi + (k << 20),
                          low ? 0 : __double2loint(x));
}
__device__ __forceinline__ float scale_exp(float x, int k) {
  const int b = __float_as_int(x), ex = (b >> 23) & 0xff;
  return __int_as_float(ex == 0 || ex + k <= 0 ? (b & 0x80000000) | 0x00800000 : b + (k << 23));
}
__device__ __forceinline__ int exponent(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
__device__ __forceinline__ int exponent(float x) { return (__float_as_int(x) >> 23) & 0xff; }
__device__ __forceinline__ int high_word(double x) { return __double2hiint(x); }
__device__ __forceinline__ int high_word(float x) { return __float_as_int(x); }

// Eigenvalues of the scaled T below each of the PTS points x, the recurrences
// interleaved (one is a chain of dependent FP64 instructions): three FP64
// instructions a step and point, the sign changes by integer ones.
template <typename T, int PTS>
__device__ __forceinline__ void sturm_counts(const T* __restrict__ d, const T* __restrict__ e2,
                                             int n, const T (&x)[PTS], int (&cnt)[PTS]) {
  constexpr int BIAS = sizeof(T) == 8 ? 1023 : 127;
  T p0[PTS], p1[PTS];
  const T d0 = d[0];
#pragma unroll
  for (int q = 0; q < PTS; ++q) {
    p0[q] = (T)1;
    p1[q] = d0 - x[q];
    cnt[q] = (unsigned)high_word(p1[q]) >> 31;
  }
  auto step = [&](int i) {
    const T di = d[i], ee = e2[i - 1];
#pragma unroll
    for (int q = 0; q < PTS; ++q) {
      const T p2 = fma(di - x[q], p1[q], -ee * p0[q]);
      cnt[q] += (unsigned)(high_word(p2) ^ high_word(p1[q])) >> 31;
      p0[q] = p1[q];
      p1[q] = p2;
    }
  };
  int i = 1;
  for (; i + 3 < n; i += 4) {
#pragma unroll
    for (int u = 0; u < 4; ++u) step(i + u);
#pragma unroll
    for (int q = 0; q < PTS; ++q) {   // the larger of the two back to about 1
      const int k = BIAS - max(exponent(p0[q]), exponent(p1[q]));
      p0[q] = scale_exp(p0[q], k);
      p1[q] = scale_exp(p1[q], k);
    }
  }
  for (; i < n; ++i) step(i);
}

__global__ void eigh_bisect_kernel(const double* __restrict__ tri, const float* __restrict__ trif,
                                   const double* __restrict__ lim, int n, int64_t batch, double* ws, int* status) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= batch * n) return;
  const int64_t b = t / n;
  const int j = (int)(t % n);
  const double* d = tri + b * 2 * n;
  const double* e2 = d + n;
  double lo = lim[4 * b], hi = lim[4 * b + 1];
  const double pivmin = lim[4 * b + 2];
  // FP32 down to about 1e-6 of |T|; the interval is widened by that form's
  // rounding and kept only if FP64 counts at its ends agree
  {
    float flo = (float)lo, fhi = (float)hi;
    for (int it = 0; it < 10; ++it) {
      const float w = 0.25f * (fhi - flo);
      const float x[3] = {flo + w, flo + 2.0f * w, flo + 3.0f * w};
      int cnt[3];
      sturm_counts<float, 3>(trif + b * 2 * n, trif + b * 2 * n + n, n, x, cnt);
      const int below = (cnt[0] <= j) + (cnt[1] <= j) + (cnt[2] <= j);
      fhi = below < 3 ? x[below] : fhi;
      flo = below > 0 ? x[below - 1] : flo;
    }
    const double x[2] = {(double)flo - 2e-6, (double)fhi + 2e-6};
    int cnt[2];
    sturm_counts<double, 2>(d, e2, n, x, cnt);
    if (cnt[0] <= j && cnt[1] > j) {
      lo = fmax(lo, x[0]);
      hi = fmin(hi, x[1]);
    }
  }
  for (int it = 0; it < 64; ++it) {
    const double w = 0.25 * (hi - lo);
    const double x[3] = {lo + w, lo + 2.0 * w, lo + 3.0 * w};
    // (an interval that is not a number ends it too)
    if (!(hi - lo > 2.0 * DBL_EPSILON * fmax(fabs(lo), fabs(hi)) + pivmin) || x[1] <= lo ||
        x[1] >= hi)
      break;
    int cnt[3];
    sturm_counts<double, 3>(d, e2, n, x, cnt);
    const int below = (cnt[0] <= j) + (cnt[1] <= j) + (cnt[2] <= j);
    hi = below < 3 ? x[below] : hi;
    lo = below > 0 ? x[below - 1] : lo;
  }
  const double lam = scalbn(0.5 * (lo + hi), (int)lim[4 * b + 3]) + 0.0 * pivmin;
  if (!isfinite(lam) && status) atomicOr(status, QSX_ERR_NONFINITE);
  ws[b * n + j] = lam;
}

// ---- C. eigenvectors of T by inverse iteration, one thread per eigenvalue
// of every matrix; eigenvalues closer than 1e-5 |T| form a cluster handled
// by its first thread in order, with modified Gram-Schmidt against the
// cluster's earlier vectors.  Z[b] row-major, column j for eigenvalue j.
// Vectors further apart, up to 1e-3 |T|, overlap by less than eps / 1e-5 and
// are orthogonalised once afterwards (eigh_orthogonalise_kernel): solving
// them in turn made a warp wait for its longest run of close eigenvalues.
constexpr double CLUSTER_TIGHT = 1e-5, CLUSTER_WIDE = 1e-3;

__global__ void eigh_invit_kernel(const double* __restrict__ de, const double* __restrict__ ws,
                                  int n, int64_t batch, double* Z, double* scratch) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= batch * n) return;
  const int64_t b = t / n;
  const int j = (int)(t % n);
  const double* d = de + b * 2 * (int64_t)n;
  const double* e = d + n;
  const double* w = ws + b * (int64_t)n;
  double* z = Z + b * (int64_t)n * n;
  double tnorm = 0.0;
  for (int i = 0; i < n; ++i)
    tnorm = fmax(tnorm, fabs(d[i]) + fabs(e[i]) + (i ? fabs(e[i - 1]) : 0.0));
  const double ortol = fmax(CLUSTER_TIGHT * tnorm, 1e-100);
  // (a zero matrix, such as the two-exciton energy of a dimer in its mean
  // rotating frame, would leave a subnormal whose reciprocal overflows)
  const double tiny = fmax(DBL_EPSILON * tnorm, 1e-100);
  if (j > 0 && w[j] - w[j - 1] < ortol) return;  // not the first of its cluster
  int jend = j + 1;
  while (jend < n && w[jend] - w[jend - 1] < ortol) ++jend;
  // vector q of this thread at [q][i][lane]: a warp's accesses are one line
  struct Lane {
    double* p;
    __device__ double& operator[](int i) const { return p[(int64_t)i * 32]; }
  };
  double* sc = scratch + (t / 32) * 5 * (int64_t)n * 32 + t % 32;
  const Lane u1{sc}, u2{sc + 32 * (int64_t)n}, u3{sc + 64 * (int64_t)n},
      lm{sc + 96 * (int64_t)n}, x{sc + 128 * (int64_t)n};   // u1: reciprocal pivots
  for (int jj = j; jj < jend; ++jj) {
    // equal eigenvalues of a cluster are pulled apart slightly so that each
    // factorisation differs
    const double lam = w[jj] + (jj - j) * 10.0 * tiny;
    // LU with partial pivoting of T - lam I: u1, u2, u3 the three diagonals
    // of U, lm the multipliers (|l| <= 1; l + 4 where rows i, i+1 swapped)
    double pp = d[0] - lam, qq = n > 1 ? e[0] : 0.0;
    for (int i = 0; i < n - 1; ++i) {
      const double sub = e[i];
      const double an = d[i + 1] - lam, en = (i + 1 < n - 1) ? e[i + 1] : 0.0;
      if (fabs(pp) >= fabs(sub)) {
        if (fabs(pp) < tiny) pp = copysign(tiny, pp);
        const double inv = 1.0 / pp, l = sub * inv;
        u1[i] = inv;
        u2[i] = qq;
        u3[i] = 0.0;
        lm[i] = l;
        pp = an - l * qq;
        qq = en;
      } else {
        const double piv = fabs(sub) < tiny ? copysign(tiny, sub) : sub;
        const double inv = 1.0 / piv, l = pp * inv;
        u1[i] = inv;
        u2[i] = an;
        u3[i] = en;
        lm[i] = l + 4.0;
        const double np = qq - l * an;
        qq = -l * en;
        pp = np;
      }
    }
    u1[n - 1] = 1.0 / (fabs(pp) < tiny ? copysign(tiny, pp) : pp);
    // the first solve uses U only.  Later vectors of a cluster start from
    // scattered signs and sizes: T - lam I may be one and the same for them
    // (a matrix that is diagonal there), and a start shared with the vectors
    // they are orthogonalised against would leave nothing
    for (int i = 0; i < n; ++i) {
      const unsigned hash = ((unsigned)i * 2654435761u) ^ ((unsigned)jj * 2246822519u);
      x[i] = jj == j ? 1.0 : 1.0 - (double)((hash * 3266489917u) >> 8) * (2.0 / 16777216.0);
    }
    for (int it = 0; it < 3; ++it) {
      if (it > 0) {
        for (int i = 0; i < n - 1; ++i) {
          const double tt = lm[i];
          if (tt > 2.0) {
            const double l = tt - 4.0;
            const double xi = x[i];
            x[i] = x[i + 1];
            x[i + 1] = xi - l * x[i];
          } else {
            x[i + 1] -= tt * x[i];
          }
        }
      }
      for (int i = n - 1; i >= 0; --i) {
        double vv = x[i];
        if (i + 1 < n) vv -= u2[i] * x[i + 1];
        if (i + 2 < n) vv -= u3[i] * x[i + 2];
        x[i] = vv * u1[i];
      }
      for (int k = j; k < jj; ++k) {
        double dot = 0.0;
        for (int i = 0; i < n; ++i) dot = fma(z[(int64_t)i * n + k], x[i], dot);
        for (int i = 0; i < n; ++i) x[i] -= dot * z[(int64_t)i * n + k];
      }
      double nrm = 0.0;
      for (int i = 0; i < n; ++i) nrm = fma(x[i], x[i], nrm);
      const double inv = nrm > 0.0 ? rsqrt(nrm) : 0.0;
      for (int i = 0; i < n; ++i) x[i] *= inv;
    }
    for (int i = 0; i < n; ++i) z[(int64_t)i * n + jj] = x[i];
  }
}

// One warp per run of eigenvalues whose neighbours are closer than
// CLUSTER_WIDE |T|: modified Gram-Schmidt in order, lanes over the components.
__global__ void __launch_bounds__(128)
    eigh_orthogonalise_kernel(const double* __restrict__ de, const double* __restrict__ ws, int n,
                              int64_t batch, double* Z) {
  const int64_t t = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5);
  if (t >= batch * n) return;   // whole warps
  const int64_t b = t / n;
  const int j = (int)(t % n), lane = threadIdx.x & 31;
  const double* d = de + b * 2 * (int64_t)n;
  const double* e = d + n;
  const double* w = ws + b * (int64_t)n;
  double tnorm = 0.0;
  for (int i = lane; i < n; i += 32)
    tnorm = fmax(tnorm, fabs(d[i]) + fabs(e[i]) + (i ? fabs(e[i - 1]) : 0.0));
  for (int o = 16; o; o >>= 1) tnorm = fmax(tnorm, __shfl_xor_sync(0xffffffffu, tnorm, o));
  const double wide = CLUSTER_WIDE * tnorm;
  if (j > 0 && w[j] - w[j - 1] < wide) return;   // not the first of its run
  double* z = Z + b * (int64_t)n * n;
  for (int jj = j + 1; jj < n && w[jj] - w[jj - 1] < wide; ++jj) {
    for (int k = j; k < jj; ++k) {
      double dot = 0.0;
      for (int i = lane; i < n; i += 32)
        dot = fma(z[(int64_t)i * n + k], z[(int64_t)i * n + jj], dot);
      for (int o = 16; o; o >>= 1) dot += __shfl_xor_sync(0xffffffffu, dot, o);
      for (int i = lane; i < n; i += 32) z[(int64_t)i * n + jj] -= dot * z[(int64_t)i * n + k];
    }
    double nrm = 0.0;
    for (int i = lane; i < n; i += 32) nrm = fma(z[(int64_t)i * n + jj], z[(int64_t)i * n + jj], nrm);
    for (int o = 16; o; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
    const double inv = nrm > 0.0 ? rsqrt(nrm) : 0.0;
    for (int i = lane; i < n; i += 32) z[(int64_t)i * n + jj] *= inv;
  }
}

// ---- D. back-transform U = H_0 H_1 ... H_{n-3} Z (reflector k acts on rows
// k+1 ..), applied from k = n-3 down to 0; writes E and U.  Columns are
// independent: CTA blockIdx.x of a matrix keeps `cols` of them in shared
// memory, `parts` neighbouring lanes to a column.
constexpr int BT_THREADS = 512;

__global__ void __launch_bounds__(BT_THREADS)
    eigh_backtransform_kernel(const double* __restrict__ W, const double* __restrict__ ws,
                              const double* __restrict__ expo, int n, int cols, int parts,
                              const double* __restrict__ Z, double* __restrict__ E,
                              double* __restrict__ U) {
  extern __shared__ __align__(16) double sm[];
  const int ld = tri_ld(n);
  double* z = sm;                       // [cols][ld]
  double* v = z + (size_t)cols * ld;    // [2][n] reflector k at v[k & 1], its tau below
  double* tau = v + 2 * n;              // [2]
  const int tid = threadIdx.x;
  const int64_t b = blockIdx.y, nn = (int64_t)n * n;
  const int c0 = blockIdx.x * cols, nc = min(cols, n - c0);
  const double* Wm = W + b * nn;
  for (int64_t i = tid; i < (int64_t)n * nc; i += blockDim.x) {
    const int r = (int)(i / nc), q = (int)(i % nc);
    z[(size_t)q * ld + r] = Z[b * nn + (int64_t)r * n + c0 + q];
  }
  auto fetch = [&](int k) {
    for (int i = k + 1 + tid; i < n; i += blockDim.x) v[(k & 1) * n + i] = Wm[(int64_t)k * n + i];
    if (tid == 0) tau[k & 1] = Wm[(int64_t)k * n + k];
  };
  if (n >= 3) fetch(n - 3);
  __syncthreads();
  const int pt = tid % parts, q = tid / parts;
  double* x = z + (size_t)min(q, nc - 1) * ld;
  for (int k = n - 3; k >= 0; --k) {
    if (k > 0) fetch(k - 1);   // the other buffer
    const double t = tau[k & 1];
    const double* vk = v + (k & 1) * n;
    if (t != 0.0) {   // the same for all threads
      double a0 = 0.0, a1 = 0.0;
      int i = q < nc ? k + 1 + pt : n;
      for (; i + parts < n; i += 2 * parts) {
        a0 = fma(x[i], vk[i], a0);
        a1 = fma(x[i + parts], vk[i + parts], a1);
      }
      if (i < n) a0 = fma(x[i], vk[i], a0);
      double s = a0 + a1;
      for (int o = parts / 2; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      s *= t;
      if (q < nc)
        for (i = k + 1 + pt; i < n; i += parts) x[i] = fma(-s, vk[i], x[i]);
      __syncwarp();
    }
    __syncthreads();
  }
  for (int i = tid; i < nc; i += blockDim.x) E[b * n + c0 + i] = scalbn(ws[b * n + c0 + i], (int)expo[b]);
  for (int64_t i = tid; i < (int64_t)n * nc; i += blockDim.x) {
    const int r = (int)(i / nc), c = (int)(i % nc);
    U[b * nn + (int64_t)r * n + c0 + c] = z[(size_t)c * ld + r];
  }
}

}  // namespace qsx

using namespace qsx;

extern "C" size_t qsx_eigh_large_workspace_bytes(int n, int64_t batch) {
  if (n < 1 || batch < 0) return 0;
  // reduction matrix and eigenvectors (n^2 each), inverse-iteration scratch
  // (5 n per eigenvalue, whole warps), d/e, their scaled copies and the sorted
  // eigenvalues, limits (4) and the scale, FP32 copy of T
  return (((size_t)7 * n * n + (size_t)5 * n) * (size_t)batch + (size_t)5 * 32 * n +
          (size_t)5 * batch + (size_t)n * batch) * sizeof(double);
}

extern "C" int qsx_eigh_large_batched(const double* H, int n, int64_t batch, double* E,
                                      double* U, void* workspace, size_t workspace_bytes,
                                      int32_t* status, void* stream) {
  QSX_CHECK_ARG(n >= 1 && n <= 2048, "qsx_eigh_large_batched: n=%d outside 1..2048", n);
  QSX_CHECK_ARG(batch >= 0 && batch <= 0x7fffffff, "qsx_eigh_large_batched: bad batch");
  if (batch == 0) return QSX_OK;
  QSX_CHECK_ARG(H && E && U && status, "qsx_eigh_large_batched: null pointer");
  const size_t need = qsx_eigh_large_workspace_bytes(n, batch);
  QSX_CHECK_ARG(workspace && workspace_bytes >= need,
                "qsx_eigh_large_batched: workspace of %zu bytes needed (got %zu)", need,
                workspace_bytes);
  cudaStream_t s = (cudaStream_t)stream;
  const size_t nnb = (size_t)n * n * batch;
  double* W = (double*)workspace;
  double* Z = W + nnb;
  double* scratch = Z + nnb;
  double* de = scratch + 5 * nnb + 5 * 32 * (size_t)n;
  double* tri = de + 2 * (size_t)n * batch;
  double* ws = de + 4 * (size_t)n * batch;
  double* lim = ws + (size_t)n * batch;
  double* expo = lim + 4 * (size_t)batch;
  float* trif = (float*)(expo + batch);
  int dev = 0, sms = 0;
  cudaError_t err = cudaGetDevice(&dev);
  if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (err != cudaSuccess) return cuda_status(err, "qsx_eigh_large_batched");
  // Tridiagonal form: what holds a matrix's columns, and from there as many
  // CTAs as leave every SM one (more would wait for a place) with 32 columns
  // each at least (two cluster barriers a step cost as much as that)
  const size_t most = 220 * 1024;
  auto tri_smem = [&](int c) {
    return ((size_t)((n + c - 1) / c) * tri_ld(n) + 3 * (size_t)n + 6) *
           sizeof(double);
  };
  int c = 1;
  while (c < TC_MAX_CLUSTER && (tri_smem(c) > most || (2 * c * batch <= sms && n >= 64 * c)))
    c *= 2;
  const size_t smemA = tri_smem(c);
  if (smemA <= most && batch * c <= 0x7fffffffLL) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(batch * c));
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smemA;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = c;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    err = cudaFuncSetAttribute(eigh_tridiag_cluster_kernel,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemA);
    if (err == cudaSuccess)
      err = cudaLaunchKernelEx(&cfg, eigh_tridiag_cluster_kernel, H, n, c, W, de, expo);
  } else {
    const int threads = n >= TQ_THREADS ? TQ_THREADS : ((n + 31) / 32) * 32;
    const size_t smem = ((size_t)2 * n + 32) * sizeof(double);
    err = cudaFuncSetAttribute(eigh_tridiag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smem);
    if (err == cudaSuccess)
      eigh_tridiag_kernel<<<(unsigned)batch, threads, smem, s>>>(H, n, W, de, expo);
  }
  if (err != cudaSuccess) return cuda_status(err, "qsx_eigh_large_batched");
  const int64_t nt = batch * n;
  eigh_scale_kernel<<<(unsigned)((batch + 3) / 4), 128, 0, s>>>(de, n, batch, tri, trif, lim);
  eigh_bisect_kernel<<<(unsigned)((nt + 127) / 128), 128, 0, s>>>(tri, trif, lim, n, batch, ws,
                                                                   status);
  eigh_invit_kernel<<<(unsigned)((nt + 127) / 128), 128, 0, s>>>(de, ws, n, batch, Z, scratch);
  eigh_orthogonalise_kernel<<<(unsigned)((nt + 3) / 4), 128, 0, s>>>(de, ws, n, batch, Z);
  // Back-transform: a tile of columns per SM and matrix, what fits, and as
  // many lanes to a column as fill the CTA's warps
  const int per = std::max<int>(1, (int)(sms / batch));
  int cols = (n + per - 1) / per;
  cols = std::min<int>(cols, (int)((most / sizeof(double) - 2 * n - 2) / tri_ld(n)));
  cols = std::min(std::max(cols, 1), BT_THREADS / 4);
  int parts = 4;
  while (parts < 32 && 2 * parts * cols <= BT_THREADS) parts *= 2;
  const size_t smemD = ((size_t)cols * tri_ld(n) + 2 * (size_t)n + 2) * sizeof(double);
  err = cudaFuncSetAttribute(eigh_backtransform_kernel,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smemD);
  if (err != cudaSuccess) return cuda_status(err, "qsx_eigh_large_batched");
  for (int64_t b0 = 0; b0 < batch; b0 += 65535) {   // the grid's second dimension
    const int64_t nb = std::min<int64_t>(65535, batch - b0);
    const int64_t nn = (int64_t)n * n;
    eigh_backtransform_kernel<<<dim3((unsigned)((n + cols - 1) / cols), (unsigned)nb),
                                (cols * parts + 31) / 32 * 32, smemD, s>>>(
        W + b0 * nn, ws + b0 * n, expo + b0, n, cols, parts, Z + b0 * nn, E + b0 * n, U + b0 * nn);
  }
  QSX_LAUNCH_CHECK("qsx_eigh_large_batched");
  return QSX_OK;
}
