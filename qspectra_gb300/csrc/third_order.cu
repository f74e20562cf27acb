// Third-order response at large site counts: the two-exciton (f) manifold
// in operator form.
//
// The reference builds the dense Redfield tensor of the whole 'gef' space
// (qspectra/dynamics/redfield.py:9-74) and slices Liouville blocks out of it
// (liouville_space.py:316-341); at 24 sites that tensor has 301^4 entries.
// The generator is block-diagonal over manifolds, so the 'fe' block used by
// the excited-state-absorption pathways of third_order_response
// (qspectra/simulate/response.py:297-336) needs only the f-manifold
// operators M_i^f, the e-manifold operators M_i^e and the two Hamiltonians.
//
// Entry points (declared in include/qsx.h):
//   qsx_fblock_tensor        eigenbasis tensor Kt_i o C of the f manifold
//                            (redfield.py:41-69 restricted to one manifold)
//   qsx_fe_generator         Q_b = M_b^f - G^f - i uc H^f, the column
//                            operators of the 'fe' block
//   qsx_fe_heisenberg_rk4    RK4 on the transposed 'fe' block
//   qsx_csr_map_batched      sparse dipole super-operator maps between blocks
#include <algorithm>

#include "qsx_bath.cuh"
#include "qsx_common.cuh"

namespace qsx {

// ------------------------------------------------------------------ f tensor
// Kt_i = U^T diag(occ_i) U over the pair states p = (k, l) (occ_i(p) = 1 when
// i is k or l), and Y_i[c][d] = uc * Kt_i[c][d] * C(E_d - E_c): the operator
// M_i^f = U Y_i U^T in the site basis (the same construction as the dense
// Redfield operators kernel, per manifold).  Output layout, per sample, is
// Y[c][plane][d] with planes 0..N-1 the real parts and N..2N-1 the imaginary
// parts, so that U @ Y and (U Y) @ U^T are two plain batched GEMMs.
constexpr int FT = 16;  // tile edge

template <typename T>
__global__ void __launch_bounds__(256)
    fblock_tensor_kernel(const double* __restrict__ E, const double* __restrict__ U, int P,
                         int N, const int* __restrict__ site_pairs, DebyeParams bath, double uc,
                         T* __restrict__ Y) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double* sUc = (double*)smraw;           // [P][FT]
  double* sUd = sUc + (size_t)P * FT;     // [P][FT]
  T* sMir = (T*)(sUd + (size_t)P * FT);   // [2][FT][FT + 1] mirror staging
  int* sPairs = (int*)(sMir + 2 * FT * (FT + 1));  // [N][N - 1]
  const int64_t s = blockIdx.y;
  // upper-triangular tile pair (tc <= td) from the linear block index
  const int ntile = (P + FT - 1) / FT;
  int t = blockIdx.x, tc = 0;
  while (t >= ntile - tc) {
    t -= ntile - tc;
    ++tc;
  }
  const int td = tc + t;
  const int c0 = tc * FT, d0 = td * FT;
  const double* u = U + s * (int64_t)P * P;
  for (int e = threadIdx.x; e < P * FT; e += blockDim.x) {
    const int p = e / FT, j = e % FT;
    sUc[e] = c0 + j < P ? u[(int64_t)p * P + c0 + j] : 0.0;
    sUd[e] = d0 + j < P ? u[(int64_t)p * P + d0 + j] : 0.0;
  }
  for (int e = threadIdx.x; e < N * (N - 1); e += blockDim.x) sPairs[e] = site_pairs[e];
  __syncthreads();
  const int r = threadIdx.x / FT, q = threadIdx.x % FT;
  const int c = c0 + r, d = d0 + q;
  const bool live = c < P && d < P;
  double2 cp = make_double2(0.0, 0.0), cn = cp;
  if (live) debye_corr_pair(bath, E[s * P + d] - E[s * P + c], cp, cn);
  const bool mirror = tc != td;
  T* y = Y + s * (int64_t)P * 2 * N * P;
  for (int i = 0; i < N; ++i) {
    double acc = 0.0;
    if (live) {
      const int* pi = sPairs + i * (N - 1);
      for (int j = 0; j < N - 1; ++j) {
        const int p = pi[j];
        acc = fma(sUc[p * FT + r], sUd[p * FT + q], acc);
      }
      acc *= uc;
      y[((int64_t)c * 2 * N + i) * P + d] = (T)(acc * cp.x);
      y[((int64_t)c * 2 * N + N + i) * P + d] = (T)(acc * cp.y);
    }
    if (mirror) {
      // Y_i[d][c] = acc * C(E_c - E_d): staged so the stores run along c
      sMir[r * (FT + 1) + q] = (T)(acc * cn.x);
      sMir[FT * (FT + 1) + r * (FT + 1) + q] = (T)(acc * cn.y);
      __syncthreads();
      const int dm = d0 + r, cm = c0 + q;
      if (dm < P && cm < P) {
        y[((int64_t)dm * 2 * N + i) * P + cm] = sMir[q * (FT + 1) + r];
        y[((int64_t)dm * 2 * N + N + i) * P + cm] = sMir[FT * (FT + 1) + q * (FT + 1) + r];
      }
      __syncthreads();
    }
  }
}

// --------------------------------------------------------------- fe generator
// Q[s][q][b][r] = M_b[q][r] - G[q][r] - i uc H[q][r], with M in the plane
// layout above and G = sum_i diag(occ_i) M_i, whose row q (pair (k, l)) is
// M_k[q] + M_l[q].
template <typename T>
__global__ void fe_generator_kernel(const T* __restrict__ M, const double* __restrict__ H,
                                    int P, int N, int64_t batch,
                                    const int* __restrict__ pair_sites, double uc,
                                    typename cplx<T>::type* __restrict__ Q) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= batch * P * P) return;
  const int64_t s = e / ((int64_t)P * P);
  const int q = (int)((e / P) % P), r = (int)(e % P);
  const T* m = M + (s * P + q) * (int64_t)2 * N * P;
  const int k = pair_sites[2 * q], l = pair_sites[2 * q + 1];
  const T gx = m[(int64_t)k * P + r] + m[(int64_t)l * P + r];
  const T gy = m[(int64_t)(N + k) * P + r] + m[(int64_t)(N + l) * P + r];
  const T hy = (T)(uc * H[s * (int64_t)P * P + (int64_t)q * P + r]);
  typename cplx<T>::type* out = Q + (s * P + q) * (int64_t)N * P + r;
  for (int b = 0; b < N; ++b)
    out[(int64_t)b * P] = cmk(m[(int64_t)b * P + r] - gx, m[(int64_t)(N + b) * P + r] - gy - hy);
}

// ------------------------------------------------------------- fe RK4 stage
// The 'fe' block acts on X (P x N: rows pair states, columns e sites; the
// column-stacked vector of the block is X column-major) as
//   (L X)[:, b] = Q_b X[:, b] + row terms,  (L X)[p, :] += X[p, :] R_p^T,
// Q_b = M_b^f - A_f, R_p = conj(M_k^e + M_l^e - A_e) for p = (k, l),
// A = G + i uc H (operator form of the site-basis Redfield generator:
// dX = -A X - X A^+ + sum_i (M_i X K_i + K_i X M_i^+)).  Its plain
// transpose, the Heisenberg-picture generator, is
//   (L^T X)[:, b] = Q_b^T X[:, b] + sum_c X[:, c] R_p[c][b]  (row p),
// so column b reads Q_b[q][r] along r: coalesced in the layout Q[s][q][b][r].
struct FeP {
  int P, N;
  const void* Q;          // [batch][P][N][P] complex (T)
  const void* R;          // [batch][N b][N c][N site] complex (T), see fe_rows_kernel
  const int* pair_sites;  // [P][2]
  double h;
};

// The row operators by column: R[b][c][site] = conj(Me[site][c][b] - Ae[c][b] / 2);
// lanes on consecutive pairs read consecutive sites
template <typename T>
__global__ void fe_rows_kernel(const typename cplx<T>::type* __restrict__ Me,
                               const typename cplx<T>::type* __restrict__ Ae, int N, int64_t batch,
                               typename cplx<T>::type* __restrict__ R) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, nn = (int64_t)N * N;
  if (e >= batch * nn * N) return;
  const int64_t s = e / (nn * N);
  const int b = (int)(e / nn % N), c = (int)(e / N % N), site = (int)(e % N);
  const typename cplx<T>::type m = Me[(s * N + site) * nn + (int64_t)c * N + b];
  const typename cplx<T>::type a = Ae[s * nn + (int64_t)c * N + b];
  R[e] = cmk(m.x - (T)0.5 * a.x, -(m.y - (T)0.5 * a.y));
}

// V values of one load: V = 2 takes two complex64 at once (even P keeps them
// on 16 bytes), V = 1 one complex value
template <typename T, int V> struct FeVec;
template <> struct FeVec<float, 2> { using type = float4; };
template <> struct FeVec<float, 1> { using type = float2; };
template <> struct FeVec<double, 1> { using type = double2; };

__device__ __forceinline__ void fe_mac(float2 (&k)[2], float4 q, float2 x) {
  cfma(k[0], make_float2(q.x, q.y), x);
  cfma(k[1], make_float2(q.z, q.w), x);
}
__device__ __forceinline__ void fe_mac(float2 (&k)[1], float2 q, float2 x) { cfma(k[0], q, x); }
__device__ __forceinline__ void fe_mac(double2 (&k)[1], double2 q, double2 x) { cfma(k[0], q, x); }

// One cooperative kernel runs the loop of all samples, a group of them at a
// time: Q is read once a stage, so the bound is its traffic, and a group is as
// many samples as leave Q in the L2 through all their stages (7 of 24 sites,
// 102 MB).  A launch a stage over all 32 samples streamed Q from HBM at 5.0
// TB/s, 93 us; 66 us in groups.  (One CTA a column, a launch a stage, 113 us.
// Two or four independent teams of half- or quarter-size CTAs, one's barrier
// behind the other's loads: 78 and 100 us, their items too few to come out
// even.)
//
// Work: an item is a tile of rows of one column; four warps share it, each a
// quarter of the sum over q with eight 16-byte loads a lane in flight, and
// add up through shared memory.  Eight items run in a CTA, one CTA an SM; the
// plan picks the tile so that the items come out even over the SMs.
//
// The states cross between SMs once a stage: they are read past the L1
// (ld.global.cg), written, and fenced before the barrier.  Waits are bounded;
// a barrier that never fills sets QSX_ERR_CUDA and everyone leaves.
constexpr int FE_ITEM_WARPS = 4;
constexpr int FE_ITEMS = 8;   // at most: fewer where their shared memory does not fit
constexpr int FE_THREADS = 32 * FE_ITEM_WARPS * FE_ITEMS;

struct FeLoop {
  int64_t batch, y0_stride;
  int group, ntile, tile, nsteps;   // tile: rows of an item, a multiple of V
  const double2* y0;
  void *yh, *yl, *acc, *s0, *s1;    // [group][P N] complex (T)
  double2* out;
  int* status;
  unsigned* barrier;                // zeroed: arrivals, then the abort word
};

// All CTAs of the grid; false when the wait ran out or somebody's did.
__device__ __forceinline__ bool fe_grid_barrier(unsigned* bar, unsigned target, int* status) {
  __shared__ int good;
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(bar, 1u);
    bool done = false;
    for (int i = 0; i < (1 << 24); ++i) {
      unsigned seen;
      asm volatile("ld.acquire.gpu.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
      if ((int)(seen - target) >= 0) {
        done = true;
        break;
      }
      if ((i & 255) == 255 && *(volatile unsigned*)(bar + 1)) break;
    }
    if (!done) {
      atomicExch(bar + 1, 1u);
      if (status) atomicOr(status, QSX_ERR_CUDA);
    }
    good = done;
  }
  __syncthreads();
  return good;
}

template <typename T, int V>
__global__ void __launch_bounds__(FE_THREADS, 1) fe_loop_kernel(FeP p, FeLoop l) {
  using C = typename cplx<T>::type;
  using L = typename FeVec<T, V>::type;
  constexpr bool SPLIT = sizeof(T) == 4;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int P = p.P, N = p.N, per = P * N;
  const int it = threadIdx.x / (32 * FE_ITEM_WARPS), tid = threadIdx.x % (32 * FE_ITEM_WARPS);
  const int lane = tid & 31, w = tid >> 5;
  // this item's column of the stage input, row operators and partial sums
  C* sxb = (C*)smraw + (size_t)it * (P + N * N + FE_ITEM_WARPS * 32 * V);
  C* sR = sxb + P;
  C* part = sR + N * N;
  auto item_sync = [&] {
    asm volatile("bar.sync %0, %1;" ::"r"(it + 1), "r"(32 * FE_ITEM_WARPS) : "memory");
  };
  C *yh = (C*)l.yh, *yl = (C*)l.yl, *acc = (C*)l.acc, *s0 = (C*)l.s0, *s1 = (C*)l.s1;
  const int ctas = gridDim.x;
  const T h = (T)p.h, s6 = h / (T)6;
  unsigned target = 0;
  bool ok = true;
  const int64_t tid_all = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t threads_all = (int64_t)ctas * blockDim.x;
  const int places = blockDim.x / (32 * FE_ITEM_WARPS);
  for (int64_t g0 = 0; g0 < l.batch; g0 += l.group) {
    const int live = (int)min((int64_t)l.group, l.batch - g0);
    for (int64_t e = tid_all; e < (int64_t)live * per; e += threads_all) {
      const int64_t s = g0 + e / per, r = e % per;
      const double2 v = l.y0[s * l.y0_stride + r];
      const C hi = cmk((T)v.x, (T)v.y);
      yh[e] = hi;
      if (SPLIT) yl[e] = cmk((T)(v.x - (double)hi.x), (T)(v.y - (double)hi.y));
      l.out[s * (l.nsteps + 1) * (int64_t)per + r] = v;
    }
    target += ctas;
    if (!fe_grid_barrier(l.barrier, target, l.status)) return;
    const int items = live * N * l.ntile;
    for (int step = 1; step <= l.nsteps; ++step) {
#pragma unroll 1
      for (int stage = 0; stage < 4; ++stage) {
        const C* in = stage == 0 ? yh : (stage & 1) ? s0 : s1;
        C* next = (stage & 1) ? s1 : s0;
        for (int i = blockIdx.x + it * ctas; i < items; i += places * ctas) {
          const int col = i / l.ntile, row0 = i % l.ntile * l.tile;
          const int sl = col / N, b = col % N;
          const int64_t s = g0 + sl;
          const C* x = in + (int64_t)sl * per;
          const C* gr = (const C*)p.R + (s * N + b) * (int64_t)N * N;
          for (int e = tid; e < P; e += 32 * FE_ITEM_WARPS) sxb[e] = __ldcg(x + (int64_t)b * P + e);
          for (int e = tid; e < N * N; e += 32 * FE_ITEM_WARPS) sR[e] = __ldcg(gr + e);
          item_sync();
          // this warp's part of the column term sum_q Q_b[q][row] X[q][b]
          const int row = row0 + V * lane;
          const bool active = V * lane < l.tile && row < P;   // V = 2: P and the tile are even
          const int q0 = P * w / FE_ITEM_WARPS, q1 = P * (w + 1) / FE_ITEM_WARPS;
          C k[V];
#pragma unroll
          for (int v = 0; v < V; ++v) k[v] = cmk((T)0, (T)0);
          if (active) {
            const C* qcol = (const C*)p.Q + (s * P * N + b) * (int64_t)P + row;
            constexpr int U = 8;
            int q = q0;
            for (; q + U <= q1; q += U) {
              L a[U];
#pragma unroll
              for (int t = 0; t < U; ++t)
                a[t] = __ldcg(reinterpret_cast<const L*>(qcol + (int64_t)(q + t) * per));
#pragma unroll
              for (int t = 0; t < U; ++t) fe_mac(k, a[t], sxb[q + t]);
            }
            for (; q < q1; ++q)
              fe_mac(k, __ldcg(reinterpret_cast<const L*>(qcol + (int64_t)q * per)), sxb[q]);
            // and of the row term sum_c X[row][c] (T_k + T_l)[c]
#pragma unroll
            for (int v = 0; v < V; ++v) {
              const int kk = p.pair_sites[2 * (row + v)], ll = p.pair_sites[2 * (row + v) + 1];
              for (int c = w; c < N; c += FE_ITEM_WARPS) {
                const C ra = sR[c * N + kk], rb = sR[c * N + ll];
                cfma(k[v], __ldcg(x + (int64_t)c * P + row + v), cmk(ra.x + rb.x, ra.y + rb.y));
              }
            }
          }
#pragma unroll
          for (int v = 0; v < V; ++v) part[w * 32 * V + V * lane + v] = k[v];
          item_sync();
          if (tid < l.tile && row0 + tid < P) {
            C kk = part[tid];
#pragma unroll
            for (int q = 1; q < FE_ITEM_WARPS; ++q) kk = cadd2(kk, part[q * 32 * V + tid]);
            const int r = b * P + row0 + tid;
            const int64_t idx = (int64_t)sl * per + r;
            const C y = __ldcg(yh + idx);
            if (stage == 0) {
              acc[idx] = kk;
              next[idx] = cmk(y.x + (T)0.5 * h * kk.x, y.y + (T)0.5 * h * kk.y);
            } else if (stage < 3) {
              const C a0 = __ldcg(acc + idx);
              acc[idx] = cmk(a0.x + (T)2 * kk.x, a0.y + (T)2 * kk.y);
              const T cst = stage == 1 ? (T)0.5 * h : h;
              next[idx] = cmk(y.x + cst * kk.x, y.y + cst * kk.y);
            } else {
              const C a0 = __ldcg(acc + idx);
              const T ix = s6 * (a0.x + kk.x), iy = s6 * (a0.y + kk.y);
              double2 o;
              if constexpr (SPLIT) {
                // split-word state: hi + lo with a TwoSum update
                const C lo = __ldcg(yl + idx);
                float hx = y.x, lx = lo.x, hy = y.y, ly = lo.y;
                dd_add(hx, lx, ix);
                dd_add(hy, ly, iy);
                yh[idx] = cmk(hx, hy);
                yl[idx] = cmk(lx, ly);
                o = make_double2((double)hx + (double)lx, (double)hy + (double)ly);
              } else {
                o = cmk(y.x + ix, y.y + iy);
                yh[idx] = o;
              }
              ok = ok && finite2(o);
              l.out[(s * (l.nsteps + 1) + step) * (int64_t)per + r] = o;
            }
          }
        }
        target += ctas;
        if (!fe_grid_barrier(l.barrier, target, l.status)) return;
      }
    }
  }
  if (!ok && l.status) atomicOr(l.status, QSX_ERR_NONFINITE);
}

// The loop with Q on chip.  Every stage reads all of Q, so past the sizes of
// one CTA its traffic bounds the loop wherever Q lies: from the L2 6.6 TB/s.
// Here a team of CTAs, one an SM, holds a sample's Q in shared memory and
// registers through all its steps, and the teams work through the samples.
//
// A CTA owns consecutive elements of X (column by column, `rows` of them) and
// for each the P values Q[.][b][row], laid out one element a row; warp w holds
// `rs` of its rows in shared memory and RREG in registers.  The lanes split the
// sum over q, each with its part of X's column in registers, and four rows at a
// time add up through shuffles.  The row term, a sum over the columns of X, is
// split over all warps, from the L2, its operators T_k + T_l in shared memory.
// Thread i then holds the state, its low word and the stage sum of element i.
// X crosses between the CTAs of a team once a stage, through the L2 and a
// barrier of the team.
//
// Bound: latency.  Of a stage of 5.7 us (three teams of 50 CTAs, 24 sites) the
// round trip of X takes 2.0, the column terms 2.5 and the row terms 1.2; 16
// warps of 128 registers took 7.1, their row terms with operators from the L1.
// us a stage, the loop over the L2 against this one: 24 sites, FP32, 1 / 3 / 32
// samples 10.2 / 12.2 / 66 and 4.1 / 6.1 / 61; 20 sites 7.2 / 9.9 / 85 and 3.5 /
// 4.6 / 31; 13 sites, 32 samples 15.5 and 6.2; FP64, one sample of 16 / 20 / 22
// sites 13 / 32 / 46 and 6.7 / 9.9 / 16.
constexpr int FE_TEAM_WARPS = 8, FE_TEAM_THREADS = 32 * FE_TEAM_WARPS;
constexpr int FE_TEAM_CT = 8;     // columns of a row-term task
constexpr int FE_TEAM_RREG = 6;   // FP32 rows that a warp can keep in registers
// Terms a lane, of up to 128, 192 and 288 pairs (24 sites).  Past nine the six
// register rows and a lane's part of X no longer fit: 236 registers at nine, 255
// and spills at ten.  25 to 31 sites take the loop over the L2.
constexpr int FE_TEAM_NQ[3] = {4, 6, 9};

struct FeTeam {
  int64_t batch, y0_stride;
  int csize, teams;      // CTAs of a team, teams
  int rows, rw, rs;      // elements a CTA, rows a warp, of them in shared memory
  int nb, parts, nsteps; // columns that a CTA's elements touch, parts of a row term
  const double2* y0;
  void* x;               // [teams][2][P N] complex (T): stage inputs
  double2* out;
  int* status;
  unsigned* barrier;     // [teams][2] zeroed: arrivals, abort word
};

// Elements of the rows in shared memory.  The lanes take 32 NQ terms of a sum
// over P, those past P times 0: in a row's case the rows after it, in the last
// one's zeros, since whatever an earlier kernel left may be NaN.
template <int NQ>
__host__ __device__ constexpr size_t fe_team_held(int P, int rs) {
  return rs ? (size_t)FE_TEAM_WARPS * rs * P + (32 * NQ - P) : 0;
}

template <typename T, int NQ, int RREG>
__global__ void __launch_bounds__(FE_TEAM_THREADS, 1) fe_team_kernel(FeP p, FeTeam t) {
  using C = typename cplx<T>::type;
  constexpr bool SPLIT = sizeof(T) == 4;
  constexpr unsigned ALL = 0xffffffffu;
  constexpr int CT = FE_TEAM_CT;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int P = p.P, N = p.N, per = P * N, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  C* sQ = (C*)smraw;                                  // [warps][rs][P], then zeros
  C* sx = sQ + fe_team_held<NQ>(P, t.rs);             // [nb P] the columns of the input
  C* kq = sx + (size_t)t.nb * P;                      // [rows] column terms
  C* part = kq + t.rows;                              // [parts][rows] row terms
  const int team = blockIdx.x / t.csize;
  const int rho0 = blockIdx.x % t.csize * t.rows, nr = max(0, min(t.rows, per - rho0));
  const int b0 = min(rho0, per - 1) / P, nx = min(t.nb * P, per - b0 * P);
  // this warp's rows; the column of the first one and where the next begins
  const int first = w * t.rw, bf = min(rho0 + first, per - 1) / P;
  const C* wQ = sQ + (size_t)w * t.rs * P;
  C* sW = part + t.parts * t.rows;                    // [N][rows] row operators T_k + T_l
  // row terms: 32 elements of X and CT columns a task
  const int chunks = max(1, (nr + 31) / 32), tasks = nr ? chunks * t.parts : 0;
  const bool own = tid < nr;
  const int me = rho0 + tid;
  C* xbuf = (C*)t.x + (size_t)team * 2 * per;
  const T h = (T)p.h, s6 = h / (T)6;
  unsigned target = 0;
  bool ok = true;
  if (t.rs)
    for (int e = FE_TEAM_WARPS * t.rs * P + tid; sQ + e < sx; e += FE_TEAM_THREADS)
      sQ[e] = cmk((T)0, (T)0);
  for (int64_t s = team; s < t.batch; s += t.teams) {
    const C* Qg = (const C*)p.Q + s * (int64_t)per * P + rho0;
    const C* Rg = (const C*)p.R + s * (int64_t)N * N * N;
    double2* o = t.out + s * (t.nsteps + 1) * (int64_t)per;
    const int held = FE_TEAM_WARPS * t.rs;
    for (int e = tid; e < held * P; e += FE_TEAM_THREADS) {
      const int i = e % held, q = e / held, local = i / t.rs * t.rw + i % t.rs;
      sQ[(size_t)i * P + q] = local < nr ? Qg[(int64_t)q * per + local] : cmk((T)0, (T)0);
    }
    C qr[RREG ? RREG : 1][NQ];
#pragma unroll
    for (int i = 0; i < RREG; ++i)
#pragma unroll
      for (int j = 0; j < NQ; ++j) {
        const int q = lane + 32 * j, local = first + t.rs + i;
        qr[i][j] = (i + t.rs < t.rw && local < nr && q < P) ? Qg[(int64_t)q * per + local]
                                                            : cmk((T)0, (T)0);
      }
    for (int e = tid; e < N * nr; e += FE_TEAM_THREADS) {
      const int c = e / nr, rl = e % nr, row = (rho0 + rl) % P;
      const C* r = Rg + ((size_t)((rho0 + rl) / P) * N + c) * N;
      sW[c * t.rows + rl] = cadd2(r[p.pair_sites[2 * row]], r[p.pair_sites[2 * row + 1]]);
    }
    C yh = cmk((T)0, (T)0), yl = yh, ac = yh;
    if (own) {
      const double2 v = t.y0[s * t.y0_stride + me];
      yh = cmk((T)v.x, (T)v.y);
      if (SPLIT) yl = cmk((T)(v.x - (double)yh.x), (T)(v.y - (double)yh.y));
      xbuf[me] = yh;
      o[me] = v;
    }
    target += t.csize;
    if (!fe_grid_barrier(t.barrier + 2 * team, target, t.status)) return;
    int cur = 0;
    for (int step = 1; step <= t.nsteps; ++step) {
#pragma unroll 1
      for (int stage = 0; stage < 4; ++stage, cur ^= 1) {
        const C* in = xbuf + (size_t)cur * per;
        for (int e = tid; e < nx; e += FE_TEAM_THREADS) sx[e] = __ldcg(in + b0 * P + e);
        __syncthreads();
        // odd warps form row terms before their column terms, even warps after:
        // the trips to the L2 lie under the others' sums
        auto row_terms = [&] {
          for (int i = w; i < tasks; i += FE_TEAM_WARPS) {
            const int pt = i / chunks, rl = i % chunks * 32 + lane;
            if (rl >= nr) continue;
            const C* at = in + (size_t)pt * CT * P + (rho0 + rl) % P;
            const C* u = sW + (size_t)pt * CT * t.rows + rl;
            C x[CT], k = cmk((T)0, (T)0);
            const int n = N - pt * CT;
#pragma unroll
            for (int c = 0; c < CT; ++c) x[c] = c < n ? __ldcg(at + (size_t)c * P) : cmk((T)0, (T)0);
#pragma unroll
            for (int c = 0; c < CT; ++c) cfma(k, x[c], u[min(c, n - 1) * t.rows]);
            part[pt * t.rows + rl] = k;
          }
        };
        if (w & 1) row_terms();
        if (first < nr) {
          C xr[NQ];
          int b = bf, bend = (bf + 1) * P - rho0;
          auto column = [&] {
#pragma unroll
            for (int j = 0; j < NQ; ++j) {
              const int q = lane + 32 * j;
              xr[j] = q < P ? sx[(b - b0) * P + q] : cmk((T)0, (T)0);
            }
          };
          column();
          // the sums of R rows over the lanes: halves of the 2 R words change
          // sides until each lane holds a part of one word
          auto add_up = [&](auto& k, int local, int count) {
            constexpr int R = sizeof(k) / sizeof(C);
            T v[2 * R];
#pragma unroll
            for (int i = 0; i < R; ++i) {
              v[2 * i] = k[i].x;
              v[2 * i + 1] = k[i].y;
            }
            constexpr int STEP = 32 / (2 * R);     // lanes that share a word
#pragma unroll
            for (int n = R; n >= 1; n /= 2) {
              const bool hi = lane & (STEP * n);
#pragma unroll
              for (int i = 0; i < n; ++i) {
                const T keep = hi ? v[i + n] : v[i], give = hi ? v[i] : v[i + n];
                v[i] = keep + __shfl_xor_sync(ALL, give, STEP * n);
              }
            }
#pragma unroll
            for (int n = STEP / 2; n >= 1; n /= 2) v[0] += __shfl_xor_sync(ALL, v[0], n);
            const int at = lane / STEP;
            if (lane % STEP == 0 && at / 2 < count && local + at / 2 < nr)
              reinterpret_cast<T*>(kq)[2 * local + at] = v[0];
          };
          constexpr int R = 4;
#pragma unroll 1
          for (int i0 = 0; i0 < t.rs; i0 += R) {
            C k[R];
#pragma unroll
            for (int i = 0; i < R; ++i) k[i] = cmk((T)0, (T)0);
            const C* q = wQ + (size_t)i0 * P + lane;
            const int last = min(R, t.rs - i0) - 1;
            if (first + i0 + last < min(nr, bend) && (SPLIT || last == R - 1)) {
              // past P: what follows, times 0; past the last row: that row again
              const C* qi[R];
#pragma unroll
              for (int i = 0; i < R; ++i) qi[i] = q + min(i, last) * P;
#pragma unroll
              for (int j = 0; j < NQ; ++j)
#pragma unroll
                for (int i = 0; i < R; ++i) cfma(k[i], qi[i][32 * j], xr[j]);
            } else {
#pragma unroll
              for (int i = 0; i < R; ++i) {
                if (i0 + i >= t.rs || first + i0 + i >= nr) continue;
                if (first + i0 + i >= bend) {
                  ++b;
                  bend += P;
                  column();
                }
#pragma unroll
                for (int j = 0; j < NQ; ++j) cfma(k[i], q[i * P + 32 * j], xr[j]);
              }
            }
            add_up(k, first + i0, t.rs - i0);   // rows past rs are others'
          }
          if constexpr (RREG > 0) {
            constexpr int R2 = RREG > 4 ? 8 : 4;
            static_assert(RREG <= 8, "one batch of register rows");
            C k[R2];
#pragma unroll
            for (int i = 0; i < R2; ++i) k[i] = cmk((T)0, (T)0);
#pragma unroll
            for (int i = 0; i < RREG; ++i) {
              const int local = first + t.rs + i;
              if (local >= bend && local < nr) {
                ++b;
                bend += P;
                column();
              }
#pragma unroll
              for (int j = 0; j < NQ; ++j) cfma(k[i], qr[i][j], xr[j]);
            }
            add_up(k, first + t.rs, t.rw - t.rs);
          }
        }
        if (!(w & 1)) row_terms();
        __syncthreads();
        if (own) {
          C k = kq[tid];
          for (int i = 0; i < t.parts; ++i) k = cadd2(k, part[i * t.rows + tid]);
          C next;
          if (stage < 3) {
            ac = stage == 0 ? k : cmk(ac.x + (T)2 * k.x, ac.y + (T)2 * k.y);
            const T cst = stage < 2 ? (T)0.5 * h : h;
            next = cmk(yh.x + cst * k.x, yh.y + cst * k.y);
          } else {
            const T ix = s6 * (ac.x + k.x), iy = s6 * (ac.y + k.y);
            double2 v;
            if constexpr (SPLIT) {
              dd_add(yh.x, yl.x, ix);
              dd_add(yh.y, yl.y, iy);
              v = make_double2((double)yh.x + (double)yl.x, (double)yh.y + (double)yl.y);
            } else {
              yh = cmk(yh.x + ix, yh.y + iy);
              v = yh;
            }
            ok = ok && finite2(v);
            o[(int64_t)step * per + me] = v;
            next = yh;
          }
          xbuf[(size_t)(cur ^ 1) * per + me] = next;
        }
        target += t.csize;
        if (!fe_grid_barrier(t.barrier + 2 * team, target, t.status)) return;
      }
    }
  }
  if (!ok && t.status) atomicOr(t.status, QSX_ERR_NONFINITE);
}

// A team of csize CTAs for P pairs and N sites, rreg register rows a warp;
// false when it does not fit
template <typename T>
static bool fe_team_shape(int P, int N, int csize, int rreg, FeTeam* t, size_t* smem) {
  using C = typename cplx<T>::type;
  const int per = P * N;
  t->csize = csize;
  t->rows = (per + csize - 1) / csize;
  if (t->rows > FE_TEAM_THREADS) return false;
  t->rw = (t->rows + FE_TEAM_WARPS - 1) / FE_TEAM_WARPS;
  t->rs = std::max(0, t->rw - rreg);
  t->nb = std::min(N, (t->rows + P - 2) / P + 1);
  t->parts = (N + FE_TEAM_CT - 1) / FE_TEAM_CT;
  const size_t held = P <= 32 * FE_TEAM_NQ[0]   ? fe_team_held<FE_TEAM_NQ[0]>(P, t->rs)
                      : P <= 32 * FE_TEAM_NQ[1] ? fe_team_held<FE_TEAM_NQ[1]>(P, t->rs)
                                                : fe_team_held<FE_TEAM_NQ[2]>(P, t->rs);
  *smem = (held + (size_t)t->nb * P +
           (size_t)(1 + t->parts + N) * t->rows) * sizeof(C);
  return *smem <= 226 * 1024;
}

template <typename T>
static const void* fe_team_entry(int P, int rreg) {
#define FE_TEAM(NQ)                                                                        \
  if (P <= 32 * NQ) {                                                                      \
    if constexpr (sizeof(T) == 4) {                                                        \
      if (rreg) return (const void*)fe_team_kernel<T, NQ, FE_TEAM_RREG>;                   \
    }                                                                                      \
    return rreg ? nullptr : (const void*)fe_team_kernel<T, NQ, 0>;                         \
  }
  FE_TEAM(FE_TEAM_NQ[0]) FE_TEAM(FE_TEAM_NQ[1]) FE_TEAM(FE_TEAM_NQ[2])
#undef FE_TEAM
  return nullptr;
}

// The whole loop of samples whose Q fits one CTA's shared memory, one launch
// and one CTA a sample: thread e owns the elements e, e + 256, .. of X, its
// state and stage sums in registers, the stage inputs in shared memory.  For
// these sizes a stage is shorter than its launch: 4 sites, one FP64 sample,
// 99 steps were 496 launches, 2.2 ms on the device and more between them.
constexpr int FE_CTA = 256;
constexpr int FE_EPT = 2;   // elements a thread

template <typename T>
__global__ void __launch_bounds__(FE_CTA)
    fe_cta_kernel(FeP p, const double2* __restrict__ y0, int64_t y0_stride, int nsteps,
                  double2* __restrict__ out, int* status) {
  using C = typename cplx<T>::type;
  constexpr bool SPLIT = sizeof(T) == 4;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int P = p.P, N = p.N, per = P * N;
  C* sQ = (C*)smraw;               // [P][N][P]
  C* sR = sQ + (size_t)per * P;    // [N b][N c][N site]
  C* sx = sR + (size_t)N * N * N;  // [2][P N] stage input
  const int64_t s = blockIdx.x;
  for (int i = threadIdx.x; i < per * P; i += FE_CTA) sQ[i] = ((const C*)p.Q)[s * per * P + i];
  for (int i = threadIdx.x; i < N * N * N; i += FE_CTA)
    sR[i] = ((const C*)p.R)[s * (int64_t)N * N * N + i];
  C yh[FE_EPT], yl[FE_EPT], ac[FE_EPT];
  int row[FE_EPT], col[FE_EPT], ka[FE_EPT], kb[FE_EPT];
  double2* o = out + s * (nsteps + 1) * (int64_t)per;
#pragma unroll
  for (int i = 0; i < FE_EPT; ++i) {
    const int e = threadIdx.x + i * FE_CTA;
    const bool live = e < per;
    const double2 v = live ? y0[s * y0_stride + e] : make_double2(0.0, 0.0);
    yh[i] = cmk((T)v.x, (T)v.y);
    yl[i] = SPLIT ? cmk((T)(v.x - (double)yh[i].x), (T)(v.y - (double)yh[i].y))
                  : cmk((T)0, (T)0);
    ac[i] = cmk((T)0, (T)0);
    row[i] = live ? e % P : 0;
    col[i] = live ? e / P : 0;
    ka[i] = live ? p.pair_sites[2 * row[i]] : 0;
    kb[i] = live ? p.pair_sites[2 * row[i] + 1] : 0;
    if (live) {
      sx[e] = yh[i];
      o[e] = make_double2((double)yh[i].x + (double)yl[i].x, (double)yh[i].y + (double)yl[i].y);
    }
  }
  __syncthreads();
  const T h = (T)p.h, s6 = h / (T)6;
  bool ok = true;
  int cur = 0;
  for (int step = 1; step <= nsteps; ++step) {
#pragma unroll 1
    for (int stage = 0; stage < 4; ++stage, cur ^= 1) {
      const C* in = sx + cur * per;
      C* nx = sx + (cur ^ 1) * per;
#pragma unroll
      for (int i = 0; i < FE_EPT; ++i) {
        const int e = threadIdx.x + i * FE_CTA;
        if (e >= per) break;
        const C* q = sQ + e;              // Q[q][col][row] at q * per + e
        const C* xb = in + col[i] * P;
        C k0 = cmk((T)0, (T)0), k1 = k0;
        int j = 0;
        for (; j + 1 < P; j += 2) {
          cfma(k0, q[(size_t)j * per], xb[j]);
          cfma(k1, q[(size_t)(j + 1) * per], xb[j + 1]);
        }
        if (j < P) cfma(k0, q[(size_t)j * per], xb[j]);
        const C* r = sR + col[i] * N * N;
        for (int c = 0; c < N; ++c) {
          const C ra = r[c * N + ka[i]], rb = r[c * N + kb[i]];
          cfma(k1, in[c * P + row[i]], cmk(ra.x + rb.x, ra.y + rb.y));
        }
        const C k = cadd2(k0, k1);
        if (stage == 0) {
          ac[i] = k;
        } else if (stage < 3) {
          ac[i] = cmk(ac[i].x + (T)2 * k.x, ac[i].y + (T)2 * k.y);
        } else {
          const T ix = s6 * (ac[i].x + k.x), iy = s6 * (ac[i].y + k.y);
          if (SPLIT) {
            float hx = (float)yh[i].x, lx = (float)yl[i].x, hy = (float)yh[i].y,
                  ly = (float)yl[i].y;
            dd_add(hx, lx, (float)ix);
            dd_add(hy, ly, (float)iy);
            yh[i] = cmk((T)hx, (T)hy);
            yl[i] = cmk((T)lx, (T)ly);
          } else {
            yh[i] = cmk(yh[i].x + ix, yh[i].y + iy);
          }
        }
        const T cst = stage < 2 ? (T)0.5 * h : h;
        nx[e] = stage < 3 ? cmk(yh[i].x + cst * k.x, yh[i].y + cst * k.y) : yh[i];
        if (stage == 3) {
          const double2 v = make_double2((double)yh[i].x + (double)yl[i].x,
                                         (double)yh[i].y + (double)yl[i].y);
          ok = ok && finite2(v);
          o[(int64_t)step * per + e] = v;
        }
      }
      __syncthreads();
    }
  }
  if (!ok && status) atomicOr(status, QSX_ERR_NONFINITE);
}

// ------------------------------------------------------------------ CSR map
// out[b][r] = sum_k vals[k] in[b][cols[k]] over rowptr[r] <= k < rowptr[r+1].
__global__ void csr_map_kernel(const double2* __restrict__ in, int64_t n_in, int64_t batch,
                               const int* __restrict__ rowptr, const int* __restrict__ cols,
                               const double2* __restrict__ vals, int n_out,
                               double2* __restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= batch * n_out) return;
  const int64_t b = e / n_out;
  const int r = (int)(e % n_out);
  const double2* x = in + b * n_in;
  double2 acc = make_double2(0.0, 0.0);
  for (int k = rowptr[r]; k < rowptr[r + 1]; ++k) {
    const double2 v = vals[k], xv = x[cols[k]];
    acc.x = fma(v.x, xv.x, fma(-v.y, xv.y, acc.x));
    acc.y = fma(v.x, xv.y, fma(v.y, xv.x, acc.y));
  }
  out[e] = acc;
}

}  // namespace qsx

using namespace qsx;

extern "C" int qsx_fblock_tensor(const double* E, const double* U, int P, int N,
                                 const int* site_pairs, int64_t batch, double temperature,
                                 double reorg_energy, double cutoff_freq, int matsubara_cutoff,
                                 int discard_imag_corr, double unit_convert, int precision,
                                 void* Y, void* stream) {
  QSX_CHECK_ARG(N >= 2 && N <= 64 && P == N * (N - 1) / 2,
                "qsx_fblock_tensor: P=%d must be N(N-1)/2 for N=%d sites", P, N);
  QSX_CHECK_ARG(batch >= 0 && batch <= 65535, "qsx_fblock_tensor: batch out of range");
  QSX_CHECK_ARG(precision == QSX_FP32 || precision == QSX_FP64,
                "qsx_fblock_tensor: bad precision");
  QSX_CHECK_ARG(temperature > 0 && cutoff_freq > 0 && matsubara_cutoff >= 1,
                "qsx_fblock_tensor: bad bath parameters");
  if (batch == 0) return QSX_OK;
  QSX_CHECK_ARG(E && U && site_pairs && Y, "qsx_fblock_tensor: null pointer");
  const DebyeParams bath = make_debye(temperature, reorg_energy, cutoff_freq, matsubara_cutoff,
                                      discard_imag_corr != 0);
  const int ntile = (P + FT - 1) / FT;
  const dim3 grid((unsigned)(ntile * (ntile + 1) / 2), (unsigned)batch);
  cudaStream_t s = (cudaStream_t)stream;
  auto run = [&](auto tag) -> int {
    using T = decltype(tag);
    const size_t smem = 2 * (size_t)P * FT * sizeof(double) + 2 * FT * (FT + 1) * sizeof(T) +
                        (size_t)N * (N - 1) * sizeof(int);
    QSX_CHECK_ARG(smem <= 227 * 1024, "qsx_fblock_tensor: %d pair states exceed shared memory",
                  P);
    cudaError_t e = cudaFuncSetAttribute(fblock_tensor_kernel<T>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_status(e, "qsx_fblock_tensor");
    fblock_tensor_kernel<T><<<grid, FT * FT, smem, s>>>(E, U, P, N, site_pairs, bath,
                                                        unit_convert, (T*)Y);
    QSX_LAUNCH_CHECK("qsx_fblock_tensor");
    return QSX_OK;
  };
  return precision == QSX_FP32 ? run(0.0f) : run(0.0);
}

extern "C" int qsx_fe_generator(const void* M, const double* H, int P, int N, int64_t batch,
                                const int* pair_sites, double unit_convert, int precision,
                                void* Q, void* stream) {
  QSX_CHECK_ARG(N >= 2 && N <= 64 && P == N * (N - 1) / 2,
                "qsx_fe_generator: P=%d must be N(N-1)/2 for N=%d sites", P, N);
  QSX_CHECK_ARG(batch >= 0, "qsx_fe_generator: negative batch");
  QSX_CHECK_ARG(precision == QSX_FP32 || precision == QSX_FP64,
                "qsx_fe_generator: bad precision");
  if (batch == 0) return QSX_OK;
  QSX_CHECK_ARG(M && H && pair_sites && Q, "qsx_fe_generator: null pointer");
  const int64_t n = batch * P * P;
  const unsigned grid = (unsigned)((n + 255) / 256);
  cudaStream_t s = (cudaStream_t)stream;
  if (precision == QSX_FP32)
    fe_generator_kernel<float><<<grid, 256, 0, s>>>((const float*)M, H, P, N, batch, pair_sites,
                                                    unit_convert, (float2*)Q);
  else
    fe_generator_kernel<double><<<grid, 256, 0, s>>>((const double*)M, H, P, N, batch,
                                                     pair_sites, unit_convert, (double2*)Q);
  QSX_LAUNCH_CHECK("qsx_fe_generator");
  return QSX_OK;
}

extern "C" size_t qsx_fe_heisenberg_workspace_bytes(int P, int N, int64_t batch, int precision) {
  if (P < 1 || N < 1 || batch < 0) return 0;
  const size_t cs = precision == QSX_FP32 ? sizeof(float2) : sizeof(double2);
  const size_t n = (size_t)P * N * (size_t)batch;
  return 16 + ((precision == QSX_FP32 ? 5 : 4) * n + (size_t)N * N * N * (size_t)batch) * cs;
}

extern "C" int qsx_fe_heisenberg_rk4(const void* Q, const void* Ae, const void* Me,
                                     const int* pair_sites, int P, int N, int64_t batch,
                                     int precision, const double* y0, int64_t y0_stride,
                                     int nsteps, double h, double* out, void* workspace,
                                     size_t workspace_bytes, int32_t* status, void* stream) {
  QSX_CHECK_ARG(N >= 2 && N <= 64 && P == N * (N - 1) / 2,
                "qsx_fe_heisenberg_rk4: P=%d must be N(N-1)/2 for N=%d sites", P, N);
  QSX_CHECK_ARG(batch >= 0 && batch <= 65535 && nsteps >= 0,
                "qsx_fe_heisenberg_rk4: batch or step count out of range");
  QSX_CHECK_ARG(precision == QSX_FP32 || precision == QSX_FP64,
                "qsx_fe_heisenberg_rk4: bad precision");
  if (batch == 0) return QSX_OK;
  QSX_CHECK_ARG(Q && Ae && Me && pair_sites && y0 && out && status,
                "qsx_fe_heisenberg_rk4: null pointer");
  const size_t need = qsx_fe_heisenberg_workspace_bytes(P, N, batch, precision);
  QSX_CHECK_ARG(workspace && workspace_bytes >= need,
                "qsx_fe_heisenberg_rk4: workspace of %zu bytes needed (got %zu)", need,
                workspace_bytes);
  cudaStream_t s = (cudaStream_t)stream;
  FeP p;
  p.P = P;
  p.N = N;
  p.Q = Q;
  p.pair_sites = pair_sites;
  p.h = h;
  const int64_t per = (int64_t)P * N;
  const int64_t n = per * batch;
  int dev = 0, sms = 0, l2 = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev);
  if (e != cudaSuccess) return cuda_status(e, "qsx_fe_heisenberg_rk4");
  auto run = [&](auto tag) -> int {
    using T = decltype(tag);
    using C = typename cplx<T>::type;
    unsigned* barrier = (unsigned*)workspace;
    C* yh = (C*)((char*)workspace + 16);
    C* yl = sizeof(T) == 4 ? yh + n : nullptr;
    C* acc = yh + (sizeof(T) == 4 ? 2 : 1) * n;
    C* s0 = acc + n;
    C* s1 = s0 + n;
    C* R = s1 + n;
    p.R = R;
    const int64_t rows = batch * (int64_t)N * N * N;
    fe_rows_kernel<T><<<(unsigned)((rows + 255) / 256), 256, 0, s>>>((const C*)Me, (const C*)Ae,
                                                                     N, batch, R);
    // One CTA a sample while Q fits beside the state, and while its stage
    // (multiply-adds at an SM's rate: 128 a clock in FP32, 2 in FP64, from
    // shared memory a quarter of the FP32 rate) costs less than the 6 us that
    // a launched stage takes at least
    const size_t cta = ((size_t)per * P + (size_t)N * N * N + 2 * (size_t)per) * sizeof(C);
    const double fma = 4.0 * (double)per * (P + 2 * N);
    const double stage_us = fma / (sizeof(T) == 4 ? 32.0 : 2.0) / 1900.0 *
                            (double)((batch + sms - 1) / sms);
    if (per <= FE_CTA * FE_EPT && cta <= 200 * 1024 && stage_us < 6.0) {
      e = cudaFuncSetAttribute(fe_cta_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)cta);
      if (e != cudaSuccess) return cuda_status(e, "qsx_fe_heisenberg_rk4");
      fe_cta_kernel<T><<<(unsigned)batch, FE_CTA, cta, s>>>(p, (const double2*)y0, y0_stride,
                                                          nsteps, (double2*)out, status);
      QSX_LAUNCH_CHECK("qsx_fe_heisenberg_rk4");
      return QSX_OK;
    }
    // Q on chip when a team of CTAs holds it, with the team and the register
    // rows of the shortest loop.  A stage in us, fitted to 11 to 24 sites and 1
    // to 64 samples: 2.5 for its round trip and 110 ps an element of Q that a
    // CTA holds; in FP64 3.5 and the multiply-adds at two a clock.  The loop
    // over the L2 takes its traffic at 6.6 TB/s at least, and 3 us; in FP64
    // 1.35 times its multiply-adds, and 6 us.
    const double elements = (double)per * P * (double)batch;
    const double over_l2 = sizeof(T) == 4 ? 3.0 + elements * sizeof(C) / 6.6e6
                                          : 6.0 + 1.35 * 4.0 * elements / (2.0 * sms * 1900.0);
    const double lanes = P <= 128 ? 128 : P <= 192 ? 192 : 288;
    FeTeam team, pick;
    size_t tsmem = 0, psmem = 0;
    const void* pentry = nullptr;
    double pcost = 0;
    for (int rreg = 0; rreg <= FE_TEAM_RREG; rreg += FE_TEAM_RREG) {
      const void* entry = fe_team_entry<T>(P, rreg);
      for (int c = 1; entry && c <= sms; ++c) {
        if (!fe_team_shape<T>(P, N, c, rreg, &team, &tsmem)) continue;
        team.teams = (int)std::min<int64_t>(batch, sms / c);
        const double cost = (double)((batch + team.teams - 1) / team.teams) *
                            (sizeof(T) == 4 ? 2.5 + 110e-6 * team.rows * P
                                            : 3.5 + team.rows * lanes * 4.0 / (2.0 * 1900.0));
        if (cost < (pentry ? pcost : over_l2)) {
          pick = team;
          pentry = entry;
          psmem = tsmem;
          pcost = cost;
        }
      }
    }
    if (pentry) {
      pick.batch = batch;
      pick.y0 = (const double2*)y0;
      pick.y0_stride = y0_stride;
      pick.nsteps = nsteps;
      pick.x = yh;                       // two of the five state arrays
      pick.out = (double2*)out;
      pick.status = status;
      pick.barrier = (unsigned*)(yh + 2 * n);
      e = cudaMemsetAsync(pick.barrier, 0, 2 * sizeof(unsigned) * pick.teams, s);
      if (e == cudaSuccess)
        e = cudaFuncSetAttribute(pentry, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)psmem);
      void* args[] = {&p, &pick};
      if (e == cudaSuccess)
        e = cudaLaunchCooperativeKernel(pentry, dim3(pick.teams * pick.csize),
                                        dim3(FE_TEAM_THREADS), args, psmem, s);
      if (e != cudaSuccess) return cuda_status(e, "qsx_fe_heisenberg_rk4");
      QSX_LAUNCH_CHECK("qsx_fe_heisenberg_rk4");
      return QSX_OK;
    }
    constexpr int V2 = sizeof(T) == 4 ? 2 : 1;
    const bool wide = P % 2 == 0 && ((uintptr_t)Q & 15) == 0;
    const int V = wide ? V2 : 1;
    auto kern = wide ? fe_loop_kernel<T, V2> : fe_loop_kernel<T, 1>;
    FeLoop l;
    // samples whose Q stays in the L2 (a fifth is left for the states), the
    // groups equal
    const double sample = (double)per * P * sizeof(C);
    const int64_t fit = std::max<int64_t>(1, (int64_t)(0.8 * l2 / sample));
    const int64_t groups = (batch + fit - 1) / fit;
    l.group = (int)((batch + groups - 1) / groups);
    const size_t item = ((size_t)P + (size_t)N * N + FE_ITEM_WARPS * 32 * V) * sizeof(C);
    QSX_CHECK_ARG(item <= 220 * 1024,
                  "qsx_fe_heisenberg_rk4: %zu bytes of column state exceed shared memory", item);
    const int places = (int)std::min<size_t>(FE_ITEMS, 220 * 1024 / item);
    // rows of an item: the fewest rows that one place works through in a stage
    int64_t best = INT64_MAX;
    for (int nt = (P + 32 * V - 1) / (32 * V); nt <= (P + 7) / 8; ++nt) {
      const int tile = ((P + nt - 1) / nt + V - 1) / V * V;
      const int64_t items = (int64_t)l.group * N * ((P + tile - 1) / tile);
      const int64_t all = (int64_t)places * sms, cost = (items + all - 1) / all * tile;
      if (cost < best) {
        best = cost;
        l.tile = tile;
        l.ntile = (P + tile - 1) / tile;
      }
    }
    l.batch = batch;
    l.y0 = (const double2*)y0;
    l.y0_stride = y0_stride;
    l.nsteps = nsteps;
    l.yh = yh;
    l.yl = yl;
    l.acc = acc;
    l.s0 = s0;
    l.s1 = s1;
    l.out = (double2*)out;
    l.status = status;
    l.barrier = barrier;
    const size_t smem = places * item;
    e = cudaMemsetAsync(barrier, 0, 16, s);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int grid = (int)std::min<int64_t>(sms, (int64_t)l.group * N * l.ntile);
    void* args[] = {&p, &l};
    if (e == cudaSuccess)
      e = cudaLaunchCooperativeKernel((const void*)kern, dim3(grid),
                                      dim3(32 * FE_ITEM_WARPS * places), args, smem, s);
    if (e != cudaSuccess) return cuda_status(e, "qsx_fe_heisenberg_rk4");
    QSX_LAUNCH_CHECK("qsx_fe_heisenberg_rk4");
    return QSX_OK;
  };
  return precision == QSX_FP32 ? run(0.0f) : run(0.0);
}

extern "C" int qsx_csr_map_batched(const double* in, int64_t n_in, int64_t batch,
                                   const int* rowptr, const int* cols, const double* vals,
                                   int n_out, double* out, void* stream) {
  QSX_CHECK_ARG(n_in >= 1 && n_out >= 1 && batch >= 0, "qsx_csr_map_batched: bad sizes");
  if (batch == 0) return QSX_OK;
  QSX_CHECK_ARG(in && rowptr && cols && vals && out, "qsx_csr_map_batched: null pointer");
  const int64_t n = batch * n_out;
  csr_map_kernel<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
      (const double2*)in, n_in, batch, rowptr, cols, (const double2*)vals, n_out,
      (double2*)out);
  QSX_LAUNCH_CHECK("qsx_csr_map_batched");
  return QSX_OK;
}
