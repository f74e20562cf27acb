// HEOM time loop for one-exciton blocks in FP32: one cluster of CTAs per
// sample holds the whole hierarchy on chip for all steps (the generator of
// qspectra/dynamics/heom.py:298-443, see heom.cu for its formula).
//
// Per CTA: its nodes' state and two stage inputs in shared memory, the stage
// sums in registers; the low words of the split state, touched once a step,
// stay in the L2.  A stage reads neighbours through distributed shared memory
// and ends in one cluster barrier.  The per-stage kernels it replaces moved
// the state, the stage sums and the inputs through the L2 in every stage and
// read each neighbour there.  Microseconds a stage, per-stage kernels against
// this one, 495 nodes of 8 x 8: 36.4 / 16.0 for 64 samples, 21.8 / 8.2 for 32,
// 7.3 / 5.2 for one.  Against the cluster form of heom.cu (what ran small
// hierarchies): 3.1 / 2.9 for one sample of 120 nodes of 3 x 3, 15.0 / 2.9 for
// 64; 9.2 / 3.0 and 17.7 (per-stage) / 4.3 with 120 nodes of 7 x 7.  Every one
// of 68 sizes measured, 3 to 8 sites, 4 to 495 nodes and 1 to 300 samples, is
// faster here.
//
// A thread owns a 2 x 2 tile of a node's block, the same tile for up to four
// nodes, with its two rows of Hx and two columns of Hy in registers.  With
// number-operator couplings element (a, b) couples to the terms of the sites
// of a and of b alone, so a stage reads one 16-byte record per row and per
// column: the neighbours "up" and "down" that site, the imaginary coefficient
// of the first and the complex one of the second.  Nodes with more terms a
// site than that, and blocks whose states sit on several sites, go through
// their whole term list instead.
//
// Bound: shared memory and its latency (64% of the L1's throughput, an
// instruction in 0.38 of the cycles), about 130 bytes an element and stage: 64
// of them for the commutator's 2 x 2 tile, 32 for the neighbours.  Blocks of 8
// columns are swizzled so that the lanes of a quarter-warp (16-byte accesses)
// or half-warp (8-byte ones) spread over the banks: plain columns lost 57% of
// the wavefronts to conflicts, 28% are left (neighbours at arbitrary places).
#include <algorithm>

#include "cluster_choice.h"
#include "heom_site.cuh"

namespace qsx {

namespace {

constexpr int HS_THREADS = 512;
constexpr int HS_SLOTS = 4;      // nodes a thread
constexpr int HS_MAX_CLUSTER = 8;

struct HsP {
  int n, nnodes, nterms, n_sites, nsave, save_every, nsteps, keep, csize, npcta;
  int64_t batch, H_stride, y0_stride;
  const double *Hx, *Hy, *occx, *occy, *W, *shift;
  const int *nbr, *site;
  const int *order, *place;        // node at each place, and the place of each node
  const double2 *alpha, *beta;
  const double2* y0;
  double2* saves;
  float2* low;          // [batch][nnodes by place][E] low words
  double uc64;          // uc
  float h;
  int* status;
};

// terms of a site as a row or a column sees them: coefficient i s of "up" and c
// of "down", in units of the step's scale uc
struct __align__(16) HsRecord {
  float s, cx, cy, pad;
};
// where "up" and "down" are in the state buffer: addresses in the cluster
struct __align__(8) HsLinks {
  unsigned up, down;
};

template <int NB>
__host__ __device__ constexpr size_t hs_node_bytes(int n_sites) {
  // state and two inputs, row and column records and links, shift and a flag
  return 3 * (size_t)NB * NB * sizeof(float2) +
         (size_t)n_sites * (2 * sizeof(HsRecord) + sizeof(HsLinks)) + 8;
}
template <int NB>
__host__ __device__ constexpr size_t hs_smem_bytes(int npcta, int n_sites) {
  return npcta * hs_node_bytes<NB>(n_sites) + 2 * sizeof(HsRecord) + sizeof(HsLinks);
}

__device__ __forceinline__ unsigned hs_remote(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float2 hs_load2(unsigned addr) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(addr));
  return v;
}
__device__ __forceinline__ float4 hs_load4(unsigned addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(addr));
  return v;
}
__device__ __forceinline__ void hs_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;"
               ::: "memory");
}

// o += i s u + c d
__device__ __forceinline__ void hs_couple(float2& o, const HsRecord& r, float2 u, float2 d) {
  o.x = fmaf(-r.s, u.y, fmaf(r.cx, d.x, fmaf(-r.cy, d.y, o.x)));
  o.y = fmaf(r.s, u.x, fmaf(r.cx, d.y, fmaf(r.cy, d.x, o.y)));
}

// o += -i h (vx + i vy)
__device__ __forceinline__ void hs_rotate(float2& o, float h, float vx, float vy) {
  o.x = fmaf(h, vy, o.x);
  o.y = fmaf(-h, vx, o.y);
}

// Place of element (a, b) in a block.  NB = 8: column b's 64 bytes in half
// (b ^ b / 4) & 1 of its 128-byte line, rows of a pair swapped when b / 2 is
// odd; pairs of rows stay side by side.
template <int NB>
__host__ __device__ constexpr int hs_at(int a, int b) {
  return NB == 8 ? 8 * (b ^ ((b >> 2) & 1)) + (a ^ ((b >> 1) & 1)) : a + NB * b;
}

template <int NB>
__global__ void __launch_bounds__(HS_THREADS, 1) heom_site_kernel(HsP p) {
  constexpr int E = NB * NB, HALF = NB / 2, TPN = HALF * HALF, NPP = HS_THREADS / TPN;
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* sx = (float2*)smraw;       // [3][npcta][E]: state, stage inputs
  HsRecord* srow = (HsRecord*)(sx + 3 * (size_t)p.npcta * E);   // [npcta][n_sites], then none
  HsRecord* scol = srow + (size_t)p.npcta * p.n_sites + 1;
  HsLinks* slink = (HsLinks*)(scol + (size_t)p.npcta * p.n_sites + 1);
  float* sshift = (float*)(slink + (size_t)p.npcta * p.n_sites + 1);   // [npcta]
  int* slist = (int*)(sshift + p.npcta);                     // [npcta] whole term list wanted
  __shared__ int several;   // a state on several sites: every node's whole list
  unsigned rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int64_t smp = blockIdx.x / p.csize;
  const int n = p.n, tid = threadIdx.x;
  const int node0 = (int)rank * p.npcta, nloc = max(0, min(p.nnodes - node0, p.npcta));
  const int q = tid % TPN, g = tid / TPN;
  // tile: rows a0 + {0, 1}, the one stored first being a0 + sw, columns
  // b0 + {0, 1}; NB = 8 deals the columns 0, 4, 2, 6 so that a quarter-warp's
  // two lie in different halves of their lines
  const int qb = q / HALF;
  const int a0 = 2 * (q % HALF), b0 = 2 * (NB == 8 ? (qb >> 1) | ((qb & 1) << 1) : qb);
  const int sw = NB == 8 ? (b0 >> 1) & 1 : 0;
  const int rows[2] = {a0 + sw, a0 + 1 - sw};
  const bool worker = g < NPP;

  const unsigned sx_addr = (unsigned)__cvta_generic_to_shared(sx);

  // ---- tables, all times uc
  if (tid == 0) several = 0;
  __syncthreads();
  // the site of each of this thread's rows and columns: -1 none
  int ra[2], cb[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    ra[i] = cb[i] = -1;
    bool bad = false;
    for (int j = 0; j < p.n_sites; ++j) {
      const double ox = rows[i] < n ? p.occx[j * n + rows[i]] : 0.0;
      const double oy = b0 + i < n ? p.occy[j * n + b0 + i] : 0.0;
      if (ox != 0.0) {
        bad |= ox != 1.0 || ra[i] >= 0;
        ra[i] = j;
      }
      if (oy != 0.0) {
        bad |= oy != 1.0 || cb[i] >= 0;
        cb[i] = j;
      }
    }
    if (bad) several = 1;
  }
  __syncthreads();
  for (int i = tid; i < p.npcta; i += HS_THREADS) {
    sshift[i] = i < nloc ? (float)(p.uc64 * p.shift[p.order[node0 + i]]) : 0.f;
    slist[i] = several;
  }
  __syncthreads();
  const int nrec = p.npcta * p.n_sites;
  for (int i = tid; i <= nrec; i += HS_THREADS) {
    const int l = i / p.n_sites, j = i % p.n_sites;
    // a missing link reads a node of this CTA, times 0: its own, and the record
    // of "no site" the first one, as the slots past nloc are never written
    const unsigned self =
        hs_remote(sx_addr + (unsigned)((l < nloc ? l : 0) * E * sizeof(float2)), rank);
    HsRecord r = {0.f, 0.f, 0.f, 0.f}, c = r;
    HsLinks k = {self, self};
    if (i < nrec && l < nloc && !several) {
      int up = 0, down = 0;
      const int64_t t0 = (int64_t)p.order[node0 + l] * p.nterms;
      for (int t = 0; t < p.nterms; ++t) {
        if (p.nbr[t0 + t] < 0 || p.site[t0 + t] != j) continue;
        const int m = p.place[p.nbr[t0 + t]];
        const double2 al = p.alpha[t0 + t], be = p.beta[t0 + t];
        const unsigned at = hs_remote(
            sx_addr + (unsigned)(m % p.npcta * E * sizeof(float2)), (unsigned)(m / p.npcta));
        if (al.x == 0.0 && be.x == 0.0 && !up) {
          up = 1;
          k.up = at;
          r.s = (float)(p.uc64 * al.y);
          c.s = (float)(p.uc64 * be.y);
        } else if (!down) {
          down = 1;
          k.down = at;
          r.cx = (float)(p.uc64 * al.x);
          r.cy = (float)(p.uc64 * al.y);
          c.cx = (float)(p.uc64 * be.x);
          c.cy = (float)(p.uc64 * be.y);
        } else {
          slist[l] = 1;
        }
      }
    }
    srow[i] = r;
    scol[i] = c;
    slink[i] = k;
  }
  const double* hx = p.Hx + smp * p.H_stride;
  const double* hy = p.Hy + smp * p.H_stride;
  float h0[NB], h1[NB], k0[NB], k1[NB], wt[4];
#pragma unroll
  for (int c = 0; c < NB; ++c) {
    const bool in = c < n;
    // the row of Hx in the order in which the column is stored
    const int cs = c ^ sw;
    h0[c] = cs < n && rows[0] < n ? (float)(p.uc64 * hx[rows[0] * n + cs]) : 0.f;
    h1[c] = cs < n && rows[1] < n ? (float)(p.uc64 * hx[rows[1] * n + cs]) : 0.f;
    k0[c] = in && b0 < n ? -(float)(p.uc64 * hy[c * n + b0]) : 0.f;
    k1[c] = in && b0 + 1 < n ? -(float)(p.uc64 * hy[c * n + b0 + 1]) : 0.f;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int a = rows[i & 1], b = b0 + (i >> 1);
    wt[i] = p.W && a < n && b < n ? (float)(p.uc64 * p.W[a + n * b]) : 0.f;
  }
  // ---- state: element i of a tile is (rows[i & 1], b0 + (i >> 1)), at place
  // t0 (first two) and t1 (last two) of the block
  const int t0 = hs_at<NB>(rows[0], b0), t1 = hs_at<NB>(rows[0], b0 + 1);
  const int col0 = t0 - a0, col1 = t1 - a0;   // first element of the columns
  float2 acc[HS_SLOTS][4];
  const double2* y0 = p.y0 + smp * p.y0_stride;
  float2* low = p.low + ((size_t)smp * p.nnodes + node0) * E;
#pragma unroll
  for (int u = 0; u < HS_SLOTS; ++u) {
    const int l = g + u * NPP;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int a = rows[i & 1], b = b0 + (i >> 1);
      acc[u][i] = make_float2(0.f, 0.f);
      if (worker && l < nloc) {
        float2 hi = make_float2(0.f, 0.f), lo = hi;
        if (a < n && b < n) {
          const double2 v = y0[(int64_t)p.order[node0 + l] * n * n + a + n * b];
          hi = make_float2((float)v.x, (float)v.y);
          lo = make_float2((float)(v.x - (double)hi.x), (float)(v.y - (double)hi.y));
        }
        const int e = l * E + hs_at<NB>(a, b);
        sx[e] = hi;
        low[e] = lo;
      }
    }
  }
  auto save = [&](int k) {   // this thread's own elements
#pragma unroll 1
    for (int u = 0; u < HS_SLOTS; ++u) {
      const int l = g + u * NPP;
      if (!worker || l >= nloc) continue;
      const int node = p.order[node0 + l];
      if (node >= p.keep) continue;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int a = rows[i & 1], b = b0 + (i >> 1);
        if (a >= n || b >= n) continue;
        const int e = l * E + hs_at<NB>(a, b);
        const float2 hi = sx[e], lo = low[e];
        const double2 v = make_double2((double)hi.x + (double)lo.x, (double)hi.y + (double)lo.y);
        if (p.status && !finite2(v)) atomicOr(p.status, QSX_ERR_NONFINITE);
        p.saves[((smp * p.nsave + k) * (int64_t)p.keep + node) * n * n + a + n * b] = v;
      }
    }
  };
  save(0);
  const float s6 = p.h / 6.f;
  const unsigned buf_bytes = (unsigned)(p.npcta * E * sizeof(float2));
  for (int step = 0; step < p.nsteps; ++step) {
#pragma unroll 1
    for (int stage = 0; stage < 4; ++stage) {
      // state -> input 1 -> input 2 -> input 1 -> state
      const int in = stage == 0 ? 0 : 1 + ((stage & 1) ^ 1), to = stage == 3 ? 0 : 1 + (stage & 1);
      hs_cluster_sync();           // this stage's input is complete cluster-wide
      const float2* xin = sx + (size_t)in * p.npcta * E;
      float2* xout = sx + (size_t)to * p.npcta * E;
      const unsigned shift_buf = in * buf_bytes;
      const float cnext = stage == 2 ? p.h : 0.5f * p.h;
      const float wg = (stage == 0 || stage == 3) ? 1.f : 2.f;
#pragma unroll
      for (int u = 0; u < HS_SLOTS; ++u) {
        const int l = g + u * NPP;
        if (!worker || l >= nloc) continue;
        const unsigned o00 = shift_buf + (unsigned)(t0 * sizeof(float2));
        const unsigned o01 = shift_buf + (unsigned)(t1 * sizeof(float2));
        const float2* x = xin + l * E;
        const bool whole = slist[l] != 0;
        float2 o[4];
        // the rows' neighbours are in flight during Hx x, the columns' during x Hy
        int i0 = ra[0] < 0 ? nrec : l * p.n_sites + ra[0];
        int i1 = ra[1] < 0 ? nrec : l * p.n_sites + ra[1];
        HsRecord r0 = srow[i0], r1 = srow[i1];
        HsLinks n0 = slink[i0], n1 = slink[i1];
        {
          // (rows[1]'s element is the other one of the pair)
          const float2 ru00 = hs_load2(n0.up + o00), ru01 = hs_load2(n0.up + o01);
          const float2 rd00 = hs_load2(n0.down + o00), rd01 = hs_load2(n0.down + o01);
          const float2 ru10 = hs_load2(n1.up + o00 + 8), ru11 = hs_load2(n1.up + o01 + 8);
          const float2 rd10 = hs_load2(n1.down + o00 + 8), rd11 = hs_load2(n1.down + o01 + 8);
          // -(shift + W) x - i Hx x
          const float4 x0 = *reinterpret_cast<const float4*>(x + t0);
          const float4 x1 = *reinterpret_cast<const float4*>(x + t1);
          const float sh = -sshift[l];
          o[0] = make_float2((sh - wt[0]) * x0.x, (sh - wt[0]) * x0.y);
          o[1] = make_float2((sh - wt[1]) * x0.z, (sh - wt[1]) * x0.w);
          o[2] = make_float2((sh - wt[2]) * x1.x, (sh - wt[2]) * x1.y);
          o[3] = make_float2((sh - wt[3]) * x1.z, (sh - wt[3]) * x1.w);
#pragma unroll
          for (int c = 0; c < NB; c += 2) {
            const float4 p0 = *reinterpret_cast<const float4*>(x + col0 + c);
            const float4 p1 = *reinterpret_cast<const float4*>(x + col1 + c);
            hs_rotate(o[0], h0[c], p0.x, p0.y);
            hs_rotate(o[0], h0[c + 1], p0.z, p0.w);
            hs_rotate(o[1], h1[c], p0.x, p0.y);
            hs_rotate(o[1], h1[c + 1], p0.z, p0.w);
            hs_rotate(o[2], h0[c], p1.x, p1.y);
            hs_rotate(o[2], h0[c + 1], p1.z, p1.w);
            hs_rotate(o[3], h1[c], p1.x, p1.y);
            hs_rotate(o[3], h1[c + 1], p1.z, p1.w);
          }
          if (!whole) {
            hs_couple(o[0], r0, ru00, rd00);
            hs_couple(o[2], r0, ru01, rd01);
            hs_couple(o[1], r1, ru10, rd10);
            hs_couple(o[3], r1, ru11, rd11);
          }
        }
        i0 = cb[0] < 0 ? nrec : l * p.n_sites + cb[0];
        i1 = cb[1] < 0 ? nrec : l * p.n_sites + cb[1];
        r0 = scol[i0];
        r1 = scol[i1];
        n0 = slink[i0];
        n1 = slink[i1];
        {
          const float4 u0 = hs_load4(n0.up + o00), d0 = hs_load4(n0.down + o00);
          const float4 u1 = hs_load4(n1.up + o01), d1 = hs_load4(n1.down + o01);
          // + i x Hy (k = -Hy), by row: which of a column's pair is row a0 is
          // known for each c, which one is rows[0] only here
          float2 t[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) t[i] = make_float2(0.f, 0.f);
#pragma unroll
          for (int c = 0; c < NB; ++c) {
            const bool swapped = NB == 8 && ((c >> 1) & 1);
            const float4 v = *reinterpret_cast<const float4*>(
                x + a0 + (NB == 8 ? 8 * (c ^ ((c >> 2) & 1)) : NB * c));
            const float2 lo = swapped ? make_float2(v.z, v.w) : make_float2(v.x, v.y);
            const float2 up = swapped ? make_float2(v.x, v.y) : make_float2(v.z, v.w);
            hs_rotate(t[0], k0[c], lo.x, lo.y);
            hs_rotate(t[1], k0[c], up.x, up.y);
            hs_rotate(t[2], k1[c], lo.x, lo.y);
            hs_rotate(t[3], k1[c], up.x, up.y);
          }
          o[0] = cadd2(o[0], sw ? t[1] : t[0]);
          o[1] = cadd2(o[1], sw ? t[0] : t[1]);
          o[2] = cadd2(o[2], sw ? t[3] : t[2]);
          o[3] = cadd2(o[3], sw ? t[2] : t[3]);
          if (!whole) {
            hs_couple(o[0], r0, make_float2(u0.x, u0.y), make_float2(d0.x, d0.y));
            hs_couple(o[1], r0, make_float2(u0.z, u0.w), make_float2(d0.z, d0.w));
            hs_couple(o[2], r1, make_float2(u1.x, u1.y), make_float2(d1.x, d1.y));
            hs_couple(o[3], r1, make_float2(u1.z, u1.w), make_float2(d1.z, d1.w));
          }
        }
        if (whole) {
          const int64_t list = (int64_t)p.order[node0 + l] * p.nterms;
#pragma unroll 1
          for (int t = 0; t < p.nterms; ++t) {
            const int j = p.site[list + t];
            if (p.nbr[list + t] < 0) continue;
            const int m = p.place[p.nbr[list + t]];
            const double2 al = p.alpha[list + t], be = p.beta[list + t];
            const unsigned base = hs_remote(
                sx_addr + (unsigned)(m % p.npcta * E * sizeof(float2)), (unsigned)(m / p.npcta));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const int a = rows[i & 1], b = b0 + (i >> 1);
              const float oa = a < n ? (float)p.occx[j * n + a] : 0.f;
              const float ob2 = b < n ? (float)p.occy[j * n + b] : 0.f;
              const float fr = (float)(p.uc64 * al.x) * oa + (float)(p.uc64 * be.x) * ob2;
              const float fi = (float)(p.uc64 * al.y) * oa + (float)(p.uc64 * be.y) * ob2;
              const float2 v = hs_load2(base + (i >> 1 ? o01 : o00) + (i & 1 ? 8u : 0u));
              o[i].x = fmaf(fr, v.x, fmaf(-fi, v.y, o[i].x));
              o[i].y = fmaf(fr, v.y, fmaf(fi, v.x, o[i].y));
            }
          }
        }
        const float4 y0v = *reinterpret_cast<const float4*>(sx + l * E + t0);
        const float4 y1v = *reinterpret_cast<const float4*>(sx + l * E + t1);
        float2 y[4] = {make_float2(y0v.x, y0v.y), make_float2(y0v.z, y0v.w),
                       make_float2(y1v.x, y1v.y), make_float2(y1v.z, y1v.w)};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float2 d = o[i];
          acc[u][i] = stage == 0 ? d : make_float2(fmaf(wg, d.x, acc[u][i].x),
                                                   fmaf(wg, d.y, acc[u][i].y));
          if (stage < 3) y[i] = make_float2(fmaf(cnext, d.x, y[i].x), fmaf(cnext, d.y, y[i].y));
        }
        if (stage == 3) {
          float4* lo = reinterpret_cast<float4*>(low + l * E);
          float4 w[2] = {lo[t0 / 2], lo[t1 / 2]};
          float* wl = reinterpret_cast<float*>(w);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            dd_add(y[i].x, wl[2 * i], s6 * acc[u][i].x);
            dd_add(y[i].y, wl[2 * i + 1], s6 * acc[u][i].y);
          }
          lo[t0 / 2] = w[0];
          lo[t1 / 2] = w[1];
        }
        *reinterpret_cast<float4*>(xout + l * E + t0) = make_float4(y[0].x, y[0].y, y[1].x, y[1].y);
        *reinterpret_cast<float4*>(xout + l * E + t1) = make_float4(y[2].x, y[2].y, y[3].x, y[3].y);
      }
    }
    if ((step + 1) % p.save_every == 0) save((step + 1) / p.save_every);
  }
  hs_cluster_sync();   // peers may still read this CTA's buffers
}

// The order in which nodes are dealt to the CTAs of a cluster: by their
// occupation numbers, first site first, so that the links of the last sites
// stay inside a CTA (30% of the links of 495 nodes of 8 sites cross between
// four CTAs, 79% in the order of the table, which goes by level).  A node's
// numbers follow from the first path that reaches it: node 0 has none, and a
// link of site j from a node of one level to an unreached one adds one.  Only
// the speed depends on them.  One CTA, once a call.
__global__ void __launch_bounds__(1024)
    hs_order_kernel(const int* __restrict__ nbr, const int* __restrict__ site, int nnodes,
                    int nterms, int* __restrict__ order, int* __restrict__ place) {
  extern __shared__ unsigned long long key[];   // [nnodes], then levels
  int* level = (int*)(key + nnodes);
  for (int i = threadIdx.x; i < nnodes; i += blockDim.x) {
    key[i] = i == 0 ? 0ull : ~0ull;
    level[i] = i == 0 ? 0 : -1;
  }
  for (int depth = 0; depth < 64; ++depth) {
    int found = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < nnodes; i += blockDim.x) {
      if (level[i] != depth) continue;
      for (int t = 0; t < nterms; ++t) {
        const int m = nbr[(int64_t)i * nterms + t], j = site[(int64_t)i * nterms + t];
        if (m < 0 || m >= nnodes || atomicCAS(level + m, -1, depth + 1) != -1) continue;
        key[m] = key[i] + (1ull << (8 * (7 - min(max(j, 0), 7))));
        found = 1;
      }
    }
    if (!__syncthreads_or(found)) break;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < nnodes; i += blockDim.x) {
    const unsigned long long k = key[i];
    int r = 0;
    for (int m = 0; m < nnodes; ++m) r += key[m] < k || (key[m] == k && m < i);
    order[r] = i;
    place[i] = r;
  }
}

template <int NB>
bool hs_launch(HsP p, cudaStream_t s, int* st) {
  constexpr int TPN = (NB / 2) * (NB / 2), NPP = HS_THREADS / TPN;
  const size_t most = 226 * 1024;
  cudaError_t e = cudaSuccess;
  // as few CTAs as hold the hierarchy; more of them, down to a pass of nodes
  // each, while there are SMs to spare
  auto fits = [&](int c) {
    const int np = (p.nnodes + c - 1) / c;
    return np <= HS_SLOTS * NPP && hs_smem_bytes<NB>(np, p.n_sites) <= most;
  };
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute at[1];
  cfg.blockDim = dim3(HS_THREADS);
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  auto configure = [&](int size) {   // how many clusters of this size run at once
    p.csize = size;
    p.npcta = (p.nnodes + size - 1) / size;
    cfg.gridDim = dim3((unsigned)(p.batch * size));
    cfg.dynamicSmemBytes = hs_smem_bytes<NB>(p.npcta, p.n_sites);
    at[0].val.clusterDim.x = size;
    int clusters = 0;
    e = cudaFuncSetAttribute(heom_site_kernel<NB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)cfg.dynamicSmemBytes);
    if (e == cudaSuccess)
      e = cudaOccupancyMaxActiveClusters(&clusters, heom_site_kernel<NB>, &cfg);
    if (e != cudaSuccess) {
      cudaGetLastError();   // the other forms of the loop still run
      e = cudaSuccess;
      clusters = 0;
    }
    return clusters;
  };
  const int c = choose_cluster(p.batch, HS_MAX_CLUSTER, fits,
                               [&](int size) { return p.nnodes > size * NPP; }, configure);
  if (!c || configure(c) < 1) return false;
  const size_t osmem = (size_t)p.nnodes * 12;
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(hs_order_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)osmem);
  if (e == cudaSuccess) {
    hs_order_kernel<<<1, 1024, osmem, s>>>(p.nbr, p.site, p.nnodes, p.nterms, (int*)p.order,
                                           (int*)p.place);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, heom_site_kernel<NB>, p);
  *st = e == cudaSuccess ? QSX_OK : cuda_status(e, "qsx_heom_rk4 (site form)");
  return true;
}

}  // namespace

bool heom_site_run(const qsx_heom_args* a, double2* saves, float2* low, int* order,
                   cudaStream_t s, int* st) {
  if (a->precision != QSX_FP32 || a->nx != a->ny || a->nx < 3 || a->nx > 8 || a->gamma ||
      a->nterms < 1 || a->nterms > 2 * a->n_sites || a->nx > a->n_sites)
    return false;
  HsP p;
  p.n = a->nx;
  p.nnodes = a->nnodes;
  p.nterms = a->nterms;
  p.n_sites = a->n_sites;
  p.nsave = a->nsteps / a->save_every + 1;
  p.save_every = a->save_every;
  p.nsteps = a->nsteps;
  p.keep = a->save_nodes;
  p.batch = a->batch;
  p.H_stride = a->H_stride ? (int64_t)a->nx * a->nx : 0;
  p.y0_stride = a->y0_stride ? (int64_t)a->nnodes * a->nx * a->ny : 0;
  p.Hx = a->Hx;
  p.Hy = a->Hy;
  p.occx = a->occx;
  p.occy = a->occy;
  p.W = a->W;
  p.shift = a->shift;
  p.nbr = a->nbr;
  p.site = a->site;
  p.alpha = (const double2*)a->alpha;
  p.beta = (const double2*)a->beta;
  p.y0 = (const double2*)a->y0;
  p.saves = saves;
  p.low = low;
  p.order = order;
  p.place = order + a->nnodes;
  p.uc64 = a->unit_convert;
  p.h = (float)a->h;
  p.status = a->status;
  if (a->nx <= 4) return hs_launch<4>(p, s, st);
  return a->nx <= 6 ? hs_launch<6>(p, s, st) : hs_launch<8>(p, s, st);
}

}  // namespace qsx
