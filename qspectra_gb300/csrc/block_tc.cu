// Real K-step blocked matrices on the 5th-generation tensor cores (tcgen05).
//
// Same output as block_matrix_real_kernel (qsx_rk4_block_matrix_real_batched):
// per sample, rows 0..m-1 = D_K = P^K - I and the selected rows R_k of
// D_k = P^k - I (k = 1..K-1), for the FP32 real (Hermitian) form, m <= 64.
//
// Phase j multiplies the stacked operand A = [D_{2^j} ; R_1..R_{2^j}] by
// B = D_{2^j} in one M = 128, N = NP, K = KP tcgen05.mma chain: the square
// and the row product share B.  D rows sit in A rows 0..31 and 64..95, R rows
// in 32..63 and 96..127, so that each of the four TMEM lane quarters (one per
// SM sub-partition) carries half square work and half row work.  FP32
// accuracy comes from 3xTF32: A = A_hi + A_lo, B = B_hi + B_lo (each rounded
// to TF32), A B ~ A_hi B_hi + A_hi B_lo + A_lo B_hi, 3 KP / 8 MMAs into one
// FP32 accumulator in tensor memory.  The epilogue (eight warps: lane quarter
// = warp % 4, column half = warp / 4; tcgen05.ld) forms
// D_{2^{j+1}} = 2 D + D D and R_{i + 2^j} = R_i + R_{2^j} + R_i D_{2^j} and
// the next operands.  D_K for K = 2^J + 1 is a final chain D_1 D_{2^J} (powers
// of P commute), for K = 2^J the last square.
//
// A is in tensor memory: a D row stays in its own lane (tcgen05.st), a new R
// row passes through the R rows' buffer in shared memory to the lane of its A
// row, behind a barrier of the R warps alone.  B is in shared memory.  With A
// there too, written and read by every MMA, a phase moved 250 KB through it and
// a CTA took 118 KB at K = 17, so that one ran on an SM; now two do from 70 KB
// each.  Bound: the latency of a phase, about 1700 cycles of MMAs and 2000 of
// the D warps' epilogue, two CTAs under each other.  16384 samples of m = 49,
// seven rows: K = 9 740 us before and 490 here, K = 17 1300 and 498.
//
// The kernel is persistent: each CTA loops over samples, keeps its tensor
// memory, barrier and zero padding, and prefetches the next sample's D with
// cp.async while the current one is in the product chain.  For odd m, whose
// rows need no padding against bank conflicts, D_K and the R rows lie in shared
// memory as they do in the output and leave by one bulk copy.
//
// Layout of B (SWIZZLE_NONE, K-major, B^T row-major): 8-row x 16-byte core
// matrices, element (n, k) at (n / 8) * SBO + (k / 4) * LBO + (n % 8) * 16 +
// (k % 4) * 4 bytes.  LBO = 144 bytes between K-adjacent core matrices: the 32
// lanes of a warp hold 32 consecutive k of a column n and meet 32 banks when
// they write it (128 bytes would put them on four).
//
// Every wait on the MMA completion barrier is bounded; on a timeout the CTA
// records QSX_ERR_CUDA in the status word, stops issuing work, waits once more
// (bounded) for its MMA chain, and still frees its tensor memory.
#include <stdint.h>

#include <algorithm>
#include <type_traits>

#include "qsx_common.cuh"
#include "qsx_tc.cuh"

namespace qsx {

namespace tc {

// One sample's D (m x m contiguous floats in global memory) into the staging
// buffer: the enclosing 16-byte-aligned range keeps its alignment, so the
// sample starts at float offset (address % 16) / 4 of sd; the interior moves
// in 16-byte cp.async chunks, the ragged head and tail element by element.
// Returns that offset.
__device__ __forceinline__ int prefetch_sample(const float* d, float* sd, int mm, int tid,
                                               int nthreads) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(d);
  const int shift = (int)((a & 15) >> 2);
  const int head = (4 - shift) & 3;                         // elements before the first chunk
  const int nchunk = mm > head ? (mm - head) >> 2 : 0;
  const int tail0 = head + 4 * nchunk;
  const uint32_t base = (uint32_t)__cvta_generic_to_shared(sd + shift);
  for (int c = tid; c < nchunk; c += nthreads) {
    const int e = head + 4 * c;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(base + 4u * e), "l"(d + e)
                 : "memory");
  }
  const int nedge = min(head, mm) + (mm - tail0 > 0 ? mm - tail0 : 0);
  for (int t = tid; t < nedge; t += nthreads) {
    const int e = t < min(head, mm) ? t : tail0 + (t - min(head, mm));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(base + 4u * e), "l"(d + e)
                 : "memory");
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  return shift;
}

__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

}  // namespace tc

constexpr uint32_t BT_LBO = 144;

// Shapes for m in (KP - 8, KP].  The CTA has four warps per 32 columns, warp w
// reading TMEM lane quarter w % 4 and columns 32 (w / 4) ...
template <int KP>
struct BlockTc {
  static constexpr int HALVES = KP > 32 ? 2 : 1, NT = 128 * HALVES;
  static constexpr int W = 32 * HALVES;                   // columns of a tensor-memory plane
  static constexpr uint32_t TMEM = KP > 32 ? 256 : 128;   // three planes, rounded up
  static constexpr int N0 = KP < 32 ? KP : 32, N1 = KP > 32 ? KP - 32 : 8;
  static constexpr int NP = (KP + 15) & ~15;
  static constexpr uint32_t SBO = KP / 4 * BT_LBO, PB = NP / 8 * SBO;
  static size_t smem(int m, int nr) {
    // B^T hi/lo, the staging copy of the sample's D (m*m + 4 FP32,
    // contiguous), D_K and the R rows ((m + nr) x SP FP32, SP = m | 1), the
    // mbarrier and the tensor-memory address
    const size_t sp = m | 1;
    return ((2 * (size_t)PB + ((((size_t)m * m + 4 + 3) & ~(size_t)3) + (m + nr) * sp) * 4 + 15) &
            ~(size_t)15) + 16;
  }
};

template <int KP>
__global__ void __launch_bounds__(BlockTc<KP>::NT, 2)
    block_matrix_tc_kernel(const float* __restrict__ D, int m, int K, int J,
                           const int* __restrict__ sel, int nsel, float* __restrict__ out,
                           int* status, int64_t batch) {
  using namespace tc;
  using S = BlockTc<KP>;
  constexpr int NT = S::NT, NW = NT / 32, W = S::W;
  constexpr uint32_t PB = S::PB;
  extern __shared__ __align__(128) unsigned char smraw[];
  const int sp = m | 1;
  unsigned char* b_hi = smraw;
  unsigned char* b_lo = b_hi + PB;
  const int mm = m * m;
  const int nr = nsel * (K - 1);
  float* Sd = reinterpret_cast<float*>(b_lo + PB);   // [mm + 4], 16-byte aligned
  float* stg = Sd + ((mm + 4 + 3) & ~3);             // [m][sp]: D_K
  float* Rp = stg + m * sp;                          // [(K-1) nsel][sp]
  const uint32_t off_mbar =
      (2 * PB + (uint32_t)(((mm + 4 + 3) & ~3) + (m + nr) * sp) * 4 + 15) & ~15u;
  uint64_t* mbar_p = reinterpret_cast<uint64_t*>(smraw + off_mbar);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(mbar_p + 1);
  __shared__ int s_abort;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int lg = warp & 3;
  const bool dwarp = (lg & 1) == 0;           // D rows; otherwise R rows
  const int r = 32 * (lg >> 1) + lane;        // D row, or R row index
  const int myq = r % nsel;
  int mysel = 0;
  if (!dwarp && r < nsel) {
    mysel = sel[r];
    mysel = (mysel >= 0 && mysel < m) ? mysel : 0;
  }
  const int rows_out = m + nr;
  const int64_t ostride = ((int64_t)rows_out * m + 3) & ~(int64_t)3;
  const uint32_t mbar = (uint32_t)__cvta_generic_to_shared(mbar_p);
  const uint64_t db_hi = smem_desc((uint32_t)__cvta_generic_to_shared(b_hi), S::SBO, BT_LBO);
  const uint64_t db_lo = smem_desc((uint32_t)__cvta_generic_to_shared(b_lo), S::SBO, BT_LBO);
  const uint32_t idesc = make_idesc(S::NP);
  const bool pow2 = (K & (K - 1)) == 0;

  // zero padding of the operand planes (kept zero across samples)
  for (uint32_t e = tid; e < 2 * PB / 16; e += NT)
    reinterpret_cast<uint4*>(smraw)[e] = make_uint4(0, 0, 0, 0);
  if (tid == 0) {
    s_abort = 0;
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     (uint32_t)__cvta_generic_to_shared(tmem_slot)),
                 "r"(S::TMEM)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;
  const bool bulk = (m & 1) && (reinterpret_cast<uintptr_t>(out) & 15) == 0;

  // f(N, C0): this warp's N columns from column C0, both known to the compiler
  auto columns = [&](auto f) {
    if (S::HALVES == 1 || warp < 4)
      f(std::integral_constant<int, S::N0>{}, std::integral_constant<int, 0>{});
    else
      f(std::integral_constant<int, S::N1>{}, std::integral_constant<int, 32>{});
  };
  // this thread's lane in the accumulator; A's planes follow W and 2 W columns on
  const uint32_t taddr = tmem + ((uint32_t)(32 * lg) << 16);
  // B^T column k = r: element (n, r) at n's offset from here
  const uint32_t boff = (uint32_t)(r >> 2) * BT_LBO + (uint32_t)(r & 3) * 4;
  // operands from this thread's columns: A row = lane (a), B row k = r (b)
  auto operands = [&](auto n_, auto c0_, auto& v, bool a, bool b) {
    constexpr int N = n_.value, C0 = c0_.value;
    float hi[N], lo[N];
#pragma unroll
    for (int c = 0; c < N; ++c) {
      hi[c] = tf32_round(v[c]);
      lo[c] = tf32_round(v[c] - hi[c]);
    }
    if (a) {
      tmem_store_cols(taddr + W + C0, hi);
      tmem_store_cols(taddr + 2 * W + C0, lo);
    }
    if (b && r < KP) {
#pragma unroll
      for (int c = 0; c < N; ++c) {
        const uint32_t off = (uint32_t)((C0 + c) >> 3) * S::SBO + (uint32_t)((C0 + c) & 7) * 16;
        *reinterpret_cast<float*>(b_hi + boff + off) = hi[c];
        *reinterpret_cast<float*>(b_lo + boff + off) = lo[c];
      }
    }
    if (a) tmem_store_wait();
  };
  // one product chain, waited for; false when it did not come
  uint32_t parity = 0;
  auto product = [&]() {
    if (tid == 0) {
      issue_product_ts<KP / 8>(tmem, tmem + W, tmem + 2 * W, db_hi, db_lo, idesc, mbar, BT_LBO);
      if (!wait_parity(mbar, parity)) {
        if (status) atomicOr(status, QSX_ERR_CUDA);
        s_abort = 1;
      }
    }
    __syncthreads();  // the other threads wait here, off the issue slots
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (s_abort) return false;
    parity ^= 1;
    return true;
  };
  // operands written: visible to the tensor cores, every thread there
  auto published = [&]() {
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    __syncthreads();
  };

  int64_t s = blockIdx.x;
  int shift = 0, next_shift = 0;
  if (s < batch) next_shift = prefetch_sample(D + s * mm, Sd, mm, tid, NT);
  for (; s < batch; s += gridDim.x) {
    const int64_t next = s + gridDim.x;
    shift = next_shift;
    const float* sd = Sd + shift;   // this sample's D, row-major, stride m
    cp_async_wait_all();
    __syncthreads();
    // D warps: this thread's part of D_{2^j}, zero outside m x m.  R warps: R_i +
    // R_{2^j} of the row this thread forms next, fetched under the product
    float dr[32];
    columns([&](auto n_, auto c0_) {
      constexpr int N = n_.value, C0 = c0_.value;
      const bool act = r < (dwarp ? m : nsel);
      const float* src = sd + (dwarp ? r : mysel) * m + C0;
      float v[N];
#pragma unroll
      for (int c = 0; c < N; ++c)
        v[c] = (act && (C0 + c < KP - 7 || C0 + c < m)) ? src[c] : 0.f;
#pragma unroll
      for (int c = 0; c < N; ++c) dr[c] = v[c];
      operands(n_, c0_, v, true, dwarp);
    });
    // the previous sample's rows have left shared memory
    if (tid == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    published();
    if (!dwarp && r < nsel)
      columns([&](auto n_, auto c0_) {
        constexpr int N = n_.value, C0 = c0_.value;
#pragma unroll
        for (int c = 0; c < N; ++c) {
          if (C0 + c < KP - 7 || C0 + c < m) Rp[r * sp + C0 + c] = dr[c];
          dr[c] += dr[c];
        }
      });
    if (pow2 && next < batch) next_shift = prefetch_sample(D + next * mm, Sd, mm, tid, NT);

    int have = 1;
    for (int j = 0;; ++j) {
      const bool square = j < J;
      const int add = have < K - 1 ? min(1 << j, K - 1 - have) : 0;
      const bool last = !(j + 1 < J || have + add < K - 1);
      if (!product()) break;
      columns([&](auto n_, auto c0_) {
        constexpr int N = n_.value, C0 = c0_.value;
        float acc[N];
        tmem_load_cols(taddr + C0, acc);
        if (dwarp) {
          if (square) {
#pragma unroll
            for (int c = 0; c < N; ++c) dr[c] = fmaf(2.f, dr[c], acc[c]);
            if (!last) {
              operands(n_, c0_, dr, true, true);
            } else if (!pow2) {
              // operands of the final chain D_1 D_{2^J}; dr becomes D_{2^J} + D_1
              operands(n_, c0_, dr, false, true);
              const float* src = sd + r * m + C0;
#pragma unroll
              for (int c = 0; c < N; ++c)
                acc[c] = (r < m && (C0 + c < KP - 7 || C0 + c < m)) ? src[c] : 0.f;
              operands(n_, c0_, acc, true, false);
#pragma unroll
              for (int c = 0; c < N; ++c) dr[c] += acc[c];
            }
          }
        } else {
          if (r < add * nsel) {
            // new row R_{have + 1 + r / nsel}
            float* dst = Rp + (have * nsel + r) * sp + C0;
#pragma unroll
            for (int c = 0; c < N; ++c)
              if (C0 + c < KP - 7 || C0 + c < m) dst[c] = dr[c] + acc[c];
          }
          if (!last) {
            // every new row is in shared memory: the lanes take their A rows,
            // in warps that have new ones
            asm volatile("bar.sync 1, %0;" ::"r"(NT / 2) : "memory");
            if (32 * (lg >> 1) < (have + add) * nsel && 32 * (lg >> 1) + 32 > have * nsel) {
              const bool act = r < (have + add) * nsel;
              const float* src = Rp + r * sp + C0;
#pragma unroll
              for (int c = 0; c < N; ++c)
                acc[c] = (act && (C0 + c < KP - 7 || C0 + c < m)) ? src[c] : 0.f;
              operands(n_, c0_, acc, true, false);
            }
          }
        }
      });
      have += add;
      published();
      if (last) break;
      if (!dwarp && r < min(2 << j, K - 1 - have) * nsel)
        columns([&](auto n_, auto c0_) {
          constexpr int N = n_.value, C0 = c0_.value;
          const float* ri = Rp + r * sp + C0;                                 // R_{1 + r / nsel}
          const float* rj = Rp + (((2 << j) - 1) * nsel + myq) * sp + C0;     // R_{2^{j + 1}}
#pragma unroll
          for (int c = 0; c < N; ++c)
            dr[c] = (C0 + c < KP - 7 || C0 + c < m) ? ri[c] + rj[c] : 0.f;
        });
    }
    if (s_abort) break;
    if (!pow2) {
      if (next < batch) next_shift = prefetch_sample(D + next * mm, Sd, mm, tid, NT);
      if (!product()) break;
      columns([&](auto n_, auto c0_) {
        constexpr int N = n_.value, C0 = c0_.value;
        float acc[N];
        tmem_load_cols(taddr + C0, acc);
#pragma unroll
        for (int c = 0; c < N; ++c) dr[c] += acc[c];
      });
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    }
    if (dwarp && r < m)
      columns([&](auto n_, auto c0_) {
        constexpr int N = n_.value, C0 = c0_.value;
#pragma unroll
        for (int c = 0; c < N; ++c)
          if (C0 + c < KP - 7 || C0 + c < m) stg[r * sp + C0 + c] = dr[c];
      });
    float* o = out + s * ostride;
    if (bulk) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncthreads();
      if (tid == 0) {
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(o),
                     "r"((uint32_t)__cvta_generic_to_shared(stg)), "r"((uint32_t)ostride * 4u)
                     : "memory");
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
      continue;   // the rows may be written again once the copy has read them
    }
    __syncthreads();
#pragma unroll 4
    for (int row = warp; row < rows_out; row += NW) {
      const float* src = stg + row * sp;
      const float v0 = lane < m ? src[lane] : 0.f;
      const float v1 = lane + 32 < m ? src[lane + 32] : 0.f;
      if (lane < m) o[row * m + lane] = v0;
      if (lane + 32 < m) o[row * m + lane + 32] = v1;
    }
    // the next iteration's first barrier orders these reads before new writes
  }
  cp_async_wait_all();
  if (tid == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  if (s_abort && tid == 0) wait_parity(mbar, parity);  // let an unfinished chain drain
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(S::TMEM)
                 : "memory");
}

template <int KP>
static int block_tc_launch(const float* D, int m, int64_t batch, int K, int J, const int* select,
                           int nselect, float* out, int32_t* status, cudaStream_t st) {
  using S = BlockTc<KP>;
  const size_t smem = S::smem(m, nselect * (K - 1));
  auto kern = block_matrix_tc_kernel<KP>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout,
                             (int)cudaSharedmemCarveoutMaxShared);
  int dev = 0, sms = 0, per_sm = 0;
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, S::NT, smem);
  if (e != cudaSuccess) return cuda_status(e, "qsx_rk4_block_matrix_real_tc");
  // Two resident CTAs per SM overlap one CTA's epilogue with the other's MMA
  // chain; the occupancy query can report fewer than fit, and a second wave
  // is harmless because every CTA strides over the samples on its own.
  const int64_t grid = std::min<int64_t>(batch, (int64_t)std::max(per_sm, 2) * sms);
  kern<<<(unsigned)grid, S::NT, smem, st>>>(D, m, K, J, select, nselect, out, status, batch);
  QSX_LAUNCH_CHECK("qsx_rk4_block_matrix_real_tc");
  return QSX_OK;
}

}  // namespace qsx

using namespace qsx;

// Shapes the tensor-core form handles: m <= 64, K = 2^J or 2^J + 1, and at
// most 64 selected rows entering a product.
extern "C" int qsx_rk4_block_matrix_real_tc_supported(int m, int K, int nselect) {
  if (m < 1 || m > 64 || K < 2 || K > 64 || nselect < 1 || nselect > m) return 0;
  const bool pow2 = (K & (K - 1)) == 0, pow2p1 = ((K - 1) & (K - 2)) == 0 && K > 2;
  if (!pow2 && !pow2p1) return 0;
  // the last doubling multiplies R_1..R_b, b the largest power of two < K - 1
  int b = 1;
  while (2 * b < K - 1) b *= 2;
  return b * nselect <= 64 ? 1 : 0;
}

extern "C" int qsx_rk4_block_matrix_real_tc(const float* D, int m, int64_t batch, int K,
                                            const int* select, int nselect, float* out,
                                            int32_t* status, void* stream) {
  QSX_CHECK_ARG(batch >= 0 && batch <= 0x7fffffff, "qsx_rk4_block_matrix_real_tc: bad batch");
  if (!qsx_rk4_block_matrix_real_tc_supported(m, K, nselect)) {
    set_error("qsx_rk4_block_matrix_real_tc: shape m=%d K=%d nselect=%d not supported", m, K,
              nselect);
    return QSX_ERR_UNSUPPORTED;
  }
  if (batch == 0) return QSX_OK;
  QSX_CHECK_ARG(D && select && out, "qsx_rk4_block_matrix_real_tc: null pointer");
  QSX_CHECK_ARG((reinterpret_cast<uintptr_t>(D) & 3) == 0,
                "qsx_rk4_block_matrix_real_tc: D must be 4-byte aligned");
  int J = 0;
  while ((2 << J) <= K) ++J;
  cudaStream_t st = (cudaStream_t)stream;
  switch ((m + 7) / 8) {
#define B(G) \
  case G: return block_tc_launch<8 * G>(D, m, batch, K, J, select, nselect, out, status, st);
    B(1) B(2) B(3) B(4) B(5) B(6) B(7) B(8)
#undef B
  }
  return QSX_ERR_UNSUPPORTED;   // not reached: m <= 64
}
