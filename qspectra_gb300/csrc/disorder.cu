// Seeded static-disorder draws on the GPU, one thread per sample.
//
// Sample n of an ensemble takes its site-energy shifts from its own stream,
// RandomState(list(seed) + [n]).randn(n_sites) (qspectra/hamiltonian.py:
// 233-274, 552-578): the Mersenne Twister MT19937 seeded by an array
// (M. Matsumoto and T. Nishimura, ACM TOMACS 8, 1998; array initialisation of
// 2002), 53-bit uniforms, and Marsaglia's polar method for the normals, the
// second one of a pair first.  The host's stream objects cost 88 us a sample:
// 178 of the 180 ms of a 2001-sample ensemble call were draws.
//
// What bounds it: the seeding's two passes over 624 words are one serial
// chain of about 25 cycles a word.  Each thread keeps its words in shared
// memory, lanes side by side (word i of lane l in bank l), 78 KB a warp and
// two warps an SM, so 9728 samples run as one wave.  Words are twisted only
// as they are drawn: 7 normals use about 21 of the 624.
//
// Integer and uniform parts are the stream's own bits.  The logarithm is
// CUDA's, so a normal can differ from the host's in its last bit.
#include "qsx_common.cuh"

namespace qsx {

namespace {

constexpr int MT_N = 624, MT_M = 397;

struct MtBase { uint32_t w[MT_N]; };

// the generator's scalar seeding with 19650218, where array seeding starts
constexpr MtBase mt_base() {
  MtBase b{};
  b.w[0] = 19650218u;
  for (int i = 1; i < MT_N; ++i)
    b.w[i] = 1812433253u * (b.w[i - 1] ^ (b.w[i - 1] >> 30)) + (uint32_t)i;
  return b;
}

__constant__ MtBase MT_BASE = mt_base();

struct MtKey { uint32_t w[QSX_DISORDER_MAX_KEY]; };

// word of the stream at position `pos`, twisted in place when it is drawn
__device__ __forceinline__ uint32_t mt_next(uint32_t* st, int& pos) {
  const int i = pos, i1 = i + 1 == MT_N ? 0 : i + 1, im = i + MT_M >= MT_N ? i + MT_M - MT_N
                                                                           : i + MT_M;
  const uint32_t y = (st[i * 32] & 0x80000000u) | (st[i1 * 32] & 0x7fffffffu);
  uint32_t v = st[im * 32] ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
  st[i * 32] = v;
  pos = i1;
  v ^= v >> 11;
  v ^= (v << 7) & 0x9d2c5680u;
  v ^= (v << 15) & 0xefc60000u;
  return v ^ (v >> 18);
}

__device__ __forceinline__ double mt_uniform(uint32_t* st, int& pos) {
  const uint32_t a = mt_next(st, pos) >> 5, b = mt_next(st, pos) >> 6;
  return __dmul_rn(__dadd_rn(__dmul_rn((double)a, 67108864.0), (double)b), 1.0 / 9007199254740992.0);
}

__global__ void __launch_bounds__(32)
    disorder_kernel(MtKey key, int nkey, uint32_t start, int64_t batch, int n_sites, double scale,
                    double* __restrict__ out) {
  extern __shared__ uint32_t words[];
  const int64_t s = (int64_t)blockIdx.x * 32 + threadIdx.x;
  if (s >= batch) return;   // lanes share nothing
  uint32_t* st = words + threadIdx.x;
  const uint32_t index = start + (uint32_t)s;   // the key's last word
  for (int i = 0; i < MT_N; ++i) st[i * 32] = MT_BASE.w[i];
  int i = 1, j = 0;
  uint32_t prev = MT_BASE.w[0];
  for (int k = 0; k < MT_N; ++k) {   // nkey < 624
    const uint32_t word = j + 1 == nkey ? index : key.w[j];
    prev = (st[i * 32] ^ ((prev ^ (prev >> 30)) * 1664525u)) + word + (uint32_t)j;
    st[i * 32] = prev;
    if (++i == MT_N) {
      st[0] = prev;
      i = 1;
    }
    if (++j == nkey) j = 0;
  }
  for (int k = 0; k < MT_N - 1; ++k) {
    prev = (st[i * 32] ^ ((prev ^ (prev >> 30)) * 1566083941u)) - (uint32_t)i;
    st[i * 32] = prev;
    if (++i == MT_N) {
      st[0] = prev;
      i = 1;
    }
  }
  st[0] = 0x80000000u;
  int pos = 0;
  for (int q = 0; q < n_sites; q += 2) {
    double x1, x2, r2;
    do {
      x1 = __dadd_rn(__dmul_rn(2.0, mt_uniform(st, pos)), -1.0);
      x2 = __dadd_rn(__dmul_rn(2.0, mt_uniform(st, pos)), -1.0);
      r2 = __dadd_rn(__dmul_rn(x1, x1), __dmul_rn(x2, x2));
    } while (r2 >= 1.0 || r2 == 0.0);
    const double f = sqrt(__dmul_rn(-2.0, log(r2)) / r2);
    out[s * n_sites + q] = __dmul_rn(scale, __dmul_rn(f, x2));
    if (q + 1 < n_sites) out[s * n_sites + q + 1] = __dmul_rn(scale, __dmul_rn(f, x1));
  }
}

}  // namespace

}  // namespace qsx

using namespace qsx;

extern "C" int qsx_disorder_draws(const uint32_t* seed, int nseed, int64_t start, int64_t batch,
                                  int n_sites, double scale, double* out, void* stream) {
  QSX_CHECK_ARG(nseed >= 0 && nseed < QSX_DISORDER_MAX_KEY && (nseed == 0 || seed),
                "qsx_disorder_draws: 0 to %d seed words", QSX_DISORDER_MAX_KEY - 1);
  QSX_CHECK_ARG(start >= 0 && batch >= 0 && start + batch <= (int64_t)1 << 32 && n_sites >= 1,
                "qsx_disorder_draws: bad sizes");
  if (batch == 0) return QSX_OK;
  QSX_CHECK_ARG(out, "qsx_disorder_draws: null pointer");
  MtKey key{};
  for (int k = 0; k < nseed; ++k) key.w[k] = seed[k];
  const size_t smem = (size_t)MT_N * 32 * sizeof(uint32_t);
  cudaError_t e = cudaFuncSetAttribute(disorder_kernel,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_status(e, "qsx_disorder_draws");
  disorder_kernel<<<(unsigned)((batch + 31) / 32), 32, smem, (cudaStream_t)stream>>>(
      key, nseed + 1, (uint32_t)start, batch, n_sites, scale, out);
  QSX_LAUNCH_CHECK("qsx_disorder_draws");
  return QSX_OK;
}
