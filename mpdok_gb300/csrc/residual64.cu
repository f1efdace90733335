// FP64 residuals R = B - A X of several columns on the tensor cores, from exact
// products of the leading digits.
//
// GB300 multiplies FP64 at two lanes per clock and SM, so a product with eight
// columns is bound by that pipe (n = 8192: 0.89 ms; reading A takes 0.08 ms).
// Here every entry becomes a 63-bit integer relative to the largest exponent of
// its row (A) or column (X), written in eight signed base-256 digits (Ozaki,
// Ogita, Oishi, Rump: error-free transformations of matrix multiplication,
// Numer. Algorithms 59, 2012).  Digits are exact FP16 numbers, products of
// digits have at most 14 bits, and the sums of up to eight digit pairs over a K
// of 128 stay below 2^24: the FP32 accumulators of the tensor cores hold them
// exactly.  Digit pairs (s, t) of equal weight s + t share an accumulator;
// weights 7 .. 14 are formed (36 of the 64 pairs).  The accumulators are drained
// as integers, so the order of the sums does not matter: a column's result
// depends neither on the other columns nor on the split of K.  The final
// subtraction from B carries its rounding error.
//
// What is dropped is relative to the largest entry of the row of A and of the
// column of X (2^E_i and 2^F: the powers of two at or below them), not to the terms
// of the sum: up to seven pairs of weight 6 for each a_ij, as many as it has digits
// (p_ij; none below 2^-61 of the largest), digits of random signs, rms 74 each,
//   dropped_i = 2^-60.2 sqrt(sum_j p_ij / 7) 2^(E_i + F).
// An FP64 product errs by some
//   rounded_i = 0.27 u g^(1/4) sqrt(sum_j a_ij^2 x_j^2),  u = 2^-53,
// with g the mean of sum_j p_ij / 7, the terms of a row that count (measured: 0.5 u
// with 13 of them, 0.9 u with 100, 1.9 u with 1400, 3.2 u with 8192).  The first
// exceeds the second where the columns of A differ in scale, or where one x_j towers
// over the others.  So every call compares their norms over the rows (once as they
// are and once relative to 2^E_i, so that small rows count too) and reports the
// columns that the FP64 product does better: those with
//   sum_j x_j^2 S_j < 2^-10.62 sqrt(g) m 2^(2 F),  m = sum_i w_i^2 2^(2 E_i),
//   S_j = sum_i w_i^2 a_ij^2,  g m = sum_j P_j,  P_j = sum_i w_i^2 2^(2 E_i) p_ij / 7,
// for w_i = 1 or w_i = 2^-E_i.  Measured (n = 2304 and 8192; kernels, random,
// positive, integer and Toeplitz matrices, graded ones): where the digits stay
// their error is 0.005 to 0.7 of the FP64 product's.
#include "common.cuh"
#include "residual64.cuh"

#include <cuda.h>
#include <cudaTypedefs.h>

#include <mutex>

namespace mpdok {
namespace r64 {

constexpr int BM = 128;       // rows of a tile
constexpr int NT = 32;        // columns of a tile
constexpr int BK = 32;        // K of a stage (64-byte rows)
constexpr int CHUNK = 128;    // K after which the accumulators are drained
constexpr int DIG = 8;        // digits
constexpr int GROUPS = 8;     // weights kept: s + t = 7 .. 14
constexpr int A_PLANE = BM * BK * 2;  // 8 KB
constexpr int X_PLANE = NT * BK * 2;  // 2 KB
constexpr int STAGE = DIG * (A_PLANE + X_PLANE);
constexpr int STAGES = 2;
constexpr int WORKERS = 8;    // warps that convert A and drain
constexpr int THREADS = 32 * (2 + WORKERS);
constexpr int NBAR = 3 * STAGES + 5;
constexpr int BAR_OFF = STAGES * STAGE;
constexpr int ALLOC = BAR_OFF + 8 * NBAR + 16 + 1024;
constexpr int TMEM_COLS = 2 * GROUPS * NT;
constexpr long long WAIT_LIMIT = 1LL << 26;
constexpr int EXP_BAD = 0x7ff;  // a row or column with an infinity or NaN
static_assert(ALLOC <= 232448 && TMEM_COLS == 512, "one CTA per SM");

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void bar_init(uint32_t bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
// false when the limit ran out or another role has given up
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, volatile int* fail) {
  for (long long i = 0; i < WAIT_LIMIT; ++i) {
    if (bar_try(bar, parity)) return true;
    if ((i & 63) == 63) {
      if (*fail) return false;
      __nanosleep(32);
    }
  }
  return false;
}
// K-major operand, 64-byte swizzle: 8-row atoms 512 bytes apart
__device__ __forceinline__ uint64_t desc_sw64(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}
__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t add) {
  asm volatile(
      "{\n"
      " .reg .pred p;\n"
      " setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(add)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(addr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// The value as an integer below 2^62 in magnitude in units of 2^(E - 1084), E the
// biased exponent of the row's or column's largest entry, plus a bias that turns
// the signed base-256 digits into bytes: digit k = byte k - 128 (UP 0, digits -128
// .. 127) or byte k - 127 (UP 1, -127 .. 128).  The two alternate along K: an
// entry's lowest digit is often a multiple of 128 or 64, and digits of one form
// would have a mean of -64 or -32 there, which the dropped pairs then sum over
// all of K (a matrix of positive entries, n = 8192: up to 1.7 times an FP64
// product's error; with both forms 0.3).
// An entry above 2^-41 of the largest that does not fit becomes odd (von
// Neumann's rounding, off by zero on average); smaller ones are cut off.
template <int UP>
__device__ __forceinline__ unsigned long long biased_digits(double a, int E) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a);
  const int e = (int)(b >> 52) & 0x7ff;
  unsigned long long m = b & 0xfffffffffffffull;
  if (e) m |= 0x10000000000000ull;
  const int sh = E - max(e, 1);
  m = (m << 9) >> min(sh, 63);
  if (__funnelshift_lc(0u, (uint32_t)b, (uint32_t)(41 - sh)) != 0u) m |= 1ull;  // the sh - 9 low bits, lost
  constexpr unsigned long long BIAS = UP ? 0x7f7f7f7f7f7f7f7full : 0x8080808080808080ull;
  return (long long)b < 0 ? BIAS - m : BIAS + m;
}
// The form of column j of A and row j of X: the parity of the low three bits of j
// (no step of two or four through K meets one form only).
constexpr int digit_form(int j) { return (j ^ j >> 1 ^ j >> 2) & 1; }

// Byte k of two biased values of forms UP and 1 - UP as two FP16 digits: 0x6400 |
// byte is 1024 + byte.
template <int UP>
__device__ __forceinline__ uint32_t digit_pair(unsigned long long a, unsigned long long b, int k) {
  const uint32_t x = k < 4 ? (uint32_t)a : (uint32_t)(a >> 32), y = k < 4 ? (uint32_t)b : (uint32_t)(b >> 32);
  const int q = k & 3;
  const uint32_t h = (__byte_perm(x, y, (uint32_t)(q | ((4 + q) << 8))) & 0x00ff00ffu) | 0x64006400u;
  constexpr uint32_t off = UP ? 0x6480647fu : 0x647f6480u;
  const __half2 d = __hsub2(*reinterpret_cast<const __half2*>(&h), *reinterpret_cast<const __half2*>(&off));
  return *reinterpret_cast<const uint32_t*>(&d);
}

// |a| relative to 2^(E - 1023), E at least its exponent, below 2; to 24 bits, and
// 0 below 2^-60.
__device__ __forceinline__ float relative_to(double a, int E) {
  const uint32_t hi = (uint32_t)__double2hiint(a), lo = (uint32_t)__double2loint(a);
  const int e = (int)(hi >> 20) & 0x7ff, d = e - E;
  return e == 0 || d < -60 ? 0.f : __uint_as_float((uint32_t)(d + 127) << 23 | (hi & 0xfffffu) << 3 | lo >> 29);
}

// E[i] = the largest biased exponent of row i (at least 1), over a column chunk.
__global__ void __launch_bounds__(256)
k_row_exponent(const double* __restrict__ A, long long lda, long long n, long long cchunk, int* __restrict__ E) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long long c0 = (long long)blockIdx.y * cchunk, c1 = min(n, c0 + cchunk);
  int m = 1;
#pragma unroll 8
  for (long long c = c0; c < c1; ++c) m = max(m, (__double2hiint(__ldg(A + i + c * lda)) >> 20) & 0x7ff);
  atomicMax(E + i, m);
}

// rel[i] = 2^(E_i - max E) (0 below 2^-60), *sum = the sum of its squares; one block.
__global__ void __launch_bounds__(1024) k_row_weights(const int* __restrict__ E, long long n, float* __restrict__ rel,
                                                      float* __restrict__ sum) {
  __shared__ int mx[32];
  __shared__ float red[32];
  int m = 1;
  for (long long i = threadIdx.x; i < n; i += blockDim.x) m = max(m, E[i]);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) mx[threadIdx.x >> 5] = m;
  __syncthreads();
  m = __reduce_max_sync(0xffffffffu, mx[threadIdx.x & 31]);
  float s = 0.f;
  for (long long i = threadIdx.x; i < n; i += blockDim.x) {
    const int d = E[i] - m;
    const float r = d < -60 ? 0.f : __uint_as_float((uint32_t)(d + 127) << 23);
    rel[i] = r;
    s = fmaf(r, r, s);
  }
  s = block_sum(s, red);
  if (threadIdx.x == 0) *sum = s;
}

// W[j] = (S_j, P_j) of the rule above with w_i = 2^-E_i, then with w_i = 1 (in units
// of the matrix's largest exponent).  A warp to a column: one more read of A
// (n = 8192: 0.12 ms a solve).
__global__ void __launch_bounds__(256)
k_column_weights(const double* __restrict__ A, long long lda, long long n, const int* __restrict__ E,
                 const float* __restrict__ rel, float4* __restrict__ W) {
  const long long j = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (j >= n) return;
  const double* a = A + j * lda;
  float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (long long i = threadIdx.x & 31; i < n; i += 32) {
    const double x = __ldg(a + i);
    const int Ei = __ldg(E + i), d = Ei - (int)((uint32_t)__double2hiint(x) >> 20 & 0x7ff);
    const float v = relative_to(x, Ei), r = __ldg(rel + i), w = v * r;
    const float p = d > 61 ? 0.f : (float)min(7, ((61 - d) >> 3) + 1) * (1.f / 7.f);
    t.x = fmaf(v, v, t.x);
    t.y += p;
    t.z = fmaf(w, w, t.z);
    t.w = fmaf(p * r, r, t.w);
  }
  t = make_float4(warp_sum(t.x), warp_sum(t.y), warp_sum(t.z), warp_sum(t.w));
  if ((threadIdx.x & 31) == 0) W[j] = t;
}

// Column of the caller's matrices that column c of the listed groups is.
__device__ __forceinline__ long long group_column(const ColGroups& g, int K, int c) { return (long long)g.id[c / K] * K + c % K; }

// Digits of the listed columns of X, one block per (padded) column: D[digit][column][k],
// k < kpad, zero past row n and for the padding columns; F[column] = exponent;
// lossy[column] = 1 where what the digits drop exceeds the rounding of an FP64
// product (a column of zeros drops nothing).
__global__ void __launch_bounds__(256)
k_column_digits(const double* __restrict__ X, long long ldx, long long n, int nc, long long kpad, int ncpad,
                int* __restrict__ F, uint32_t* __restrict__ D, const float4* __restrict__ W,
                const float* __restrict__ sum_rel, int* __restrict__ lossy, int K, const ColGroups groups) {
  __shared__ int red[8];
  __shared__ float fred[32];
  const int c = blockIdx.x;
  const long long src = c < nc ? group_column(groups, K, c) : 0;
  const double* x = X + src * ldx;
  int m = 1;
  if (c < nc)
    for (long long i = threadIdx.x; i < n; i += blockDim.x) m = max(m, (__double2hiint(x[i]) >> 20) & 0x7ff);
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  m = red[0];
#pragma unroll
  for (int w = 1; w < 8; ++w) m = max(m, red[w]);
  if (threadIdx.x == 0 && c < nc) F[c] = m;
  for (long long i = threadIdx.x; i < kpad / 2; i += blockDim.x) {
    const double a = c < nc && 2 * i < n ? x[2 * i] : 0.0, b = c < nc && 2 * i + 1 < n ? x[2 * i + 1] : 0.0;
    uint32_t* out = D + (long long)c * (kpad / 2) + i;
    const long long step = (long long)ncpad * (kpad / 2);
    static_assert(digit_form(0) == 0 && digit_form(2) == 1 && digit_form(4) == 1 && digit_form(6) == 0, "pairs");
    if ((i ^ i >> 1) & 1) {
      const unsigned long long u = biased_digits<1>(a, m), v = biased_digits<0>(b, m);
#pragma unroll
      for (int k = 0; k < DIG; ++k) out[k * step] = digit_pair<1>(u, v, k);
    } else {
      const unsigned long long u = biased_digits<0>(a, m), v = biased_digits<1>(b, m);
#pragma unroll
      for (int k = 0; k < DIG; ++k) out[k * step] = digit_pair<0>(u, v, k);
    }
  }
  if (c >= nc) return;
  // the rule above
  float q1 = 0.f, q2 = 0.f, p1 = 0.f, p2 = 0.f;
  int any = 0;
  for (long long i = threadIdx.x; i < n; i += blockDim.x) {
    const float v = relative_to(x[i], m);
    const float4 t = W[i];
    q1 = fmaf(v * v, t.x, q1);
    q2 = fmaf(v * v, t.z, q2);
    p1 += t.y;
    p2 += t.w;
    any |= x[i] != 0.0;
  }
  any = __syncthreads_or(any);
  q1 = block_sum(q1, fred);
  q2 = block_sum(q2, fred);
  p1 = block_sum(p1, fred);
  p2 = block_sum(p2, fred);
  constexpr float LIM = 6.354e-4f;  // 2^-10.62
  if (threadIdx.x == 0) lossy[src] = any && !(q1 >= LIM * sqrtf(p1 * (float)n) && q2 >= LIM * sqrtf(p2 * *sum_rel));
}

// One CTA: rows [128 bx, ..), columns [32 by, ..), K chunks [bz per, ..).  Warp 0
// loads the digits of X (TMA), warps 2 .. 9 convert A (coalesced FP64 loads, 39
// integer instructions per entry, 16-byte stores into the swizzled layout) and
// drain, warp 1 issues the MMAs: per 16-deep step 36 of 128 x 32, bound by the
// reads of A's digits from shared memory.  Two stages and two sets of
// accumulators, so converting, multiplying and draining overlap.
// n = 8192, 72 columns: 0.95 ms (FP64 pipe: nine passes of 0.89 ms).
__global__ void __launch_bounds__(THREADS, 1)
k_residual64(const double* __restrict__ A, long long lda, int n, const int* __restrict__ E,
             const __grid_constant__ CUtensorMap tmX, int nc, int nchunk, int per, long long* __restrict__ P, int* err) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gbase = smem_raw + (base - raw);
  const uint32_t bar_a = base + BAR_OFF;             // [STAGES] A converted (8 warps)
  const uint32_t bar_x = bar_a + 8 * STAGES;         // [STAGES] X landed
  const uint32_t bar_empty = bar_x + 8 * STAGES;     // [STAGES] both used
  const uint32_t bar_accf = bar_empty + 8 * STAGES;  // [2] accumulators complete
  const uint32_t bar_acce = bar_accf + 16;           // [2] accumulators drained
  const uint32_t bar_drain = bar_acce + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gbase + BAR_OFF + 8 * NBAR);
  __shared__ int s_fail;
  volatile int* fail = &s_fail;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * NT;
  const int c0 = blockIdx.z * per, c1 = min(nchunk, c0 + per);
  constexpr int SPC = CHUNK / BK;  // stages per chunk
  if (threadIdx.x == 0) {
    s_fail = 0;
    for (int st = 0; st < STAGES; ++st) {
      bar_init(bar_a + 8 * st, WORKERS);
      bar_init(bar_x + 8 * st, 1);
      bar_init(bar_empty + 8 * st, 1);
    }
    for (int a = 0; a < 2; ++a) {
      bar_init(bar_accf + 8 * a, 1);
      bar_init(bar_acce + 8 * a, WORKERS);
    }
    bar_init(bar_drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0) {
    if (lane == 0) {
      int g = 0;
      for (int c = c0; c < c1; ++c)
        for (int i = 0; i < SPC; ++i, ++g) {
          const int st = g % STAGES, round = g / STAGES;
          if (round > 0 && !bar_wait(bar_empty + 8 * st, (round - 1) & 1, fail)) {
            atomicExch(&s_fail, 1);
            c = c1;
            break;
          }
          bar_expect(bar_x + 8 * st, DIG * X_PLANE);
          asm volatile(
              "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
              ::"r"(base + st * STAGE + DIG * A_PLANE), "l"(reinterpret_cast<uint64_t>(&tmX)), "r"(bar_x + 8 * st),
              "r"(c * CHUNK + i * BK), "r"(n0), "r"(0)
              : "memory");
        }
      // loads in flight land in this CTA's shared memory: wait (bounded) for the last of each stage
      for (int st = 0; st < STAGES && st < g; ++st) {
        const int last = g - 1 - ((g - 1 - st) % STAGES);
        for (long long i = 0; i < WAIT_LIMIT && !bar_try(bar_x + 8 * st, (last / STAGES) & 1); ++i) {
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      // FP16 operands, FP32 accumulators, M = 128, N = 32
      const uint32_t idesc = (1u << 4) | ((uint32_t)(NT >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      int g = 0;
      bool ok = true;
      for (int c = c0; c < c1 && ok; ++c) {
        const int a = (c - c0) & 1, use = (c - c0) >> 1;
        if (use > 0 && !bar_wait(bar_acce + 8 * a, (use - 1) & 1, fail)) {
          atomicExch(&s_fail, 2);
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        for (int i = 0; i < SPC; ++i, ++g) {
          const int st = g % STAGES, ph = (g / STAGES) & 1;
          if (!bar_wait(bar_a + 8 * st, ph, fail) || !bar_wait(bar_x + 8 * st, ph, fail)) {
            atomicExch(&s_fail, 3);
            ok = false;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint32_t sa = base + st * STAGE, sx = sa + DIG * A_PLANE;
#pragma unroll 1
          for (int k = 0; k < BK / 16; ++k) {
            const uint32_t add = (i | k) ? 1u : 0u;
#pragma unroll
            for (int w = 0; w < GROUPS; ++w) {  // weight s + t = 7 + w
              const uint32_t d = tmem + (uint32_t)(a * GROUPS * NT + w * NT);
#pragma unroll
              for (int s = w; s < DIG; ++s)  // t = 7 + w - s
                mma(d, desc_sw64(sa + s * A_PLANE + k * 32), desc_sw64(sx + (7 + w - s) * X_PLANE + k * 32), idesc,
                    s == w ? add : 1u);
            }
          }
          mma_commit(bar_empty + 8 * st);
        }
        if (ok) mma_commit(bar_accf + 8 * a);
      }
      mma_commit(bar_drain);
      for (long long i = 0; i < WAIT_LIMIT && !bar_try(bar_drain, 0); ++i) {
        if (i > 64) __nanosleep(32);
      }
    }
  } else {
    const int t = threadIdx.x - 64;          // 0 .. 255
    const int r = t & (BM - 1), kc = t >> 7;  // this thread's row, 8-column runs kc and kc + 2 of a stage
    const int row = m0 + r;
    const bool live = row < n;
    const int Ei = live ? E[row] : 1;
    const double* Arow = A + (live ? row : 0);
    const int q = warp & 3, h = (warp - 2) >> 2;  // drain: lane quarter, column half
    long long hi[16], lo[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) hi[j] = lo[j] = 0;
    auto drain = [&](int c) {
      const int a = (c - c0) & 1, use = (c - c0) >> 1;
      if (!bar_wait(bar_accf + 8 * a, use & 1, fail)) {
        atomicExch(&s_fail, 4);
        return false;
      }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(a * GROUPS * NT + h * 16);
#pragma unroll
      for (int w = 0; w < GROUPS; ++w) {
        float v[16];
        tmem_ld16(ta + (uint32_t)(w * NT), v);
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const long long s = (long long)__float2int_rn(v[j]);
          if (w < 4) lo[j] += s * (1ll << (8 * w));
          else hi[j] += s * (1ll << (8 * (w - 4)));
        }
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) bar_arrive(bar_acce + 8 * a);
      return true;
    };
    int g = 0;
    bool ok = true;
    for (int c = c0; c < c1 && ok; ++c) {
#pragma unroll 1
      for (int i = 0; i < SPC; ++i, ++g) {
        const int st = g % STAGES, round = g / STAGES;
        const int kb = c * CHUNK + i * BK;
        double v[2][8];
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const int col = kb + 8 * (kc + 2 * u) + e;
            v[u][e] = live && col < n ? __ldg(Arow + (long long)col * lda) : 0.0;
          }
        if (round > 0 && !bar_wait(bar_empty + 8 * st, (round - 1) & 1, fail)) {
          atomicExch(&s_fail, 5);
          ok = false;
          break;
        }
        uint8_t* sa = gbase + st * STAGE;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          unsigned long long d[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) d[e] = digit_form(e) ? biased_digits<1>(v[u][e], Ei) : biased_digits<0>(v[u][e], Ei);
          uint32_t off = (uint32_t)(r * 64 + (kc + 2 * u) * 16);
          off ^= ((off >> 7) & 3u) << 4;
#pragma unroll
          for (int k = 0; k < DIG; ++k)
            *reinterpret_cast<uint4*>(sa + k * A_PLANE + off) =
                make_uint4(digit_pair<0>(d[0], d[1], k), digit_pair<1>(d[2], d[3], k), digit_pair<1>(d[4], d[5], k),
                           digit_pair<0>(d[6], d[7], k));
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) bar_arrive(bar_a + 8 * st);
      }
      if (ok && c > c0) ok = drain(c - 1);  // while the MMAs of chunk c run
    }
    if (ok && c1 > c0) ok = drain(c1 - 1);
    const int orow = m0 + q * 32 + lane;
    if (ok && orow < n) {
      long long* out = P + (long long)blockIdx.z * 2 * nc * n;
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int col = n0 + h * 16 + j;
        if (col < nc) {
          out[(long long)col * n + orow] = lo[j];
          out[(long long)(nc + col) * n + orow] = hi[j];
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0 && s_fail != 0 && err) atomicExch(err, 5);
  if (warp == 0) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS));
  }
}

// R = B - (hi 2^32 + lo) 2^(56 + E + F - 2168), the splits' integers added first.
// Four terms of at most 37 bits are exact FP64 numbers; the largest is subtracted
// with its rounding error kept.
__global__ void __launch_bounds__(256)
k_residual64_finish(const long long* __restrict__ P, int S, long long n, int nc, const int* __restrict__ E,
                    const int* __restrict__ F, const double* __restrict__ B, long long ldb, double* __restrict__ R,
                    long long ldr, int K, const ColGroups groups) {
  const long long total = n * nc;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
    const long long c = e / n, i = e % n, src = group_column(groups, K, (int)c);
    long long lo = 0, hi = 0;
    for (int s = 0; s < S; ++s) {
      lo += P[(long long)s * 2 * total + e];
      hi += P[(long long)s * 2 * total + total + e];
    }
    const int Ei = E[i], Fc = F[c];
    double r;
    if (Ei == EXP_BAD || Fc == EXP_BAD) {
      r = NAN;
    } else {
      const int w = 56 + Ei + Fc - 2168;
      constexpr long long MASK = (1ll << 27) - 1;
      const double t3 = -scalbn((double)(hi >> 27), w + 59), t2 = -scalbn((double)(hi & MASK), w + 32);
      const double t1 = -scalbn((double)(lo >> 27), w + 27), t0 = -scalbn((double)(lo & MASK), w);
      const double b = B[i + src * ldb];
      const double s = b + t3, bb = s - b;
      const double err = (b - (s - bb)) + (t3 - bb);
      const double s2 = s + t2, b2 = s2 - s;
      const double err2 = (s - (s2 - b2)) + (t2 - b2);
      r = s2 + ((t1 + t0) + (err + err2));
    }
    R[i + src * ldr] = r;
  }
}

static PFN_cuTensorMapEncodeTiled_v12000 encode() {
  static std::once_flag once;
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  return fn;
}

struct Layout {
  long long kpad = 0;
  int ncpad = 0, nchunk = 0, per = 0, S = 1;
  size_t off_E = 0, off_rel = 0, off_sum = 0, off_W = 0, off_F = 0, off_D = 0, off_P = 0, total = 0;
};

static Layout layout(long long n, int nc) {
  Layout l;
  l.nchunk = (int)((n + CHUNK - 1) / CHUNK);
  l.kpad = (long long)l.nchunk * CHUNK;
  l.ncpad = (nc + NT - 1) / NT * NT;
  // splits of K, of at least four chunks each: the number (up to 8) whose last
  // wave of one CTA per SM leaves the least idle (n = 8192, 72 columns: 192
  // tiles on 152 SMs, two waves in one piece, 9 in eight)
  const long long tiles = (n + BM - 1) / BM * (l.ncpad / NT), sms = num_sms();
  int S = 1;
  double best = 1e30;
  for (int c = 1; c <= 8 && c <= std::max(1, l.nchunk / 4); ++c) {
    const double t = (double)((tiles * c + sms - 1) / sms) / c * (1.0 + 0.02 * c);
    if (t < best) {
      best = t;
      S = c;
    }
  }
  l.per = (l.nchunk + S - 1) / S;
  l.S = (l.nchunk + l.per - 1) / l.per;
  size_t off = 0;
  auto take = [&](size_t b) { size_t o = off; off = align_up(off + b, 256); return o; };
  l.off_E = take(sizeof(int) * (size_t)n);
  l.off_rel = take(sizeof(float) * (size_t)n);
  l.off_sum = take(sizeof(float));
  l.off_W = take(sizeof(float4) * (size_t)n);
  l.off_F = take(sizeof(int) * (size_t)nc);
  l.off_D = take(sizeof(uint16_t) * (size_t)DIG * l.ncpad * l.kpad);
  l.off_P = take(sizeof(long long) * 2 * (size_t)l.S * nc * n);
  l.total = off;
  return l;
}

}  // namespace r64

bool residual64_pays(long long n, int nc) { return nc >= 4 && n >= 2048 && n <= (1LL << 30); }

// (fewer groups may need more: their K is split further)
size_t residual64_work_bytes(long long n, int K, int ng) {
  size_t most = 0;
  for (int g = 1; g <= ng && residual64_pays(n, K); ++g) most = std::max(most, r64::layout(n, K * g).total);
  return most;
}

int residual64_prepare(const double* A, long long lda, long long n, void* work, cudaStream_t s) {
  const r64::Layout l = r64::layout(n, 1);  // (what it fills lies before anything that depends on the columns)
  char* w = (char*)work;
  int* E = (int*)(w + l.off_E);
  float* rel = (float*)(w + l.off_rel);
  MPDOK_CUDA_TRY(cudaMemsetAsync(E, 0, sizeof(int) * n, s));
  const long long cchunk = std::max(256LL, (n + 65534) / 65535);
  dim3 grid((unsigned)((n + 255) / 256), (unsigned)((n + cchunk - 1) / cchunk));
  launch(r64::k_row_exponent, grid, 256, 0, s, A, lda, n, cchunk, E);
  launch(r64::k_row_weights, 1, 1024, 0, s, (const int*)E, n, rel, (float*)(w + l.off_sum));
  launch(r64::k_column_weights, (unsigned)((n + 7) / 8), 256, 0, s, A, lda, n, (const int*)E, (const float*)rel,
         (float4*)(w + l.off_W));
  MPDOK_LAUNCH_CHECK("residual weights");
  return MPDOK_OK;
}

int residual64(const double* A, long long lda, long long n, const double* X, long long ldx, int K,
               const ColGroups& groups, const double* B, long long ldb, double* R, long long ldr, void* work,
               int* lossy, int* err, cudaStream_t s) {
  using namespace r64;
  const int nc = K * groups.n;
  const Layout l = layout(n, nc);
  char* w = (char*)work;
  int* E = (int*)(w + l.off_E);
  int* F = (int*)(w + l.off_F);
  uint32_t* D = (uint32_t*)(w + l.off_D);
  long long* P = (long long*)(w + l.off_P);
  const int slot = prof_start(MPDOK_PROF_GEMV_F64, s);
  launch(k_column_digits, (unsigned)l.ncpad, 256, 0, s, X, ldx, n, nc, l.kpad, l.ncpad, F, D,
         (const float4*)(w + l.off_W), (const float*)(w + l.off_sum), lossy, K, groups);
  auto enc = encode();
  if (!enc) {
    set_error("cuTensorMapEncodeTiled unavailable from the driver");
    return MPDOK_ERR_UNSUPPORTED;
  }
  CUtensorMap tm;
  cuuint64_t gdim[3] = {(cuuint64_t)l.kpad, (cuuint64_t)l.ncpad, (cuuint64_t)DIG};
  cuuint64_t gstride[2] = {(cuuint64_t)l.kpad * 2, (cuuint64_t)l.kpad * l.ncpad * 2};
  cuuint32_t box[3] = {(cuuint32_t)BK, (cuuint32_t)NT, (cuuint32_t)DIG};
  cuuint32_t es[3] = {1, 1, 1};
  const CUresult r = enc(&tm, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, D, gdim, gstride, box, es,
                         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    set_error("cuTensorMapEncodeTiled (digits) failed (%d)", (int)r);
    return MPDOK_ERR_CUDA;
  }
  MPDOK_TRY(set_smem(k_residual64, ALLOC));
  dim3 grid((unsigned)((n + BM - 1) / BM), (unsigned)(l.ncpad / NT), (unsigned)l.S);
  k_residual64<<<grid, THREADS, ALLOC, s>>>(A, lda, (int)n, E, tm, nc, l.nchunk, l.per, P, err);
  count_launch();
  const unsigned g = (unsigned)std::max(1LL, std::min<long long>((n * nc + 255) / 256, (long long)num_sms() * 8));
  launch(k_residual64_finish, g, 256, 0, s, (const long long*)P, l.S, n, nc, (const int*)E, (const int*)F, B, ldb, R, ldr,
         K, groups);
  prof_stop(slot, s, (double)n * (double)n * 8.0 + 16.0 * (double)nc * (double)n);
  MPDOK_LAUNCH_CHECK("residual64");
  return MPDOK_OK;
}

}  // namespace mpdok
