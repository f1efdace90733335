// exp(-gamma d^2) for FP64 kernel entries without the FP64 pipe.
//
// GB300 issues two FP64 operations per clock and SM and 64 or more integer
// ones, so an exponential of about twenty FP64 operations costs what three
// hundred integer ones cost.  Here only d^2 is FP64; the exponential is about
// sixty 32-bit integer operations on its bits, in the classic table-driven form
// (Tang, ACM TOMS 15(2), 1989) carried out in 64-bit fixed point:
//
//   U = gamma log2(e) d^2              64-bit mantissa product, then a shift
//   U = ip + j / 2048 + f,  0 <= f < 2^-11
//   2^-U = 2^-ip T[j] (1 - f (c1 - f (c2 - f c3))),  T[j] = 2^(-j / 2048)
//
// The cubic interpolates (1 - 2^-f) / f on [0, 2^-11] (error 9e-18); every
// fixed-point step truncates below 2^-61 of its operand.  Against 120-bit
// values of exp(-gamma d^2) (gamma d^2 itself is not rounded here) the error is
// at most 0.71 ulp up to gamma d^2 = 50 (rms 0.292; rounding alone 0.5 and 0.289),
// 1.1 ulp up to 200 and 3.2 ulp up to 700.  exp(-(gamma * d2)) with CUDA's exp, the
// form before, is off by 0.53 ulp below gamma d^2 = 0.03 (rms 0.289), 1.14 up to 1
// (0.342), 4.5 up to 8 (1.28) and 32 up to 50 (9.2), since half an ulp of gamma d^2
// is that much of the result.  A whole matrix (1500 points in the unit cube, gamma
// = 100) against extended precision: 6.3e-17 of its norm, 7.5e-17 before, and
// 8.0e-17 for the same formula in torch.  Arguments outside the fixed-point range (results below 2^-1021,
// negative gamma, NaN, infinities) take CUDA's exp.
#pragma once

#include <stdint.h>

#include <cmath>

#include "common.cuh"

namespace mpdok {

constexpr int PHI_TAB = 2048;  // entries of the table T in shared memory (16 KB)

// gamma log2(e) = cm 2^(ce - 63) with cm in [2^63, 2^64); ce is stored with the
// offset that the shift of gauss_phi uses.
struct GaussScale {
  uint64_t cm;
  int ce;
  double gamma;
};

#ifdef __CUDA_ARCH__
__device__ __forceinline__ uint32_t phi_umulhi(uint32_t a, uint32_t b) { return __umulhi(a, b); }
#else
inline uint32_t phi_umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
#endif

// High 64 bits of a b, at most 2 below the exact value.
__host__ __device__ __forceinline__ uint64_t mulhi64(uint64_t a, uint64_t b) {
  const uint32_t ah = (uint32_t)(a >> 32), al = (uint32_t)a, bh = (uint32_t)(b >> 32), bl = (uint32_t)b;
  return (uint64_t)ah * bh + phi_umulhi(ah, bl) + phi_umulhi(al, bh);
}

__host__ __device__ inline GaussScale gauss_scale(double gamma) {
  GaussScale c;
  c.gamma = gamma;
  c.cm = 0;
  c.ce = 1 << 20;  // every argument out of range: CUDA's exp
  if (gamma > 1e-290 && gamma < 1e290) {
    int e = 0;
    const double m = frexp(gamma, &e);                          // gamma = m 2^e, m in [0.5, 1)
    const uint64_t gm = (uint64_t)(m * 9007199254740992.0) << 11;  // m 2^64, exact
    uint64_t p = mulhi64(gm, 0xb8aa3b295c17f0bcull);            // m log2(e) 2^63, log2(e) 2^63 rounded
    int s = e + 1;                                              // gamma log2(e) = p 2^-64 2^s
    if (!(p >> 63)) {
      p <<= 1;
      --s;
    }
    c.cm = p;
    // d^2 = M 2^(ed - 1086) with M its mantissa aligned to 64 bits and ed its
    // biased exponent, so U = (M cm >> 64) 2^(ed - 1086 + s)
    c.ce = s - 1086 + 64;
  }
  return c;
}

static __device__ __noinline__ double gauss_phi_wide(double d2, double gamma) { return exp(-gamma * d2); }

// 2^(-i / 32) and 2^(-i / 2048), times 2^63.
__device__ const uint64_t PHI_A[32] = {
    0x8000000000000000ull, 0x7d41d96db915019dull, 0x7a92be8a92436616ull, 0x77f25ccdee6d7ae6ull,
    0x75606373ee921c97ull, 0x72dc8373be41a454ull, 0x70666f76154a7089ull, 0x6dfddbcbed791babull,
    0x6ba27e656b4eb57aull, 0x69540ec8f895722dull, 0x6712460a8fc24072ull, 0x64dcdec3371793d1ull,
    0x62b39508aa836d6full, 0x6096266533384a2bull, 0x5e8451cfac061b5full, 0x5c7dd7a3b17dcf75ull,
    0x5a827999fcef3242ull, 0x5891fac0e95612c8ull, 0x56ac1f752150a563ull, 0x54d0ad5a753e077cull,
    0x52ff6b54d8a89c75ull, 0x513821818624b40cull, 0x4f7a993048d088d7ull, 0x4dc69cdceaa72a9cull,
    0x4c1bf828c6dc54b8ull, 0x4a7a77d47f7b84b1ull, 0x48e1e9b9d588e19bull, 0x47521cc5a2e6a9e0ull,
    0x45cae0f1f545eb73ull, 0x444c0740496d4294ull, 0x42d561b3e6243d8aull, 0x4166c34c5615d0ecull,
};
__device__ const uint64_t PHI_B[64] = {
    0x8000000000000000ull, 0x7ff4e9597bed93abull, 0x7fe9d3a8e07bf086ull, 0x7fdebeee185d94ddull,
    0x7fd3ab290e46d769ull, 0x7fc89859acede72aull, 0x7fbd867fdf0acb3bull, 0x7fb2759b8f5762aaull,
    0x7fa765aca88f6453ull, 0x7f9c56b315705eaeull, 0x7f9148aec0b9b7b1ull, 0x7f863b9f952caca0ull,
    0x7f7b2f857d8c51e5ull, 0x7f702460649d92eaull, 0x7f651a30352731eeull, 0x7f5a10f4d9f1c7ddull,
    0x7f4f08ae3dc7c426ull, 0x7f44015c4b756c94ull, 0x7f38fafeedc8dd26ull, 0x7f2df5960f9207e1ull,
    0x7f22f1219ba2b4aeull, 0x7f17eda17cce812eull, 0x7f0ceb159deae091ull, 0x7f01e97de9cf1b6eull,
    0x7ef6e8da4b544f9aull, 0x7eebe92aad557001ull, 0x7ee0ea6efaaf4479ull, 0x7ed5eca71e4069a1ull,
    0x7ecaefd302e950afull, 0x7ebff3f2938c3f4full, 0x7eb4f905bb0d4f78ull, 0x7ea9ff0c64526f40ull,
    0x7e9f06067a4360baull, 0x7e940df3e7c9b9c8ull, 0x7e8916d497d0e3f4ull, 0x7e7e20a875461c4aull,
    0x7e732b6f6b18732aull, 0x7e6837296438cc27ull, 0x7e5d43d64b99ddd7ull, 0x7e5251760c3031b1ull,
    0x7e47600890f223deull, 0x7e3c6f8dc4d7e316ull, 0x7e31800592db7078ull, 0x7e26916fe5f89f5bull,
    0x7e1ba3cca92d152cull, 0x7e10b71bc7784943ull, 0x7e05cb5d2bdb84beull, 0x7dfae090c159e250ull,
    0x7deff6b672f84e24ull, 0x7de50dce2bbd85adull, 0x7dda25d7d6b2177full, 0x7dcf3ed35ee06328ull,
    0x7dc458c0af549908ull, 0x7db9739fb31cba29ull, 0x7dae8f7055489813ull, 0x7da3ac3280e9d4a8ull,
    0x7d98c9e62113e1faull, 0x7d8de88b20dc0224ull, 0x7d8308216b594720ull, 0x7d7828a8eba492a0ull,
    0x7d6d4a218cd895e5ull, 0x7d626c8b3a11d198ull, 0x7d578fe5de6e95a0ull, 0x7d4cb431650f00fdull,
};

// T[j] = 2^(63 - j / 2048) into shared memory, by every thread of the block
// (the caller's next barrier publishes it).
__device__ __forceinline__ void phi_table(uint64_t* T) {
  for (int j = threadIdx.x; j < PHI_TAB; j += blockDim.x) {
    const uint64_t a = PHI_A[j >> 6], b = PHI_B[j & 63];
    T[j] = (j & 63) == 0 ? a : (j >> 6) == 0 ? b : __umul64hi(a, b) << 1;
  }
}

// exp(-gamma d2); T as phi_table leaves it.
__host__ __device__ __forceinline__ double gauss_phi(double d2, const GaussScale& c, const uint64_t* T) {
#ifdef __CUDA_ARCH__
  const uint32_t hi = (uint32_t)__double2hiint(d2), lo = (uint32_t)__double2loint(d2);
#else
  uint64_t bits_in;
  memcpy(&bits_in, &d2, 8);
  const uint32_t hi = (uint32_t)(bits_in >> 32), lo = (uint32_t)bits_in;
#endif
  const int sh = (int)(hi >> 20) + c.ce;  // U = P 2^(sh - 64)
  const uint64_t M = ((uint64_t)(0x80000000u | (hi << 11) | (lo >> 21)) << 32) | (lo << 11);
  const uint64_t P = mulhi64(M, c.cm);
  // integer part (sh > 0) and 64-bit fraction of U
  const int sl = sh > 0 ? sh : 0, sr = sh < 0 ? (sh > -63 ? -sh : 63) : 0;
  const uint32_t ip = (uint32_t)((uint64_t)(uint32_t)(P >> 32) << (sl & 31) >> 32);
  const uint64_t F0 = sh >= 0 ? P << (sl & 31) : P >> sr;
#ifdef __CUDA_ARCH__
  if (sh > 11 || ip > 1020u) return gauss_phi_wide(d2, c.gamma);
#else
  if (sh > 11 || ip > 1020u) return exp(-c.gamma * d2);
#endif
  const uint64_t t = T[(uint32_t)(F0 >> 53)];
  const uint64_t F = F0 << 11;
  const uint32_t Fh = (uint32_t)(F >> 32);
  const uint32_t g = 0xf5fdefd9u - phi_umulhi(Fh, 0x71a7du);                    // (c2 - f c3) 2^34
  const uint64_t q = 0xb17217f7d1ab8ceeull - (((uint64_t)Fh * g) >> 13);        // (c1 - f (..)) 2^64
  const uint64_t d = mulhi64(F, q);                                             // (1 - 2^-f) 2^75
  const uint64_t v = t - (mulhi64(t, d) >> 11);                                 // 2^(63 - U + ip)
  const uint64_t r = ((v + 512) >> 10) + ((uint64_t)(1021u - ip) << 52);
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)r);
#else
  double out;
  memcpy(&out, &r, 8);
  return out;
#endif
}

}  // namespace mpdok
