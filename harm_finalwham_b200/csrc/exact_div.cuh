// exact_div.cuh -- several correctly rounded FP64 quotients by one divisor.
//
// A divisor that many numerators share is inverted once, and each quotient
// then takes one product and two FMAs.  The results are the bits of the IEEE
// division, which the FP64 path needs (it reproduces the reference's '/').
//
// Method: Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor" (IBM J. Res. Dev. 34, 1990); also Cornea, Harrison
// and Tang, "Scientific Computing on Itanium-based Systems" (2002).
//   * rcp_rn: from a seed with a relative error below 2^-18, one cubic step
//     gives y within an ulp of 1/b, and y + y (1 - b y), rounded once by the
//     FMA, is 1/b correctly rounded unless b's significand is all ones.
//   * quot: with y = RN(1/b) and q = RN(a y), the remainder b q - a, formed by
//     an FMA, corrects q to RN(a/b).  q itself is off by less than 1.5 ulp;
//     where a/b lies near the middle of two floats q is one of those two, the
//     remainder is exact and the corrected sum lies on the same side of the
//     middle as a/b (it is nearer to a/b than any quotient of two 53-bit
//     numbers can come to a middle).  Elsewhere the last rounding decides.
//     The remainder is taken as b q - a so that a quotient +-0 by a positive
//     divisor keeps the sign that the division gives.
// The steps neither overflow nor lose bits to underflow for b in [2^-200,
// 2^200) and a = +-0 or |a| in [2^-700, 2^700); any other operand, negative
// divisors, infinities and NaN among them, takes the division itself.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define HG_HD __host__ __device__ __forceinline__
#else
#define HG_HD static inline
#endif

namespace hg {

HG_HD uint32_t hi_word(double x) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__double2hiint(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return (uint32_t)(u >> 32);
#endif
}
HG_HD uint32_t lo_word(double x) {
#ifdef __CUDA_ARCH__
  return (uint32_t)__double2loint(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return (uint32_t)u;
#endif
}

// a first approximation of 1/b (the host's stand-in keeps 19 bits, so that
// tests there see a worse seed than the device's)
HG_HD double rcp_seed(double b) {
#ifdef __CUDA_ARCH__
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
  return y;
#else
  double y = 1.0 / b;
  uint64_t u;
  memcpy(&u, &y, 8);
  u &= ~((1ull << 33) - 1);
  memcpy(&y, &u, 8);
  return y;
#endif
}

// RN(1/b) for b in the range above, significand not all ones
HG_HD double rcp_rn(double b) {
  const double y0 = rcp_seed(b);
  const double e0 = fma(-b, y0, 1.0);
  const double y1 = fma(y0, fma(e0, e0, e0), y0);
  return fma(y1, fma(-b, y1, 1.0), y1);
}

// RN(a/b) from y = RN(1/b)
HG_HD double quot(double a, double b, double y) {
  const double q = a * y;
  return fma(-y, fma(b, q, -a), q);
}

// twice the biased exponent word of 2^e (the sign shifted out)
constexpr uint32_t exp_word2(int e) { return (uint32_t)(1023 + e) << 21; }
constexpr uint32_t kNumLo = exp_word2(-700), kNumRange = exp_word2(700) - exp_word2(-700);
constexpr uint32_t kDenLo = exp_word2(-200) >> 1, kDenRange = (exp_word2(200) >> 1) - kDenLo;

// whether rcp_rn holds for b, and quot for it (a sign would leave the range)
HG_HD bool rcp_ok(double b) { return hi_word(b) - kDenLo < kDenRange && lo_word(b) != 0xffffffffu; }

// A divisor and its reciprocal.  FP32 (the mixed-precision path) divides.
template <typename T>
struct Divisor {
  T b;
};
template <>
struct Divisor<double> {
  double b, y;
  bool ok;
};

HG_HD Divisor<double> make_divisor(double b) { return Divisor<double>{b, rcp_rn(b), rcp_ok(b)}; }
HG_HD Divisor<float> make_divisor(float b) { return Divisor<float>{b}; }
// the same with a reciprocal formed earlier (0: none that holds)
HG_HD Divisor<double> known_divisor(double b, double y) { return Divisor<double>{b, y, y != 0.0}; }
HG_HD Divisor<float> known_divisor(float b, float) { return Divisor<float>{b}; }
// the reciprocal to keep for known_divisor
HG_HD double kept_rcp(double b) { return rcp_ok(b) ? rcp_rn(b) : 0.0; }
HG_HD float kept_rcp(float) { return 0.f; }

// q[i] = a[i] / d, i < N.  One maximum over the exponent words tells whether
// every numerator is in range; zeros fail it and are let through by the
// second look, which only warps with such a numerator take.
template <int N>
HG_HD void div_n(const double *a, const Divisor<double> &d, double *q) {
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < N; i++) {
    const uint32_t v = (hi_word(a[i]) << 1) - kNumLo;
    m = v > m ? v : m;
  }
  bool fast = d.ok && m < kNumRange;
  if (!fast && d.ok) {
    m = 0;
#pragma unroll
    for (int i = 0; i < N; i++) {
      const uint32_t h = hi_word(a[i]) << 1;
      const uint32_t v = (h | lo_word(a[i])) == 0 ? 0 : h - kNumLo;
      m = v > m ? v : m;
    }
    fast = m < kNumRange;
  }
  if (fast) {
#pragma unroll
    for (int i = 0; i < N; i++) q[i] = quot(a[i], d.b, d.y);
  } else {
#pragma unroll
    for (int i = 0; i < N; i++) q[i] = a[i] / d.b;
  }
}
template <int N>
HG_HD void div_n(const float *a, const Divisor<float> &d, float *q) {
#pragma unroll
  for (int i = 0; i < N; i++) q[i] = a[i] / d.b;
}

}  // namespace hg
