// Float64 square root and exponential in 64-bit integer arithmetic.
//
// This part retires a float64 warp instruction every 19 clocks per SM, so the
// math library's exp and sqrt take about 300 and 140 clocks of an SM's float64
// units per warp (measured), and evaluating a kernel function cost more than
// its distance.  The same functions from 32-bit multiplies take 25 and 20.
// Accuracy before the final rounding: sqrt 2^-58.9, exp 2^-56 up to x = 32 and
// 2^-52.9 up to 512 (sampling against 60-digit arithmetic); from 512 on the
// library's exp is called.
#pragma once
#include <cuda_runtime.h>
#include <math.h>

namespace gpk {
namespace fx {

// 1 / sqrt(m / 2^64) for 2^62 <= m < 2^64, in units of 2^-61: a float32 seed,
// then one correction y (1 + e/2 + 3 e^2/8) with e = 1 - m y^2 in integers (the
// seed is good to 2^-21, what is left out is below 2^-62).
__device__ __forceinline__ unsigned long long rsqrt_unit(unsigned long long m) {
  float f = (float)(unsigned)(m >> 32) * 2.3283064365386963e-10f;
  asm("rsqrt.approx.ftz.f32 %0, %0;" : "+f"(f));
  const unsigned y0 = (unsigned)(f * 1073741824.f);
  const unsigned long long yy = (unsigned long long)y0 * y0;              // 2^-60
  const long long e = (1LL << 60) - (long long)__umul64hi(m, yy);         // |e| < 2^40
  const int eh = (int)(e >> 10);
  const long long corr = (e >> 1) + ((3 * (((long long)eh * eh) >> 40)) >> 3);
  // y0 (1 + corr) at 2^-61, corr in two parts so that 32-bit multiplies do
  const int ch = (int)(corr >> 20), cl = (int)(corr & 0xfffff);
  const long long dy = (long long)((unsigned long long)y0 * (unsigned)cl >> 20) +
                       (long long)(int)(y0 >> 1) * ch * 2 + (long long)(int)(y0 & 1) * ch;
  return ((unsigned long long)y0 << 31) + (unsigned long long)(dy >> 9);
}

// sqrt of a positive normal number (infinities and NaNs as they are).
__device__ __forceinline__ double sqrt_pos(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const int xb = (int)(b >> 52);
  unsigned long long m = (b << 11) | (1ULL << 63);  // v = (m / 2^64) 2^(xb - 1022)
  int e = xb - 1022;
  if (e & 1) {
    m >>= 1;
    ++e;
  }
  const unsigned long long r = __umul64hi(m, rsqrt_unit(m) << 1);  // [2^61, 2^62)
  const long long out = ((long long)(1021 + e / 2) << 52) + (long long)((r + 256) >> 9);
  return xb >= 0x7ff ? v : __longlong_as_double(out);
}

// 2^(-j / 32) in units of 2^-63
static __device__ const unsigned long long kExp2Tab[32] = {
    0x8000000000000000ULL, 0x7d41d96db915019dULL, 0x7a92be8a92436616ULL, 0x77f25ccdee6d7ae5ULL,
    0x75606373ee921c97ULL, 0x72dc8373be41a454ULL, 0x70666f76154a7088ULL, 0x6dfddbcbed791baaULL,
    0x6ba27e656b4eb57aULL, 0x69540ec8f895722dULL, 0x6712460a8fc24071ULL, 0x64dcdec3371793d1ULL,
    0x62b39508aa836d6eULL, 0x6096266533384a2bULL, 0x5e8451cfac061b5fULL, 0x5c7dd7a3b17dcf74ULL,
    0x5a827999fcef3242ULL, 0x5891fac0e95612c7ULL, 0x56ac1f752150a563ULL, 0x54d0ad5a753e077cULL,
    0x52ff6b54d8a89c75ULL, 0x513821818624b40cULL, 0x4f7a993048d088d6ULL, 0x4dc69cdceaa72a9cULL,
    0x4c1bf828c6dc54b7ULL, 0x4a7a77d47f7b84b0ULL, 0x48e1e9b9d588e19bULL, 0x47521cc5a2e6a9e0ULL,
    0x45cae0f1f545eb73ULL, 0x444c0740496d4293ULL, 0x42d561b3e6243d8aULL, 0x4166c34c5615d0ebULL};

static __device__ __noinline__ double exp_far(double x) { return exp(-x); }

// exp(-x) for x >= 0.  x log2(e) = n + j / 32 + r in fixed point, then 2^-n
// from the exponent, 2^(-j / 32) from the table and exp(-z), z = r ln 2 < 2^-5.5,
// from its Taylor series: the terms from z^4 in 32 bits, the rest in 64.
__device__ __forceinline__ double exp_neg(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const int xb = (int)((b >> 52) & 0x7ff);
  if (xb >= 1032) return exp_far(x);  // 512 and above, infinities, NaNs
  const bool big = xb >= 1028;        // 32 and above: five fewer fraction bits
  const unsigned long long m = (b & 0xfffffffffffffULL) | (xb ? 1ULL << 52 : 0ULL);
  const int sh = xb - (big ? 1022 : 1017);  // x in units of 2^-53 or 2^-58
  const unsigned long long xf = sh >= 0 ? m << sh : m >> min(-sh, 63);
  const unsigned long long log2e = 0x5c551d94ae0bf85eULL;  // 2^-62
  const unsigned long long ph = __umul64hi(xf, log2e), pl = xf * log2e;
  const int n = (int)(big ? ph >> 51 : ph >> 56);
  const unsigned long long f = big ? (ph << 13) | (pl >> 51) : (ph << 8) | (pl >> 56);
  const unsigned long long T = __ldg(&kExp2Tab[f >> 59]);
  const unsigned long long z = __umul64hi(f << 5, 0xb17217f7d1cf79acULL);  // 32 z, 2^-64
  const unsigned zh = (unsigned)(z >> 32), zl = (unsigned)z;
  // 1/24 - z/120 + z^2/720 - z^3/5040 at 2^-36
  unsigned a = 0x05b05b05u - (__umulhi(0x00d00d00u, zh) >> 5);
  a = 0x22222222u - (__umulhi(a, zh) >> 5);
  a = 0xaaaaaaaau - (__umulhi(a, zh) >> 5);
  const unsigned long long za =
      (unsigned long long)zh * a + ((unsigned long long)zl * a >> 32);  // 32 z a, 2^-68
  const unsigned long long c3 = 0x2aaaaaaaaaaaaaaaULL - (za >> 9);       // 1/6 - z a
  const unsigned long long c2 = (1ULL << 63) - (__umul64hi(z, c3) >> 5);  // 1/2 - z (..)
  const unsigned long long c1 = __umul64hi(z, c2) >> 5;
  const unsigned long long u = (z >> 5) - (__umul64hi(z, c1) >> 5);       // 1 - exp(-z)
  const unsigned long long v = T - __umul64hi(T, u);                      // (2^62, 2^63]
  const int lz = (int)(v >> 63) ^ 1;
  const unsigned long long top = v << lz;
  const unsigned long long r = (top >> 11) + ((top >> 10) & 1);
  return __longlong_as_double(((long long)(1022 - n - lz) << 52) + (long long)r);
}

}  // namespace fx
}  // namespace gpk
