// Float64 Cholesky of a 64-wide block and its panel in 64-bit fixed point.
//
// This part retires one float64 warp instruction every 19 clocks per SM with a
// latency of 64 (measured; masked lanes cost the same), so a 64-step
// factorisation with float64 square roots, divisions and updates took 74 us.
// A Cholesky factor needs no floating exponent: with rows and columns scaled
// by powers of two 2^e_i >= sqrt(a_ii), every entry of the scaled matrix, of
// its Schur complements and of its factor stays within [-1, 1].  Entries are
// held as integers in units of 2^-60 (float64's own rounding is 2^-53 of the
// row's size), split into signed 32-bit halves v = vh 2^32 + vl for the
// products: three 32 x 32 + 64 multiply-adds and the high half of a fourth.
//
// A row whose entry leaves [-1, 1], or whose norm does, belongs to a matrix that
// is not positive definite; it is marked, which makes the pivot of its order
// fail.  The marks are needed beside the pivots' own signs: 63 columns can take
// 63 from a diagonal entry, which in 64 bits (a range of [-8, 8)) wraps to a
// positive number.
#pragma once
#include "gpk_common.cuh"

namespace gpk {
namespace fx {

constexpr int FRAC = 60;
constexpr long long ONE = 1LL << FRAC;
constexpr long long LIMIT = ONE + (1LL << 39);  // |L'| of a definite matrix, with rounding

struct Limbs {
  int h, l;
};
__device__ __forceinline__ Limbs limbs(long long v) {
  return {(int)((v + 0x80000000LL) >> 32), (int)v};
}

// Sums of up to eight limb products, combined into the sum's fixed-point value
// (the rows' norms are at most 1, which keeps both sums in range).  Left out is
// less than 2^-27 of a unit per product; leaving the low x low products out
// altogether cost up to 8 units each and a decimal digit of the log marginal
// likelihood of a smooth kernel, whose later columns are small.
struct Acc {
  long long hh = 0, mid = 0;
  __device__ __forceinline__ void add(const Limbs& a, const Limbs& b) {
    hh += (long long)a.h * b.h;
    mid += (long long)a.h * b.l;
    mid += (long long)a.l * b.h;
    mid += __mulhi(a.l, b.l);
  }
  __device__ __forceinline__ long long value() const { return (hh << (64 - FRAC)) + (mid >> (FRAC - 32)); }
};

// Scale exponent e of a row from its diagonal entry: 2^(2 e) >= a.
__device__ __forceinline__ int scale_of(double a) {
  const int xb = (int)((__double_as_longlong(a) >> 52) & 0x7ff);
  return (xb - 1021) >> 1;  // a < 2^(xb - 1022)
}

// a 2^-e in fixed point; *bad is set when that is not within [-2, 2].
__device__ __forceinline__ long long to_fixed(double a, int e, bool& bad) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(a);
  const int xb = (int)((b >> 52) & 0x7ff);
  const unsigned long long m = (b & 0xfffffffffffffULL) | (xb ? 1ULL << 52 : 0ULL);
  const int sh = (xb ? xb : 1) - 1075 - e + FRAC;
  if (m == 0) return 0;
  if (sh > 8 || xb == 0x7ff) {
    bad = true;
    return 0;
  }
  const long long v = sh >= 0 ? (long long)(m << sh)
                              : (sh > -55 ? (long long)((m + (1ULL << (-sh - 1))) >> -sh) : 0LL);
  return (long long)b < 0 ? -v : v;
}

// v 2^e as a float64, rounded to nearest.
__device__ __forceinline__ double to_double(long long v, int e) {
  const unsigned long long m = v < 0 ? 0ULL - (unsigned long long)v : (unsigned long long)v;
  if (m == 0) return 0.0;
  const int lz = __clzll((long long)m);
  const unsigned long long top = m << lz;
  unsigned long long r = top >> 11;
  const unsigned long long rem = top & 0x7ff;
  if (rem > 0x400 || (rem == 0x400 && (r & 1))) ++r;
  const int biased = 1023 + 63 - lz - FRAC + e;
  if (biased >= 1 && biased <= 2046)
    return __longlong_as_double((long long)((v < 0 ? 0x8000000000000000ULL : 0ULL) |
                                            (((unsigned long long)(biased - 1) << 52) + r)));
  const double x = scalbn((double)r, 63 - lz - FRAC + e - 52);
  return v < 0 ? -x : x;
}

// 1 / sqrt(d) of a fixed-point 0 < d as y 2^(-s - 61).
__device__ __forceinline__ void rsqrt_fixed(long long d, long long& y, int& s) {
  const int lz = __clzll(d);
  unsigned long long m = (unsigned long long)d << lz;
  int ex = 64 - FRAC - lz;  // d 2^-FRAC = (m / 2^64) 2^ex
  if (ex & 1) {
    m >>= 1;
    ++ex;
  }
  y = (long long)rsqrt_unit(m);
  s = ex / 2;  // ex is even
}

// a / sqrt(d) in fixed point from rsqrt_fixed's y and s (-58 <= s <= 1); *bad
// is set when it leaves the range of a definite matrix.  No branches: these
// sit on the chain of pivots.
__device__ __forceinline__ long long times_rsqrt(long long a, long long y, int s, bool& bad) {
  const long long mag = a < 0 ? -a : a;
  const bool over = (mag >> (FRAC + 1 + s)) != 0;  // the shifted operand would wrap
  const long long v = __mul64hi(a << (2 - s), y) << 1;
  const bool out = over || v > LIMIT || v < -LIMIT;
  bad = bad || out;
  return out ? 0 : v;
}

}  // namespace fx
}  // namespace gpk
