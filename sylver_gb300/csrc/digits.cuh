// Cutting FP64 rows into signed 9-bit digits for the tensor-core update of
// FP64 fronts (kernels_tc64.cu), shared by the kernels that write its operands.
// Integer and FP32 arithmetic only: the FP64 pipe runs at two per clock and SM.
#pragma once

#include "tc.hpp"

namespace sylver_gb300 {

namespace {

constexpr int OZ_NONFINITE = 1 << 20;  // scale exponent of a row with Inf / NaN
constexpr int OZ_EMPTY = -(1 << 14);   // ... of a zero row

// running sum of squares s 4^e with the exponent e of the largest entry
__device__ __forceinline__ void norm_add(int& e, float& s, long long xb, bool& bad) {
  const int ex = (int)((unsigned long long)xb >> 52) & 0x7ff;
  const unsigned long long mant = (unsigned long long)xb & 0xfffffffffffffull;
  if (ex == 0 && mant == 0) return;
  if (ex == 0x7ff) {
    bad = true;
    return;
  }
  float f = __uint_as_float(0x3f800000u | (unsigned)(mant >> 29));
  int xe = ex - 1023;
  if (ex == 0) {  // subnormal
    f -= 1.f;
    xe = -1022;
  }
  if (xe > e) {
    const int d = xe - e;
    s = d > 60 ? 0.f : s * __uint_as_float((unsigned)(127 - 2 * d) << 23);
    e = xe;
  }
  const int d = e - xe;
  if (d <= 60) {
    f *= __uint_as_float((unsigned)(127 - d) << 23);
    s = fmaf(f, f, s);
  }
}

// |round(x 2^(71 - e))| as a 72-bit integer (hi: its upper 8 bits), |x| < 2^e;
// every bit of an entry down to 2^-18 of 2^e is kept
__device__ __forceinline__ unsigned long long to_fixed(long long xb, int e, unsigned& hi) {
  const int ex = (int)((unsigned long long)xb >> 52) & 0x7ff;
  unsigned long long m = (unsigned long long)xb & 0xfffffffffffffull;
  int sh = 71 - e - 1074;  // x = m 2^(max(ex, 1) - 1075)
  if (ex) {
    m |= 1ull << 52;
    sh += ex - 1;
  }
  hi = 0;
  if (sh > 0) {
    sh = min(sh, 63);
    hi = (unsigned)(m >> (64 - sh));
    return m << sh;
  }
  if (sh < -54) return 0;
  return sh < 0 ? (m + (1ull << (-sh - 1))) >> (-sh) : m;
}

// smallest exponent with 2^e above the norm of a running sum (a margin covers
// the truncated entries and the sum's rounding)
__device__ __forceinline__ int norm_exponent(int e, float s) {
  return s > 0.f ? e + (((int)(__float_as_uint(s * 1.001f) >> 23) - 127 + 2) >> 1) : e;
}

// combine two running sums
__device__ __forceinline__ void norm_merge(int& e, float& s, int e2, float s2) {
  const int em = max(e, e2), d = em - e, d2 = em - e2;
  s = (d <= 60 ? s * __uint_as_float((unsigned)(127 - 2 * d) << 23) : 0.f) +
      (d2 <= 60 ? s2 * __uint_as_float((unsigned)(127 - 2 * d2) << 23) : 0.f);
  e = em;
}

// Balanced digits (|d| <= 256, the sign included) of one entry of a row with
// scale exponent e; zeros where the row is empty or has no finite scale.
__device__ __forceinline__ void cut_digits(long long xb, int e, int (&d)[OZ_DIGITS]) {
  unsigned hi = 0;
  const unsigned long long lo =
      e == OZ_EMPTY || e == OZ_NONFINITE ? 0ull : to_fixed(xb, e, hi);
  const int sgn = xb < 0 ? -1 : 0;
  auto cut = [](int& f) {  // the lowest digit of f; f <- the rest
    const int q = ((f + 256) & 511) - 256;
    f = (f - q) >> 9;
    return q;
  };
  int f = (int)(lo & 0x3ffff);  // digits 8, 7 and a carry
  d[7] = cut(f);
  d[6] = cut(f);
  const unsigned long long r = (((unsigned long long)hi << 46) | (lo >> 18)) + (unsigned)f;
  f = (int)(r & 0x7ffffff);  // digits 6, 5, 4 and a carry
  d[5] = cut(f);
  d[4] = cut(f);
  d[3] = cut(f);
  f += (int)(r >> 27);
  d[2] = cut(f);
  d[1] = cut(f);
  d[0] = f;
#pragma unroll
  for (int p = 0; p < OZ_DIGITS; ++p) d[p] = (d[p] ^ sgn) - sgn;
}

// Digits of two neighbouring K columns of a row with scale exponent e, one
// 4-byte store per plane at element offset o (even) of plane 0.
__device__ __forceinline__ void store_digits(long long x0, long long x1, int e, uint16_t* o,
                                             int64_t pstride) {
  int d0[OZ_DIGITS], d1[OZ_DIGITS];
  cut_digits(x0, e, d0);
  cut_digits(x1, e, d1);
#pragma unroll
  for (int p = 0; p < OZ_DIGITS; ++p) {
    // small integers are exact in BF16: the upper half of the float
    const unsigned b0 = __float_as_uint(__int2float_rn(d0[p]));
    const unsigned b1 = __float_as_uint(__int2float_rn(d1[p]));
    *reinterpret_cast<uint32_t*>(o + p * pstride) = __byte_perm(b0, b1, 0x7632);
  }
}

}  // namespace

}  // namespace sylver_gb300
