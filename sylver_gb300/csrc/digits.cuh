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

// round(x 2^(62 - e)) as a 64-bit integer, |x| < 2^e
__device__ __forceinline__ long long to_fixed(long long xb, int e) {
  const int ex = (int)((unsigned long long)xb >> 52) & 0x7ff;
  unsigned long long m = (unsigned long long)xb & 0xfffffffffffffull;
  int sh = 62 - e - 1074;  // x = m 2^(max(ex, 1) - 1075)
  if (ex) {
    m |= 1ull << 52;
    sh += ex - 1;
  }
  unsigned long long f;
  if (sh >= 0) f = m << min(sh, 63);
  else if (sh < -54) f = 0;
  else f = (m + (1ull << (-sh - 1))) >> (-sh);
  return xb < 0 ? -(long long)f : (long long)f;
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

// Digits of the fixed-point values of two neighbouring K columns, one 4-byte
// store per plane at element offset o (even) of plane 0.
__device__ __forceinline__ void store_digits(long long f0, long long f1, uint16_t* o,
                                             int64_t pstride) {
#pragma unroll
  for (int p = OZ_DIGITS - 1; p >= 0; --p) {
    int d0, d1;
    if (p > 0) {  // balanced digit in [-256, 255], the rest carries up
      d0 = (((int)f0 + 256) & 511) - 256;
      d1 = (((int)f1 + 256) & 511) - 256;
      f0 = (f0 - d0) >> 9;
      f1 = (f1 - d1) >> 9;
    } else {
      d0 = (int)f0;
      d1 = (int)f1;
    }
    // small integers are exact in BF16: the upper half of the float
    const unsigned b0 = __float_as_uint(__int2float_rn(d0));
    const unsigned b1 = __float_as_uint(__int2float_rn(d1));
    *reinterpret_cast<uint32_t*>(o + p * pstride) = __byte_perm(b0, b1, 0x7632);
  }
}

}  // namespace

}  // namespace sylver_gb300
