// Reciprocal square roots of Cholesky pivots without IEEE square root and
// division, which cost several times as long on the chain of pivots, and an FP64
// quotient off the FP64 pipe.
#pragma once

#include <cfloat>

#include "device.hpp"

namespace sylver_gb300 {

namespace {

// 1 / sqrt(d) where d has no normal exponent
__device__ __noinline__ double rsqrt64_slow(double d) { return 1.0 / sqrt(d); }

// 1 / sqrt(d), d > 0, to within 2^-57.8 before the rounding: the FP32 estimate
// y0 of the mantissa's and one step of Householder's method of third order,
// y0 (1 + e / 2 + 3 e^2 / 8), e = 1 - f y0^2, in integer arithmetic, whose latency is a
// fraction of the FP64 pipe's.  (An estimate within four ulp leaves |e| < 2^-19.9
// and 5 e^3 / 16 < 2^-61; the correction enters in units of 2^-58.)
__device__ __forceinline__ double rsqrt64(double d) {
  const long long b = __double_as_longlong(d);
  const int ex = (int)(b >> 52);  // d > 0: no sign bit
  if (ex == 0 || ex == 0x7ff) return rsqrt64_slow(d);
  const int q = (ex - 1023) >> 1, odd = (ex - 1023) & 1;
  // d = f 4^q, f = m 2^(odd - 52) in [1, 4)
  const unsigned long long m = ((unsigned long long)b & 0xfffffffffffffull) | (1ull << 52);
  const float ff = __uint_as_float(((unsigned)(127 + odd) << 23) | (unsigned)((m >> 29) & 0x7fffff));
  // y0 = Y 2^-24 in [1/2, 1)
  const unsigned Y = min((unsigned)(rsqrtf(ff) * 16777216.f), 16777215u);
  const unsigned long long P = (unsigned long long)Y * Y;
  // e in units of 2^-62
  const unsigned long long hi = __umul64hi(m << 11, P << 16);
  const long long e = (long long)((1ull << (63 - odd)) - hi) >> (1 - odd);
  const int t = (int)(e >> 21);
  const long long dl = (e >> 1) + (((long long)t * t * 3) >> 23);
  const long long y = ((long long)Y << 39) + (((long long)Y * (dl >> 4)) >> 19);
  const unsigned long long r = (unsigned long long)(y + (1 << 9)) >> 10;  // 53 bits
  return __longlong_as_double((long long)(((unsigned long long)(1021 - q) << 52) + r));
}

// a / b rounded to nearest even, bit for bit the IEEE quotient, in integer
// arithmetic: a reciprocal of b's mantissa from the FP32 estimate y0 and one step of
// the hyperpower iteration of order three, y0 (1 + e + e^2), e = 1 - f y0, a quotient
// within one unit, and its exact remainder.  About
// 45 integer instructions; the FP64 pipe takes a dozen instructions of 65 clocks.
// Operands or results without a normal exponent take the division itself.
__device__ __noinline__ double div64_slow(double a, double b) { return a / b; }
__device__ __forceinline__ double div64(double a, double b) {
  const unsigned long long ab = (unsigned long long)__double_as_longlong(a);
  const unsigned long long bb = (unsigned long long)__double_as_longlong(b);
  const int ea = (int)(ab >> 52) & 0x7ff, eb = (int)(bb >> 52) & 0x7ff;
  const int e = ea - eb + 1023;
  if (ea == 0 || eb == 0 || ea == 0x7ff || eb == 0x7ff || e < 2 || e > 2045)
    return div64_slow(a, b);
  const unsigned long long ma = (ab & 0xfffffffffffffull) | (1ull << 52);
  const unsigned long long mb = (bb & 0xfffffffffffffull) | (1ull << 52);
  const float f = __uint_as_float(0x3f800000u | (unsigned)((mb >> 29) & 0x7fffff));
  const unsigned Y = min((unsigned)(__fdividef(1.f, f) * 16777216.f), 16777215u);
  // e in units of 2^-76 (2^76 - mb Y fits 64 bits), then e + e^2
  const long long e76 = (long long)(0ull - mb * Y);
  const long long h = e76 >> 24;
  const long long d76 = e76 + ((h * h) >> 28);
  // 2^63 / f and the quotient in units of 2^-62
  const unsigned long long r63 =
      ((unsigned long long)Y << 39) + (unsigned long long)(((long long)Y * (d76 >> 17)) >> 20);
  const unsigned long long q62 = __umul64hi(ma << 11, r63);
  const int lt = ma < mb;  // the quotient of the mantissas is below one
  unsigned long long q = q62 >> (10 - lt);
  long long rem = (long long)((ma << (52 + lt)) - q * mb);
  if (rem < 0) {
    --q;
    rem += (long long)mb;
  } else if (rem >= (long long)mb) {
    ++q;
    rem -= (long long)mb;
  }
  if (2 * rem > (long long)mb || (2 * rem == (long long)mb && (q & 1))) ++q;
  return __longlong_as_double((long long)(((ab ^ bb) & 0x8000000000000000ull) |
                                          (((unsigned long long)(e - lt - 1) << 52) + q)));
}
__device__ __forceinline__ double quot(double a, double b) { return div64(a, b); }
__device__ __forceinline__ float quot(float a, float b) { return a / b; }

// the same in FP32: the hardware estimate and one Newton step y (1 + e / 2), the
// residual e = 1 - d y^2 with the product d y in two parts (0.5001 ulp)
__device__ __forceinline__ float rsqrt32(float d) {
  const float r = rsqrtf(d);
  const float h = d * r;
  const float e = fmaf(-fmaf(d, r, -h), r, fmaf(-h, r, 1.f));
  return d <= FLT_MAX ? fmaf(0.5f * r, e, r) : 0.f;
}
__device__ __forceinline__ double pivot_rsqrt(double d) { return rsqrt64(d); }
__device__ __forceinline__ float pivot_rsqrt(float d) { return rsqrt32(d); }
// sqrt(d) from r = pivot_rsqrt(d): d r corrected by its remainder (0.51 ulp where the
// remainder does not underflow)
template <typename T> __device__ __forceinline__ T pivot_sqrt(T d, T r) {
  const T s = d * r;
  return r > T(0) ? fma(fma(-s, s, d), T(0.5) * r, s) : d;
}

}  // namespace

}  // namespace sylver_gb300
