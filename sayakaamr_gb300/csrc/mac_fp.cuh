// FP64 bookkeeping on the integer pipe.
//
// GB300 issues FP64 at 2 operations per SM and clock, and its FP64 pipe
// also carries FP64 compares, min/max and the FP32 <-> FP64 conversions.
// The BiCGSTAB vector kernels of the device solve are bound by that pipe, so
// every operation here that only moves or orders bits is done on 32/64-bit
// integers instead, with results identical to the FP64 instructions:
//   * non-negative doubles order like their bit patterns read as integers,
//     and a NaN (all-ones exponent, non-zero mantissa) orders above +inf, so
//     the max of |v| over bit patterns is the NaN-propagating max of |v|;
//   * float -> double is exact: rebias the exponent, widen the mantissa
//     (denormals normalised);
//   * double -> float rounds to nearest with ties to even (IEEE 754
//     roundTiesToEven), float denormals, overflow to inf and NaN included.
#pragma once

#include <cuda_runtime.h>

namespace sayaka_gb300 {
namespace fpint {

__device__ __forceinline__ unsigned long long abs_bits(double v) {
  return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
}

// running max of |v| as bit patterns (start from 0 = +0.0)
__device__ __forceinline__ unsigned long long max_abs(unsigned long long m, double v) {
  const unsigned long long u = abs_bits(v);
  return u > m ? u : m;
}

__device__ __forceinline__ double from_bits(unsigned long long u) { return __longlong_as_double((long long)u); }

// v > 0 for v that is never a NaN (volume fractions, operator factors):
// positive doubles, and only they, have positive bit patterns as int64
__device__ __forceinline__ bool positive(double v) { return __double_as_longlong(v) > 0; }

// exact float -> double, every case on the integer pipe (no conversion
// instruction at all, so that none is issued even where the compiler
// evaluates both sides of a branch): normal floats rebias the exponent and
// widen the mantissa, zeros keep their sign; what is left (`rare`: denormals,
// normalised by moving the leading one to bit 23, inf and NaN, which keep
// their mantissa) is a call, so that a kernel that widens in many places
// stays small enough for the instruction cache
__device__ __forceinline__ bool rare(float f) {
  const unsigned a = __float_as_uint(f) << 1;
  return a != 0u && a - 0x01000000u >= 0xfe000000u;
}
__device__ __forceinline__ double widen_common(float f) {
  const unsigned u = __float_as_uint(f), a = u & 0x7fffffffu;
  const unsigned hi = (a ? (a >> 3) + 0x38000000u : 0u) | (u & 0x80000000u);
  return from_bits(((unsigned long long)hi << 32) | (u << 29));
}
static __device__ __noinline__ double widen_rare(float f) {
  const unsigned u = __float_as_uint(f);
  if (((u >> 23) & 0xffu) == 0xffu) {
    const unsigned hi = (u & 0x80000000u) | 0x7ff00000u | ((u >> 3) & 0x000fffffu);
    return from_bits(((unsigned long long)hi << 32) | (u << 29));
  }
  const unsigned m = u & 0x7fffffu;
  const unsigned long long sign = (unsigned long long)(u & 0x80000000u) << 32;
  const int s = __clz((int)m) - 8;  // m * 2^-149 = (m << s) * 2^(-149 - s), bit 23 set
  return from_bits(sign | ((unsigned long long)(897 - s) << 52) | ((unsigned long long)((m << s) & 0x7fffffu) << 29));
}
__device__ __forceinline__ double widen(float f) { return rare(f) ? widen_rare(f) : widen_common(f); }

// 0.0 + (double)f: as widen, with -0 turned into +0
__device__ __forceinline__ double widen_plus0(float f) {
  return (__float_as_uint(f) & 0x7fffffffu) == 0u ? 0.0 : widen(f);
}

// double -> float, round to nearest, ties to even, every case on the
// integer pipe: normal float results round the 52-bit mantissa to 23 bits;
// the others are a call: results below the normal range become float
// denormals (the 53-bit significand shifted into place, rounded the same
// way); |d| at or above 2^128 becomes inf; inf stays inf, NaN a quiet NaN
static __device__ __noinline__ float narrow_rare(double d) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(d);
  const unsigned sign = (unsigned)(u >> 32) & 0x80000000u;
  const int e = (int)((u >> 52) & 0x7ffu);
  const unsigned long long m = u & 0xfffffffffffffull;
  if (e == 0x7ff) return __uint_as_float(sign | 0x7f800000u | (m ? 0x400000u | (unsigned)(m >> 29) : 0u));
  if (e > 1150) return __uint_as_float(sign | 0x7f800000u);
  // |d| < 2^-126: d * 2^149 = M * 2^(e - 926) with M = 2^52 + m, rounded to
  // an integer (a carry into bit 23 gives the smallest normal float); double
  // denormals and everything below 2^-150 round to zero
  const int sh = 926 - e;  // >= 30
  if (e == 0 || sh >= 54) return __uint_as_float(sign);
  const unsigned long long M = (1ull << 52) | m;
  unsigned long long f = M >> sh;
  const unsigned long long rem = M & ((1ull << sh) - 1ull), half = 1ull << (sh - 1);
  if (rem > half || (rem == half && (f & 1ull))) f += 1ull;
  return __uint_as_float(sign | (unsigned)f);
}
__device__ __forceinline__ float narrow(double d) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(d);
  const unsigned hi = (unsigned)(u >> 32), lo = (unsigned)u;
  const unsigned sign = hi & 0x80000000u;
  const int e = (int)((hi >> 20) & 0x7ffu);
  // normal float results: biased float exponent e - 896 in [1, 254]
  if (e >= 897 && e <= 1150) {
    const unsigned rem = lo & 0x1fffffffu;  // the 29 bits dropped
    unsigned r = ((hi & 0x7fffffffu) << 3 | lo >> 29) - 0xc0000000u;
    if (rem > 0x10000000u || (rem == 0x10000000u && (r & 1u))) r += 1u;  // carry may reach the exponent
    return __uint_as_float(sign | r);  // a carry into exponent 255 is +-inf, as IEEE rounding gives
  }
  if ((u << 1) == 0ull) return __uint_as_float(sign);
  return narrow_rare(d);
}

// exact conversion To <- From between float and double on the integer pipe
// (narrowing rounds to nearest even), identity otherwise
template <typename To, typename From>
__device__ __forceinline__ To cvt(From v) {
  if constexpr (sizeof(To) == 8 && sizeof(From) == 4)
    return widen(v);
  else if constexpr (sizeof(To) == 4 && sizeof(From) == 8)
    return narrow(v);
  else
    return (To)v;
}

}  // namespace fpint
}  // namespace sayaka_gb300
