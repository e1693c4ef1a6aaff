// Integer digits of FP64 values and back (Ozaki's fixed-point splitting),
// shared by the tensor-core products at FP64 accuracy.
#pragma once
#include <cuda_runtime.h>

namespace bg {
namespace {

// 8 signed base-128 digits of round(|v| 2^(56 - f)) (|v| <= 2^(f - 1)): the
// top digit in [0, 64], the others in [-64, 63], then the sign of v. Integer
// arithmetic only (the FP64 pipe is the slow one).
__device__ __forceinline__ void oz_digits(double v, int f, int* d) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(v);
  const int be = (int)((bits >> 52) & 0x7FF);
  const unsigned long long mant = bits & ((1ull << 52) - 1);
  unsigned long long m = be ? (mant | (1ull << 52)) : mant;
  const int sh = (be ? be - 1075 : -1074) - f + 56;  // |v| 2^(56 - f) = m 2^sh, sh <= 2
  unsigned long long V;
  if (m == 0) V = 0;
  else if (sh >= 0) V = m << sh;
  else if (sh > -63) V = (m + (1ull << (-sh - 1))) >> (-sh);
  else V = 0;
  int carry = 0;
#pragma unroll
  for (int k = 7; k >= 1; --k) {
    int dk = (int)((V >> (7 * (7 - k))) & 127) + carry;
    carry = dk >= 64;
    d[k] = carry ? dk - 128 : dk;
  }
  d[0] = (int)(V >> 49) + carry;
  if (bits >> 63) {
#pragma unroll
    for (int k = 0; k < 8; ++k) d[k] = -d[k];
  }
}

// v 2^k as FP64 for a 64-bit integer v (round to nearest even); integer
// arithmetic except outside the normal range
__device__ __forceinline__ double oz_to_double(long long v, int k) {
  if (v == 0) return 0.0;
  const unsigned long long sgn = v < 0 ? (1ull << 63) : 0ull;
  const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  int top = 63 - __clzll((long long)a);
  unsigned long long m;
  if (top > 52) {
    const int sh = top - 52;
    const unsigned long long rem = a & ((1ull << sh) - 1), half = 1ull << (sh - 1);
    m = a >> sh;
    if (rem > half || (rem == half && (m & 1))) {
      ++m;
      if (m == (1ull << 53)) {
        m >>= 1;
        ++top;
      }
    }
  } else {
    m = a << (52 - top);
  }
  const int ex = top + k + 1023;
  if (ex <= 0 || ex >= 2047) return ldexp((double)v, k);
  return __longlong_as_double((long long)(sgn | ((unsigned long long)ex << 52) | (m & ((1ull << 52) - 1))));
}

}  // namespace
}  // namespace bg
