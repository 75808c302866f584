// fixed_point.cuh -- FP64 values as integers of a common exponent, on the integer
// pipe.
#pragma once

#include <cuda_runtime.h>

namespace hg {

// exponents (exp_of) of a group of values with an infinite or NaN one; of zeros only
constexpr int kNoScale = 1 << 20, kZeroExp = -(1 << 20);
// v 2^r as an integer x with |x| <= 2^(52 + kUp + 1), v 2^r = x 2^(em - 1075 - kUp), em
// the largest exponent (exp_of) of the group, rounded to nearest
template <int kUp>
__device__ __forceinline__ long long to_fixed(double v, int r, int em) {
  unsigned long long const b = (unsigned long long)__double_as_longlong(v);
  int const f = (int)((b >> 52) & 0x7FFu);
  unsigned long long const m = (b & 0xFFFFFFFFFFFFFull) | (f ? 1ull << 52 : 0ull);
  int const sh = em - (f ? f : 1) - r;
  unsigned long long x = m << kUp;
  if (sh > 0) x = sh > 60 ? 0ull : (x + (1ull << (sh - 1))) >> sh;
  return (b >> 63) ? -(long long)x : (long long)x;
}
// the biased exponent of v 2^r (no FP64 comparison: that pipe is the slow one)
__device__ __forceinline__ int exp_of(double v, int r) {
  int const hi = __double2hiint(v) & 0x7FFFFFFF, f = hi >> 20;
  return f == 0x7FF ? kNoScale : ((hi | __double2loint(v)) == 0 ? kZeroExp : max(f, 1) + r);
}
// 2^e, to zero or infinity beyond FP64's range
__device__ __forceinline__ double pow2(int e) {
  return e >= -1022 && e <= 1023 ? __hiloint2double((e + 1023) << 20, 0) : ldexp(1.0, max(-2000, min(2000, e)));
}

}  // namespace hg
