// Device helpers that fix the reference's rounding in the LU kernels (shared
// by the single-problem and the batched factorizations).
#pragma once

#include <cfloat>

namespace hb {
namespace {

template <typename T>
__device__ __forceinline__ T Sfmin();
template <>
__device__ __forceinline__ double Sfmin<double>() { return DBL_MIN; }
template <>
__device__ __forceinline__ float Sfmin<float>() { return FLT_MIN; }

// y + alpha*x in the reference's rounding for a column of length len: shorter
// than one SIMD vector of the reference's target, two roundings; otherwise
// one FMA (src/lapack/factor_kernels.cc:79-118).
template <typename T>
__device__ __forceinline__ T Axpy(T y, T alpha, T x, int len, int lanes) {
  if (len < lanes) {
    const T p = alpha * x;
    return y + p;
  }
  return fma(x, alpha, y);
}

// (value, index) candidates: larger value wins, then the smaller index.
// value < 0 marks "no candidate" (no rows, or only NaNs).
template <typename T>
__device__ __forceinline__ bool Better(T v, int i, T bv, int bi) {
  return v > bv || (v == bv && v >= T(0) && i < bi);
}

// Order of the pivot search: larger |x|, NaN below everything (0).
__device__ __forceinline__ unsigned long long PivotKey(double x) {
  const unsigned long long v = __double_as_longlong(x) & 0x7fffffffffffffffull;
  return v > 0x7ff0000000000000ull ? 0ull : v + 1;
}
__device__ __forceinline__ unsigned long long PivotKey(float x) {
  const unsigned v = __float_as_uint(x) & 0x7fffffffu;
  return v > 0x7f800000u ? 0ull : static_cast<unsigned long long>(v) + 1;
}

// The lane with the warp's largest key, the one with the smallest position if
// several hold it (kWide: 64-bit keys, whose high words nearly always decide).
template <bool kWide>
__device__ __forceinline__ int WarpBest(unsigned long long key, int pos) {
  const unsigned lo = static_cast<unsigned>(key), hi = static_cast<unsigned>(key >> 32);
  const unsigned word = kWide ? hi : lo;
  const unsigned largest = __reduce_max_sync(0xffffffffu, word);
  unsigned top = __ballot_sync(0xffffffffu, word == largest);
  if (top & (top - 1)) {
    const bool in = (top >> (threadIdx.x % 32)) & 1;
    const unsigned second = kWide && in ? lo : 0u;
    const unsigned most = __reduce_max_sync(0xffffffffu, second);  // by every lane
    const bool in2 = in && second == most;
    const int first = __reduce_min_sync(0xffffffffu, in2 ? pos : 0x7fffffff);
    top = __ballot_sync(0xffffffffu, in2 && pos == first);
  }
  return __ffs(top) - 1;
}

}  // namespace
}  // namespace hb
