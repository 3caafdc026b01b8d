// Complex arithmetic in the reference's rounding, shared by the complex level-3
// routines and the LU panel.
#pragma once

#include <cfloat>

#include "ref_order.cuh"

namespace hb {
namespace {

template <typename R>
__device__ __forceinline__ R Mul(R x, R y) {
  if constexpr (sizeof(R) == 8) return __dmul_rn(x, y);
  else return __fmul_rn(x, y);
}
template <typename R>
__device__ __forceinline__ R Add(R x, R y) {
  if constexpr (sizeof(R) == 8) return __dadd_rn(x, y);
  else return __fadd_rn(x, y);
}
template <typename R>
__device__ __forceinline__ R Sub(R x, R y) {
  if constexpr (sizeof(R) == 8) return __dsub_rn(x, y);
  else return __fsub_rn(x, y);
}
template <typename R>
__device__ __forceinline__ R Fma(R x, R y, R z) {
  if constexpr (sizeof(R) == 8) return fma(x, y, z);
  else return fmaf(x, y, z);
}

// (a + i b) / (c + i d) as the C++ runtime's complex quotient: for double,
// Smith's method with its scalings for very large and very small magnitudes
// and its alternative when the ratio is subnormal; for float, the textbook
// quotient (a c + b d, b c - a d) / (c^2 + d^2) in double precision, rounded.
// (Checked against the host compiler's complex division on random quotients
// spanning 2^-60..2^60, zero parts included; non-finite inputs are not
// reproduced.)
template <typename R>
__device__ __forceinline__ void ZDiv(R ar, R ai, R cr, R ci, R* xr, R* xi) {
  if constexpr (sizeof(R) == 8) {
    double a = ar, b = ai, c = cr, d = ci;
    const double kBig = DBL_MAX / 2, kMin = DBL_MIN, kEps = DBL_EPSILON;
    const double kScale = 1.0 / kEps, kMax2 = kBig * kEps;
    double x, y;
    if (fabs(c) < fabs(d)) {
      if (fabs(d) >= kBig) {
        a = a / 2; b = b / 2; c = c / 2; d = d / 2;
      }
      if (fabs(d) < kEps) {
        a = a * kScale; b = b * kScale; c = c * kScale; d = d * kScale;
      } else if ((fabs(a) < kMin && fabs(b) < kMax2 && fabs(d) < kMax2) ||
                 (fabs(b) < kMin && fabs(a) < kMax2 && fabs(d) < kMax2)) {
        a = a * kScale; b = b * kScale; c = c * kScale; d = d * kScale;
      }
      const double ratio = c / d;
      const double denom = __dadd_rn(__dmul_rn(c, ratio), d);
      if (fabs(ratio) > kMin) {
        x = __dadd_rn(__dmul_rn(a, ratio), b) / denom;
        y = __dsub_rn(__dmul_rn(b, ratio), a) / denom;
      } else {
        x = __dadd_rn(__dmul_rn(c, a / d), b) / denom;
        y = __dsub_rn(__dmul_rn(c, b / d), a) / denom;
      }
    } else {
      if (fabs(c) >= kBig) {
        a = a / 2; b = b / 2; c = c / 2; d = d / 2;
      }
      if (fabs(c) < kEps) {
        a = a * kScale; b = b * kScale; c = c * kScale; d = d * kScale;
      } else if ((fabs(a) < kMin && fabs(b) < kMax2 && fabs(c) < kMax2) ||
                 (fabs(b) < kMin && fabs(a) < kMax2 && fabs(c) < kMax2)) {
        a = a * kScale; b = b * kScale; c = c * kScale; d = d * kScale;
      }
      const double ratio = d / c;
      const double denom = __dadd_rn(__dmul_rn(d, ratio), c);
      if (fabs(ratio) > kMin) {
        x = __dadd_rn(__dmul_rn(b, ratio), a) / denom;
        y = __dsub_rn(b, __dmul_rn(a, ratio)) / denom;
      } else {
        x = __dadd_rn(a, __dmul_rn(d, b / c)) / denom;
        y = __dsub_rn(b, __dmul_rn(d, a / c)) / denom;
      }
    }
    *xr = x;
    *xi = y;
  } else {
    const double a = ar, b = ai, c = cr, d = ci;
    const double den = __dadd_rn(__dmul_rn(c, c), __dmul_rn(d, d));
    const double re = __dadd_rn(__dmul_rn(a, c), __dmul_rn(b, d));
    const double im = __dsub_rn(__dmul_rn(b, c), __dmul_rn(a, d));
    *xr = static_cast<float>(re / den);
    *xi = static_cast<float>(im / den);
  }
}

// 1 / (c + i d): the quotient above with numerator (1, 0).
template <typename R>
__device__ __forceinline__ void ZRecip(R cr, R ci, R* xr, R* xi) {
  ZDiv<R>(R(1), R(0), cr, ci, xr, xi);
}

template <typename R>
__device__ __forceinline__ R ZMag(R re, R im) {
  return Add(fabs(re), fabs(im));
}

template <typename R>
__device__ __forceinline__ bool ZBetter(R v, int i, R bv, int bi) {
  return v > bv || (v == bv && v >= R(0) && i < bi);
}

// std::abs(z) >= s for the safe minimum s. |z| is at least the larger part,
// so only two parts below s need the magnitude itself: they are scaled by an
// exact power of two (double) or widened (float) and the square root of the
// sum of squares is compared in double precision. (std::abs is hypot: an
// infinite part gives infinity, otherwise a NaN part gives NaN.)
template <typename R>
__device__ __forceinline__ bool ZAbsAtLeast(R re, R im, R s) {
  const R ar = fabs(re), ai = fabs(im);
  if (isinf(ar) || isinf(ai)) return true;
  if (isnan(ar) || isnan(ai)) return false;
  if ((ar > ai ? ar : ai) >= s) return true;
  const double k = sizeof(R) == 8 ? 0x1p600 : 1.0;
  const double sr = __dmul_rn(static_cast<double>(ar), k);
  const double si = __dmul_rn(static_cast<double>(ai), k);
  const double mag = sqrt(__dadd_rn(__dmul_rn(sr, sr), __dmul_rn(si, si)));
  return mag >= __dmul_rn(static_cast<double>(s), k);
}

// y += alpha x for one element of a column of len complex elements.
template <typename R>
__device__ __forceinline__ void ZAxpyRef(R& yr, R& yi, R ar, R ai, R xr, R xi, int len,
                                         int lanes) {
  if (2 * len < lanes) {
    const R pr = Sub(Mul(ar, xr), Mul(ai, xi));
    const R pi = Add(Mul(ar, xi), Mul(ai, xr));
    yr = Add(yr, pr);
    yi = Add(yi, pi);
  } else {
    const R tr = Fma(xr, ar, yr), ti = Fma(xi, ar, yi);
    yr = Fma(xi, -ai, tr);
    yi = Fma(xr, ai, ti);
  }
}

}  // namespace
}  // namespace hb
