// Scalar conversions and the logarithm of the scoring kernels: FP64 arithmetic, conversions
// included, runs at a few lanes per clock and SM, so these do with integers what they can.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "internal.h"

namespace tp3 {
namespace {

// log(x) of a positive normal double, table-driven (P. T. P. Tang, "Table-driven implementation
// of the logarithm function in IEEE floating-point arithmetic", ACM TOMS 16 (1990)): x = 2^e m
// with 0.75 <= m < 1.5, c the centre of m's interval (1/128 of its binade), r = m (1/c) - 1 with
// one rounding, log x = e ln 2 + log c + log1p(r), |r| < 2^-8.  14 FP64 operations, a third of
// log(): FP64 runs at two lanes per clock and SM here.  Within 2^-53 |log x| + 2^-60: the rounding of
// the result and of r (the first sum is exact, the series ends at r^8 / 8 < 2^-67).  tab: 1/c and
// log c, built in extended precision.
__device__ __forceinline__ double slab_log(const double x, const SlabLog* __restrict__ tab) {
  const int hi = __double2hiint(x);
  const int e = ((hi >> 20) & 0x7ff) - 1023;
  if (e < -1022 || e > 1023 || hi < 0) return log(x);  // zero, subnormal, infinite, NaN, negative
  const double m = __hiloint2double((hi & 0xfffff) | 0x3ff00000, __double2loint(x));
  const int i = (hi >> 13) & 127;
  const double inv = tab[i].inv, chi = tab[i].hi, clo = tab[i].lo;
  const double r = fma(m, inv, -1.0), r2 = r * r;
  double p = fma(r, 1.0 / 7.0, -1.0 / 6.0);
  p = fma(p, r, 0.2);
  p = fma(p, r, -0.25);
  p = fma(p, r, 1.0 / 3.0);
  p = fma(p, r, -0.5);
  const double ed = (double)(e + (i >> 6));
  constexpr double ln2_hi = 0x1.62e42fefa38p-1, ln2_lo = 0x1.ef35793c7673p-45;  // ln 2 to 41 + 53 bits
  return fma(ed, ln2_hi, chi) + (r + fma(p, r2, fma(ed, ln2_lo, clo)));  // the first sum is exact
}

// (double)x by integer arithmetic (exact); zeros, subnormals and non-finite values go through
// the conversion, which runs at FP64 rate.
__device__ __forceinline__ double widen(const float x) {
  const uint32_t u = __float_as_uint(x);
  const uint32_t e = (u >> 23) & 255;
  if (e == 0 || e == 255) return (double)x;
  return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20))), (int)(u << 29));
}

// (float)x by integer arithmetic: FP64 conversions, like all FP64 arithmetic, run at a few
// lanes per clock and SM.  Round to nearest even; subnormal and non-finite results go through
// the conversion.
__device__ __forceinline__ float narrow(const double x) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const int e = (int)((hi >> 20) & 0x7ff) - 1023 + 127;
  if (e >= 1 && e <= 254) {
    const uint32_t m = ((hi & 0xfffff) << 3) | (lo >> 29), rem = lo & 0x1fffffff;
    const uint32_t up = rem > 0x10000000u || (rem == 0x10000000u && (m & 1)) ? 1u : 0u;
    return __uint_as_float((hi & 0x80000000u) | (((uint32_t)e << 23) + m + up));
  }
  return ((hi << 1) | lo) == 0 ? __uint_as_float(hi & 0x80000000u) : (float)x;
}

}  // namespace
}  // namespace tp3
