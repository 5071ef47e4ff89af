// hyc_device.cuh -- device-side helpers shared by the advection kernels.
//
// Reference layout (mod_cb_arrays.F90, mod_dimensions.F90): a 2-D slice is
// a(1-nbdy:idm+nbdy, 1-nbdy:jdm+nbdy), column-major.  Fortran (i,j) maps to
// offset (i+nbdy-1) + (j+nbdy-1)*ld1.
//
// Comparisons on the FP64 data run on the integer pipes.  On GB300 the FP64
// pipe issues about 1/72 of the FP32 rate (a DMNMX or DSETP costs as much
// as a DFMA), while 64-bit integer compares and selects run an order of
// magnitude faster, so min/max/sign tests are done on the IEEE bit patterns.
// For non-NaN doubles the map  key(x) = bits(x) ^ ((bits(x) >> 63) >>> 1)
// is strictly increasing in x (with -0 just below +0), so a signed 64-bit
// compare of keys orders doubles.  Results equal the reference's
// max()/min() except possibly in the sign of a zero, which never changes a
// later value of this path (no division by these zeros happens).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "hyc_div.cuh"

namespace hyc {

constexpr double kOnemu = 9806.e-12;  // 1 micrometre in Pa, mod_tsadvc.F90:236
constexpr double kEpsil = 1.e-10;     // mod_tsadvc.F90:1027

__device__ __forceinline__ long long dkey(double x) {
  long long b = __double_as_longlong(x);
  return b ^ ((long long)((unsigned long long)(b >> 63) >> 1));
}
__device__ __forceinline__ double from_dkey(long long k) {  // dkey is its own inverse
  return __longlong_as_double(k ^ (long long)((unsigned long long)(k >> 63) >> 1));
}
constexpr long long kOneBits = 0x3FF0000000000000LL;  // 1.0
// max(a,b) / min(a,b) of the reference (mod_tsadvc.F90 passim)
__device__ __forceinline__ double kmax(double a, double b) { return dkey(a) > dkey(b) ? a : b; }
__device__ __forceinline__ double kmin(double a, double b) { return dkey(a) < dkey(b) ? a : b; }
// max(0.0,x) and min(0.0,x)
__device__ __forceinline__ double pos0(double x) { return __double_as_longlong(x) > 0 ? x : 0.0; }
__device__ __forceinline__ double neg0(double x) { return __double_as_longlong(x) < 0 ? x : 0.0; }
// x >= 0.0 (true for -0.0 too), x < 0.0 (false for -0.0), x > 0.0
__device__ __forceinline__ bool ge0(double x) {
  long long b = __double_as_longlong(x);
  return b >= 0 || b == (long long)0x8000000000000000ULL;
}
__device__ __forceinline__ bool lt0(double x) {
  long long b = __double_as_longlong(x);
  return b < 0 && b != (long long)0x8000000000000000ULL;
}
__device__ __forceinline__ bool gt0(double x) { return __double_as_longlong(x) > 0; }
__device__ __forceinline__ bool klt(double a, double b) { return dkey(a) < dkey(b); }

// FP32 bounds of a double for tests that need no exact value (integer pipes:
// a conversion instruction would issue at the FP64 rate).  Both truncate
// towards zero (relative error below 2^-23).  f32_below: of a value >= 0, at
// most x, and 0 where x is negative, NaN or outside FP32's normal range.
__device__ __forceinline__ float f32_below(double x) {
  const uint32_t h = (uint32_t)__double2hiint(x);
  const uint32_t f = __funnelshift_l((uint32_t)__double2loint(x), h, 3) + 0x40000000u;
  return h - 0x38100000u < 0x0FE00000u ? __uint_as_float(f) : 0.0f;
}
// f32_away: away from zero where it matters, not in the last bit: 0 only where
// x is 0, below FP32's normal range the smallest normal, above it (and for NaN)
// infinity; in the range the truncation leaves it up to 2^-23 short, which the
// tests' factors (1.000004) cover
__device__ __forceinline__ float f32_away(double x) {
  const uint32_t h = (uint32_t)__double2hiint(x), l = (uint32_t)__double2loint(x), m = h & 0x7FFFFFFFu;
  uint32_t f = __funnelshift_l(l, h, 3) + 0x40000000u;
  if (m - 0x38100000u >= 0x0FE00000u) f = m > 0x38100000u ? 0x7F800000u : (m | l) != 0 ? 0x00800000u : 0u;
  return __uint_as_float(f | (h & 0x80000000u));
}

// FP32 versions (FMNMX is cheap on the FP32 pipe)
__device__ __forceinline__ float kmax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ float kmin(float a, float b) { return fminf(a, b); }
__device__ __forceinline__ float pos0(float x) { return fmaxf(x, 0.0f); }
__device__ __forceinline__ float neg0(float x) { return fminf(x, 0.0f); }
__device__ __forceinline__ bool ge0(float x) { return x >= 0.0f; }
__device__ __forceinline__ bool lt0(float x) { return x < 0.0f; }
__device__ __forceinline__ bool gt0(float x) { return x > 0.0f; }
__device__ __forceinline__ bool klt(float a, float b) { return a < b; }

// Correctly rounded q/h given r = RN(1/h) (one reciprocal per cell shared by
// every tracer of the layer): y = RN(q*r) and one residual correction,
// RN(y + r*RN(q - h*y)) = RN(q/h) bit for bit for normal operands.
// Markstein's theorem gives this for a faithful y (below 1 ulp off), which
// RN(q*r) is where the significands satisfy q >= h.  Where q < h (take
// 1 <= h, q < 2, ulp(q/h) = 2^-53), y may be up to (q+1)/2 < 1.5 ulp off.
// With q/h = m + K*2^-106/h, m a midpoint and K odd, rounding to the wrong
// side of m needs |K| < 2|RN(e) - e|*2^105 + 2|RN(e)|*|r - 1/h|*h*2^105 for the
// residual e: with y at the nearer distance of 1/2 ulp from m, e is exact
// and the bound is below 1, and |K| >= 1; at 3/2 ulp it is below 2 + 3, but
// y lies there only if q >= 2 - |K|*2^-52/h, and q <= h - 2^-52 < 2 - 2^-52 then
// requires |K| >= 5.  1 DMUL + 2 DFMA.
__device__ __forceinline__ double div_rcp(double q, double h, double r) {
  const double y = __dmul_rn(q, r);
  return __fma_rn(__fma_rn(-y, h, q), r, y);
}

}  // namespace hyc
