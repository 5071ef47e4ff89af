// hyc_div.cuh -- IEEE double division (round to nearest) on the integer pipes.
//
// GB300 issues FP64 at about 1/70 of the FP32 rate (1.6 operations per SM
// and clock), so a hardware double division, a chain of dependent FP64
// FMAs, holds the FP64 pipe longer than the ~60 integer instructions of a
// long division hold the integer pipes -- and the FP64 pipe is what bounds
// the kernels that divide.  div_rn forms the same correctly rounded
// quotient with no FP64 operation: 287e9 divisions/s against the hardware
// division's 69e9 in a loop of nothing else.  In the kernels (FCT2 on
// 4500x3298x41: 179.7 -> 139.3 ms; cnuity on 1500x1100x41: 25.0 -> 20.1 ms;
// the tracer step there: 42.2 -> 34.0 ms) it comes with the three-operation
// div_rcp of hyc_device.cuh.
//
// Method: schoolbook long division of the 53-bit significands in two digits
// (31 and 27 bits), each digit estimated from a 32-bit reciprocal that is
// never too large (hardware FP32 seed, one integer Newton step), then one
// exact remainder comparison.  With N/m in [1,2) (N the dividend's
// significand, doubled when it is the smaller):
//   R  in (r-6.1, r],  r = 2^84/m            (32 bits)
//   Q1 in (t-8.1, t],  t = N*2^30/m          remainder N*2^30 - Q1*m < 8.1 m
//   Q2 within 1.3 below the second digit      remainder < 1.3 m
// so floor(N*2^53/m) = Q1*2^23 + Q2 + (remainder >= m), 54 bits, and the
// result is that number rounded at its last bit (a tie would need m to be a
// multiple of 2^53).  The remainders are small, so 64-bit arithmetic modulo
// 2^64 holds them.  Operands outside 2^-500 .. 2^500 (other than a zero
// dividend) take the hardware division, which covers infinities, NaNs,
// subnormals and over- and underflow.
//
// mul_rn is the multiplication in the same manner, about 30 integer
// instructions for an operation that holds the FP64 pipe 16 clocks of an SM:
// it pays where the integer pipes are idle, not everywhere (each kernel says
// which products it takes).  The fallbacks are real calls: as plain
// expressions the compiler predicates them into the main path, where a
// predicated-off FP64 instruction holds the pipe all the same (FCT2 on
// 4500x3298x41: 90 ms against 80 ms).
#pragma once
#include <cstdint>
#include <cstring>
#include <cmath>

#ifdef __CUDACC__
#define HYC_HD __host__ __device__ __forceinline__
#else
#define HYC_HD inline
#endif

namespace hyc {

namespace idiv {

HYC_HD uint32_t f2u(float f) {
#ifdef __CUDA_ARCH__
  return __float_as_uint(f);
#else
  uint32_t u;
  memcpy(&u, &f, 4);
  return u;
#endif
}
HYC_HD float u2f(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float f;
  memcpy(&f, &u, 4);
  return f;
#endif
}
HYC_HD uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
HYC_HD double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
HYC_HD uint32_t mulhi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
HYC_HD int32_t mulhi_s(int32_t a, int32_t b) {
#ifdef __CUDA_ARCH__
  return __mulhi(a, b);
#else
  return (int32_t)(((int64_t)a * b) >> 32);
#endif
}
// q*m modulo 2^64
HYC_HD uint64_t mul_lo(uint32_t q, uint64_t m) {
  return (uint64_t)q * (uint32_t)m + ((uint64_t)(q * (uint32_t)(m >> 32)) << 32);
}
// FP32 reciprocal seed of x in [1,2), relative error below 2^-22 (the
// hardware's approximate reciprocal is within 1 ulp)
HYC_HD float seed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return 1.0f / x;
#endif
}
// the FP64 pipe's own operations, for operands out of range
#ifdef __CUDACC__
static __device__ __noinline__ double slow_mul(double a, double b) { return a * b; }
static __device__ __noinline__ double slow_div(double a, double b) { return a / b; }
static __device__ __noinline__ double slow_sqrt(double a) { return sqrt(a); }
#endif
HYC_HD double fp64_mul(double a, double b) {
#ifdef __CUDA_ARCH__
  return slow_mul(a, b);
#else
  return a * b;
#endif
}
HYC_HD double fp64_div(double a, double b) {
#ifdef __CUDA_ARCH__
  return slow_div(a, b);
#else
  return a / b;
#endif
}
HYC_HD double fp64_sqrt(double a) {
#ifdef __CUDA_ARCH__
  return slow_sqrt(a);
#else
  return sqrt(a);
#endif
}
// FP32 reciprocal square root of x in [1,4), relative error below 2^-21.7
// (the hardware's approximation is within 2 ulp)
HYC_HD float rseed(float x) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return (float)(1.0 / sqrt((double)x));
#endif
}
HYC_HD uint64_t significand(uint64_t b) { return (b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull; }

// 32-bit reciprocal of a significand m in [2^52, 2^53): in (r-6.1, r], r = 2^84/m.
// The seed's argument is m's top 24 bits with the last one set: at least
// 1 + 2^-23, so the seed is below 1 and its significand is all of R0.
HYC_HD uint32_t recip32(uint64_t m) {
  const float rf = seed(u2f(0x3F800001u | ((uint32_t)(m >> 29) & 0x7FFFFFu)));
  const uint32_t R0 = 0x80000000u | (f2u(rf) << 8);
  const uint32_t x = (uint32_t)(m >> 21);
  // e = 2^63 - R0*x, |e| < 2^42; R0*(1 + e/2^63) is the Newton step
  const int32_t e = (int32_t)((0x8000000000000000ull - (uint64_t)R0 * x) >> 32);
  return R0 + (uint32_t)mulhi_s((int32_t)(R0 >> 1), e * 4) - 3u;
}

// significand of RN(N/m) (bit 52 set), N/m in [1,2), R = recip32(m)
HYC_HD uint64_t quotient(uint64_t N, uint64_t m, uint32_t R) {
  const uint32_t q1 = mulhi((uint32_t)(N >> 22), R);
  const uint64_t r1 = (N << 30) - mul_lo(q1, m);
  const uint32_t q2 = mulhi((uint32_t)(r1 >> 25), R) >> 4;
  const uint64_t r2 = (r1 << 23) - mul_lo(q2, m);
  const uint64_t q = ((uint64_t)q1 << 23) + q2 + (r2 >= m ? 1u : 0u);
  return (q + 1) >> 1;
}

// exponent field in [1023-500, 1023+500): every quotient of two such values is normal
HYC_HD bool mid_range(uint32_t hi) { return (hi & 0x7FFFFFFFu) - 0x20B00000u < 0x3E800000u; }

}  // namespace idiv

// R of a divisor that several dividends share; 0 sends them to the hardware division
HYC_HD uint32_t recip_of(double b) {
  const uint64_t ib = idiv::bits(b);
  return idiv::mid_range((uint32_t)(ib >> 32)) ? idiv::recip32(idiv::significand(ib)) : 0u;
}

// a/b, correctly rounded; R = recip_of(b)
HYC_HD double div_by(double a, double b, uint32_t R) {
  using namespace idiv;
  const uint64_t ia = bits(a), ib = bits(b);
  const uint32_t ha = (uint32_t)(ia >> 32), hb = (uint32_t)(ib >> 32);
  const bool zero = (ia << 1) == 0;
  if (!(R != 0 && (mid_range(ha) || zero))) return fp64_div(a, b);
  const uint64_t ma = significand(ia), mb = significand(ib);
  const bool less = ma < mb;
  const uint64_t q = quotient(less ? ma << 1 : ma, mb, R);
  const uint32_t sgn = (ha ^ hb) & 0x80000000u;
  // (exponent - 1) << 20, added onto the significand's own bit 52
  const uint32_t ex = (ha & 0x7FF00000u) - (hb & 0x7FF00000u) + (less ? 0x3FD00000u : 0x3FE00000u);
  const uint64_t r = q + ((uint64_t)(ex | sgn) << 32);
  return from_bits(zero ? (uint64_t)sgn << 32 : r);
}
HYC_HD double div_rn(double a, double b) { return div_by(a, b, recip_of(b)); }
// 1/b, correctly rounded
HYC_HD double rcp_rn(double b) { return div_rn(1.0, b); }

namespace idiv {
// The product of the significands a (53 bits) and b, rounded half to even to
// 53 bits (2^53 where it rounds up to that), from four 32x32-bit products
// with b shifted up 11 bits, so that its top 52 or 53 bits are the upper
// 64-bit half; sh = 1 where they were 52 (the product below 2).  a = 2^53, a
// product rounded up, is as good as 2^52 one exponent higher.
HYC_HD uint64_t product(uint64_t a, uint64_t b, uint32_t &sh) {
  const uint32_t al = (uint32_t)a, ah = (uint32_t)(a >> 32);
  const uint32_t bl = (uint32_t)(b << 11), bh = (uint32_t)(b >> 21);
  const uint64_t t0 = (uint64_t)al * bl;
  const uint64_t t1 = (uint64_t)al * bh + (t0 >> 32);
  const uint64_t t2 = (uint64_t)ah * bl + (uint32_t)t1;
  const uint64_t hi = (uint64_t)ah * bh + (t1 >> 32) + (t2 >> 32);  // in [2^51, 2^53)
  const uint32_t m = (uint32_t)t2;
  sh = 1u ^ (uint32_t)(hi >> 52);
  const uint64_t q = hi << sh | (sh & (m >> 31));
  // the rest, its sticky bits folded into the last one
  const uint32_t rest = m << sh | ((uint32_t)t0 != 0 ? 1u : 0u);
  return q + (((uint64_t)rest + 0x7FFFFFFFu + ((uint32_t)q & 1u)) >> 32);
}
}  // namespace idiv

// a*b, correctly rounded.  Out of range, zeros too: the FP64 multiply.
HYC_HD double mul_rn(double a, double b) {
  using namespace idiv;
  const uint64_t ia = bits(a), ib = bits(b);
  const uint32_t ha = (uint32_t)(ia >> 32), hb = (uint32_t)(ib >> 32);
  if (!(mid_range(ha) && mid_range(hb))) return fp64_mul(a, b);
  uint32_t sh;
  const uint64_t q = product(significand(ia), significand(ib), sh);
  // exponents and signs add; -1 for the significand's own bit 52
  const uint32_t ex = (ha & 0xFFF00000u) + (hb & 0xFFF00000u) - 0x3FF00000u - (sh << 20);
  return from_bits(q + ((uint64_t)ex << 32));
}

// x/2 and 2x, exact
HYC_HD double half_of(double x) {
  const uint64_t b = idiv::bits(x);
  return idiv::mid_range((uint32_t)(b >> 32)) ? idiv::from_bits(b - (1ull << 52)) : idiv::fp64_mul(x, 0.5);
}
HYC_HD double twice_of(double x) {
  const uint64_t b = idiv::bits(x);
  return idiv::mid_range((uint32_t)(b >> 32)) ? idiv::from_bits(b + (1ull << 52)) : idiv::fp64_mul(x, 2.0);
}

// sqrt(x), correctly rounded, on the integer pipes.  x = M*2^2k, M in
// [2^52, 2^54); q = floor(sqrt(M*2^54)) has 54 bits and its last one rounds
// (no square root of 53 bits lies halfway).  q = a*2^26 + b: a, 28 bits, from
// the FP32 seed y = 1/sqrt and one Newton step (within 2), b from the
// remainder r = 4M - a^2 times y (within 70), then from the exact remainder
// again (within 1), which also settles the last unit.  The remainders are
// below 2^62, so arithmetic modulo 2^64 holds them.
HYC_HD double sqrt_rn(double x) {
  using namespace idiv;
  const uint64_t ib = bits(x);
  const uint32_t h = (uint32_t)(ib >> 32);
  if (!(mid_range(h) && (int32_t)h > 0)) return fp64_sqrt(x);
  const uint32_t odd = ~(h >> 20) & 1u;  // of the unbiased exponent
  const uint64_t M = significand(ib) << odd;
  const float xf = u2f(((127u + odd) << 23) | ((uint32_t)(ib >> 29) & 0x7FFFFFu));
  const float y = fminf(fmaxf(rseed(xf), 0.5f), 0.99999994f);        // in [0.5, 1)
  const float af = fminf(fmaxf(xf * y, 1.0f), 1.9999999f);          // sqrt, in [1, 2)
  const int32_t yi = (int32_t)((f2u(y) & 0x7FFFFFu) | 0x800000u);   // y*2^24
  const uint32_t a0 = ((f2u(af) & 0x7FFFFFu) | 0x800000u) << 4;     // sqrt*2^27
  const uint64_t H = M << 2;
  const int64_t d = (int64_t)(H - (uint64_t)a0 * a0);
  const uint32_t a = a0 + (uint32_t)(mulhi_s((int32_t)(d >> 6), yi) >> 14);
  const int32_t r = (int32_t)(uint32_t)(H - (uint64_t)a * a);
  const int32_t b = mulhi_s(r, yi << 6);
  const uint64_t Q = ((uint64_t)a << 26) + (uint64_t)(int64_t)b;
  const uint64_t rem = ((uint64_t)(uint32_t)r << 52) - (uint64_t)(int64_t)b * (Q + ((uint64_t)a << 26));
  const int32_t db = mulhi_s((int32_t)((int64_t)rem >> 34), yi << 6) >> 18;
  uint64_t q = Q + (uint64_t)(int64_t)db;
  const int64_t rem1 = (int64_t)(rem - (uint64_t)(int64_t)db * (Q + q));
  q = rem1 < 0 ? q - 1 : rem1 > (int64_t)(q << 1) ? q + 1 : q;
  const uint32_t ex = (((h >> 20) + 1u) >> 1) + 510u;  // the result's exponent field, less one for bit 52
  return from_bits(((q + 1) >> 1) + ((uint64_t)ex << 52));
}

}  // namespace hyc
