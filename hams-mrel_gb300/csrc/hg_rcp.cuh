// Correctly rounded reciprocal of a double on the integer and FP32 pipes.
//
// GB300 retires about two FP64 operations a clock and SM, and a correctly
// rounded 1/x costs several of them, so kernels made of reciprocals (Wynn's
// epsilon table: one per entry) are bound by that pipe while the integer pipes
// idle.  Here the reciprocal of the 53-bit significand is formed in fixed
// point: a single-precision seed (22 bits), two Newton steps y += y (1 - m y)
// in 64-bit integers (43 and then over 60 bits), and a final exact comparison
// of m (2 q + 1) with 2^106 that rounds the quotient q to nearest (a tie
// cannot occur).  Three 32-bit multiplies in the first step, five in the second
// and a 64-bit product at the end, about fifty instructions in all, none of them
// FP64.
//
// Same bits as 1.0 / x for every x whose reciprocal is a normal number
// (checked against it over random and boundary significands); rcp_in_range
// says which those are.
#pragma once
#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define HG_HD __host__ __device__ __forceinline__
#else
#define HG_HD inline
#endif

namespace hg {

HG_HD uint64_t rcp_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t b;
  memcpy(&b, &x, sizeof b);
  return b;
#endif
}
HG_HD double rcp_double(uint64_t b) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)b);
#else
  double x;
  memcpy(&x, &b, sizeof x);
  return x;
#endif
}

// Exponent field 1 .. 2043: x normal, its reciprocal too.
HG_HD bool rcp_in_range(uint64_t bits) { return (((uint32_t)(bits >> 52) & 0x7ffu) - 1u) <= 2042u; }

// seed: reciprocal of the significand's top 24 bits f in [1, 2), within a few
// units of the last place (float bits).
HG_HD uint32_t rcp_seed(uint32_t f) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(f)));
  return __float_as_uint(r);
#else
  float x, r;
  memcpy(&x, &f, 4);
  r = 1.0f / x;
  uint32_t b;
  memcpy(&b, &r, 4);
  return b;
#endif
}

HG_HD uint32_t rcp_umulhi(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }

// 1 / x for rcp_in_range(bits of x).
HG_HD double rcp_from_seed(uint64_t b, uint32_t rb) {
  const uint32_t ex = (uint32_t)(b >> 52) & 0x7ffu;
  const uint64_t m = (b & 0xfffffffffffffull) | 0x10000000000000ull;
  const uint64_t M = m << 11;  // significand / 2^63 in [1, 2)
  const uint32_t Mh = (uint32_t)(M >> 32), Ml = (uint32_t)M;
  const uint32_t R = ((rb & 0x7fffffu) | 0x800000u) << ((rb >> 23) - 119u);  // seed 2^31
  // e = 2^62 (1 - m y): |e| < 2^41
  const int64_t e = (int64_t)((1ull << 62) - ((uint64_t)Mh * R + rcp_umulhi(Ml, R)));
  const int32_t es = (int32_t)(e >> 16);
  const uint64_t Y = ((uint64_t)R << 32) + (uint64_t)(((int64_t)(int32_t)(R >> 1) * es) >> 13);
  // bits 54.. of 2^126 - M Y, which is below 2^84 in magnitude
  const uint32_t Yh = (uint32_t)(Y >> 32), Yl = (uint32_t)Y;
  const uint64_t t = (uint64_t)Mh * Yl + (uint64_t)Ml * Yh + rcp_umulhi(Ml, Yl);
  const uint32_t hi = Mh * Yh + (uint32_t)(t >> 32);
  const int32_t e2 = (int32_t)((0u - hi) << 10) - (int32_t)((uint32_t)t >> 22);
  const uint64_t Y2 = Y + (uint64_t)(((int64_t)(int32_t)(Yh >> 1) * e2) >> 39);
  // q within one of 2^105 / m; up where 2^105 / m lies above q + 1/2
  uint64_t q = Y2 >> 10;
  q += (int64_t)(0ull - m * (2 * q + 1)) > 0 ? 1 : 0;
  return rcp_double((b & 0x8000000000000000ull) | (((uint64_t)(2044u - ex) << 52) + q));
}

HG_HD double rcp_rn(double x) {
  const uint64_t b = rcp_bits(x);
  return rcp_from_seed(b, rcp_seed(0x3f800000u | ((uint32_t)(b >> 29) & 0x7fffffu)));
}

// 1 / x for any x.
HG_HD double rcp_any(double x) { return rcp_in_range(rcp_bits(x)) ? rcp_rn(x) : 1.0 / x; }

HG_HD float rsqrt_seed(float f) {
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  return r;
#else
  return 1.0f / sqrtf(f);
#endif
}

// Where the seed and the steps' products are normal: 2^-122 to 2^122.
HG_HD bool rsqrt_in_range(double x) { return (uint32_t)(rcp_bits(x) >> 32) - 0x38500000u < 0x0f500000u; }

// 1 / sqrt(x), x >= 0, within a unit of the last place: a single-precision
// seed (22 bits) and one step of Householder's third-order iteration (1970) for
// 1 / y^2 - x, y (1 + e / 2 + 3 e^2 / 8) with e = 1 - x y^2, five FP64
// operations against about twenty for 1.0 / sqrt(x).  Outside the seed's range
// the latter.
HG_HD double rsqrt_from_seed(double x, double y) {
  const double e = fma(-x * y, y, 1.0);
  return fma(fma(e, 0.375, 0.5) * e, y, y);
}
HG_HD double rsqrt_near(double x) {
  return rsqrt_in_range(x) ? rsqrt_from_seed(x, (double)rsqrt_seed((float)x)) : 1.0 / sqrt(x);
}

// sqrt(x) from ix near 1 / sqrt(x) (0 for x = 0): half the exact residual of
// x ix, times ix, rounds it (Markstein 1990).  Exact roots come out exactly.
HG_HD double root_of(double x, double ix) {
  const double r = x * ix;
  return fma(fma(-r, r, x), 0.5 * ix, r);
}

// sqrt(x), x >= 0, rounded the same way, where its reciprocal is not needed: one
// coupled Newton step (Goldschmidt 1964) on the seed's root and half reciprocal,
// then the residual, seven FP64 operations.
HG_HD double sqrt_from_seed(double x, double y) {
  double g = x * y, h = 0.5 * y;
  const double r = fma(-g, h, 0.5);
  g = fma(g, r, g);
  h = fma(h, r, h);
  return fma(fma(-g, g, x), h, g);
}
HG_HD double sqrt_near(double x) { return rsqrt_in_range(x) ? sqrt_from_seed(x, (double)rsqrt_seed((float)x)) : sqrt(x); }

}  // namespace hg
