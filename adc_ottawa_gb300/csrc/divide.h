// Correctly rounded FP64 division without the FP64 pipe (GB300: 2 operations
// per cycle and SM, and a division is about nine of them).
//
// Schoolbook: a quotient estimate from single-precision arithmetic (within a
// hundred units of the last place), its exact remainder from 64-bit integers, a
// small integer correction, round to nearest even from the remainder.  Every
// step after the estimate is exact, so the result does not depend on the
// accuracy of the hardware's reciprocal: any within 2^-21 relative keeps the
// remainder inside 63 bits (rcp.approx is documented to 2^-23).
// tests/test_divide.py compares it with the host's division.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define ADC_DIV_FN __host__ __device__ __forceinline__
#else
#define ADC_DIV_FN static inline
#endif

namespace adcgpu {

ADC_DIV_FN uint64_t div_bits(double x) {
#ifdef __CUDA_ARCH__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
ADC_DIV_FN double div_double(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
ADC_DIV_FN float div_float(uint32_t u) {
#ifdef __CUDA_ARCH__
  return __uint_as_float(u);
#else
  float x;
  memcpy(&x, &u, 4);
  return x;
#endif
}
// 1 / x for x in [1, 2), about 2^-22 relative
ADC_DIV_FN float div_rcp(float x, float host_error) {
#ifdef __CUDA_ARCH__
  (void)host_error;
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
#else
  return (1.0f / x) * (1.0f + host_error);   // the test varies the estimate
#endif
}

ADC_DIV_FN double div_rn(double n, double d, float host_error = 0.0f) {
  const uint64_t un = div_bits(n), ud = div_bits(d);
  const int en = (int)((un >> 52) & 0x7ff), ed = (int)((ud >> 52) & 0x7ff);
  // zeros, subnormals, inf, NaN and quotients near the ends of the range
  if ((unsigned)(en - 600) >= 800u || (unsigned)(ed - 600) >= 800u) return n / d;
  const uint64_t frac = 0xfffffffffffffull, one = 0x10000000000000ull;
  uint64_t mn = (un & frac) | one;
  const uint64_t md = (ud & frac) | one;
  // hi: the leading 24 bits in [1, 2), lo: the other 29
  const float dh = div_float(0x3f800000u | ((uint32_t)(md >> 29) & 0x7fffffu));
  const float dl = (float)(int32_t)((uint32_t)md & 0x1fffffffu) * 0x1p-52f;
  float nh = div_float(0x3f800000u | ((uint32_t)(mn >> 29) & 0x7fffffu));
  float nl = (float)(int32_t)((uint32_t)mn & 0x1fffffffu) * 0x1p-52f;
  const int lt = mn < md;               // quotient of the mantissas into [1, 2)
  if (lt) { mn <<= 1; nh += nh; nl += nl; }
  float y = div_rcp(dh, host_error);
  y = fmaf(y, fmaf(-dl, y, fmaf(-dh, y, 1.0f)), y);   // of d, to about 2^-23
  const float q1 = nh * y;
  const float r1 = fmaf(-q1, dh, nh) + fmaf(-q1, dl, nl);
  const float q2 = r1 * y;
  // the estimate in units of 2^-52: q1 exactly, q2 to four units
  uint64_t q = ((uint64_t)(uint32_t)(q1 * 0x1p24f) << 28) + (uint64_t)((int64_t)(int32_t)(q2 * 0x1p50f) * 4);
  int64_t r = (int64_t)((mn << 52) - q * md);   // exact: |r| < 2^62
  const int32_t k = (int32_t)floorf((float)(int32_t)(r >> 32) * (y * 0x1p-20f));
  q += (uint64_t)(int64_t)k;
  r -= (int64_t)k * (int64_t)md;
  if (r < 0) { r += (int64_t)md; --q; }
  else if (r >= (int64_t)md) { r -= (int64_t)md; ++q; }
  const uint64_t r2 = 2 * (uint64_t)r;
  q += r2 > md || (r2 == md && (q & 1));
  // q in [2^52, 2^53]: its leading bit (or carry) adds to the exponent field
  const uint64_t u = ((uint64_t)(en - ed - lt + 1022) << 52) + q;
  return div_double(u | ((un ^ ud) & 0x8000000000000000ull));
}

}  // namespace adcgpu
