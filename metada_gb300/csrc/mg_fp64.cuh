// FP64 arithmetic in few FP64 instructions.  GB300 runs two FP64 lanes per
// clock per SM (a warp instruction takes its scheduler's FP64 unit 64
// cycles), and conversions between FP32 and FP64 run at the same rate, so
// divisions are replaced by a reciprocal and corrections.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace mg {

// 1 / d for d > 0 to FP64 rounding (about one ulp): an FP32 reciprocal of
// d's leading 24 bits, moved between the formats with integer operations,
// and r (1 + e + e^2) with e = 1 - d r, whose error is e^3 < 2^-66.
// Outside FP32's normal range the plain division.
__device__ __forceinline__ double recip_fp64(double d) {
  const int hi = __double2hiint(d);
  const int ex = (hi >> 20) - 1023;
  if (ex < -120 || ex > 120) return 1.0 / d;
  const float f = __int_as_float(((hi - (896 << 20)) << 3) | (int)((unsigned)__double2loint(d) >> 29));
  const int rb = __float_as_int(__frcp_rn(f));
  const double r = __hiloint2double((rb >> 3) + (896 << 20), rb << 29);
  const double e = __fma_rn(-d, r, 1.0);
  return __fma_rn(r, __fma_rn(e, e, e), r);
}

// A usable pivot: positive, and below 3e38 (so finite).  By the leading word:
// a comparison of doubles is an FP64 instruction.
__device__ __forceinline__ bool pivot_ok(double d) {
  const int hi = __double2hiint(d);
  return hi > 0 && hi < __double2hiint(3.0e38);
}

// a / b given r = 1 / b correctly rounded: one correction of a r by its exact
// remainder gives the correctly rounded quotient (Markstein, 1990) while no
// term leaves the normal range.  b and r have to be normal numbers (an infinite
// or zero b gives NaN), and an infinite a gives NaN: a caller whose result may
// then differ from the division's guards both.
__device__ __forceinline__ double div_refined(double a, double b, double r) {
  const double q = __dmul_rn(a, r);
  return __fma_rn(__fma_rn(-q, b, a), r, q);
}

// (double)x by integer operations: a conversion runs on the FP64 pipe and
// holds its scheduler for 64 cycles.  Exact for zeros and normal numbers;
// wide_special(x) tells the others (subnormals, infinities, NaN), which take
// the conversion.
__device__ __forceinline__ bool wide_special(float x) {
  const uint32_t mag = __float_as_uint(x) & 0x7fffffffu;
  return mag - 0x00800000u >= 0x7f000000u && mag != 0u;
}
__device__ __forceinline__ double wide(float x) {
  const uint32_t u = __float_as_uint(x), mag = u & 0x7fffffffu;
  const uint32_t hi = (mag ? (mag >> 3) + 0x38000000u : 0u) | (u & 0x80000000u);
  return __hiloint2double((int)hi, (int)(u << 29));
}
static __device__ __noinline__ double wide_cvt(float x) { return (double)x; }

}  // namespace mg
