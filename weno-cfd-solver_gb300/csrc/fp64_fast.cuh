// Second-order FP64 reciprocal of the FAST kernels' FP64 WENO weights (the stencils that
// the float pairs of ffw.cuh do not cover).  Everything else divides and takes roots
// with the integer forms of rn64.cuh, which need no FP64 slot.
//
// Newton's step on a hardware seed, two FP64 operations:
//  * x = m 2^E is split on its integer bits, m in [1, 2);
//  * a seed y0 of 1/m comes from the PTX instruction rcp.approx.ftz.f32 applied to the
//    leading 23 bits of m (relative error of y0 below 2^-21), widened to double on its bits;
//  * 1/m = y0 / (1 - e) = y0 (1 + e + ...), e = 1 - m y0 by one fused multiply-add,
//    truncated after e: relative error below 2^-41 (the seed's error squared), which in
//    the normalisation of the weights only scales the weighted slope added to a centre value;
//  * 2^-E is put back on the exponent bits of the result.
// Arguments whose exponent lies outside [-1000, 1000] (zero, subnormals, infinities,
// NaN) take the correctly rounded quotient.
#pragma once

#include <cuda_runtime.h>

#include "rn64.cuh"

namespace weno {
namespace f64fast {

constexpr int kExpLo = 1023 - 1000, kExpHi = 1023 + 1000;  // biased exponents of the fast range

__device__ __forceinline__ float rcp_approx(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// A positive normal float as a double, on the bits (exact).
__device__ __forceinline__ double widen(float f) {
  const unsigned b = __float_as_uint(f);
  const unsigned hi = (((b >> 23) + (1023u - 127u)) << 20) | ((b & 0x7fffffu) >> 3);
  return __hiloint2double((int)hi, (int)((b & 7u) << 29));
}

// The leading 23 mantissa bits of the double (hi, lo) under the float biased
// exponent fexp.
__device__ __forceinline__ float narrow(int hi, int lo, unsigned fexp) {
  return __uint_as_float((fexp << 23) | (((unsigned)hi & 0xfffffu) << 3) | ((unsigned)lo >> 29));
}

__device__ __forceinline__ int biased_exp(int hi) { return (hi >> 20) & 0x7ff; }

__device__ __forceinline__ double rcp2(double x) {
  const int hi = __double2hiint(x), lo = __double2loint(x);
  const int ex = biased_exp(hi);
  if (ex < kExpLo || ex > kExpHi)
    return __longlong_as_double((long long)rn64::div(0x3ff0000000000000ull, (uint64_t)__double_as_longlong(x),
                                                     [](float v) { return rcp_approx(v); }));
  const double m = __hiloint2double((hi & 0x000fffff) | 0x3ff00000, lo);
  const double y0 = widen(rcp_approx(narrow(hi, lo, 127u)));
  const double y = fma(y0, fma(-m, y0, 1.0), y0);  // in [0.5, 1]
  const int yh = __double2hiint(y) - (ex - 1023) * (1 << 20);
  return __hiloint2double(yh | (hi & (int)0x80000000), __double2loint(y));
}

}  // namespace f64fast
}  // namespace weno
