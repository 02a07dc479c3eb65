// FP64 sums and products spelled as fused multiply-adds.
//
// GB300's FP64 pipe takes a DFMA every 16 cycles per SM and warp, but a DADD, a
// DMUL, a DSETP or a DMNMX only every 19 (measured with 16 resident warps and
// register operands).  a + b = fma(a, 1, b) and a b = fma(a, b, -0) are the same
// IEEE results bit for bit, signs of zeros, infinities and NaN included.  The 1
// and the -0 come from constant memory, where no compiler can fold them back
// into an add or a multiply.
#pragma once

#include <cuda_runtime.h>

namespace weno {

static __constant__ double kOpaqueOne = 1.0;
static __constant__ double kOpaqueNegZero = -0.0;

__device__ __forceinline__ double xadd(double a, double b) { return __fma_rn(a, kOpaqueOne, b); }
__device__ __forceinline__ double xmul(double a, double b) { return __fma_rn(a, b, kOpaqueNegZero); }

}  // namespace weno
