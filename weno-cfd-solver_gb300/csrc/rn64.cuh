// Correctly rounded FP64 quotient and square root in integer and FP32 operations.
//
// GB300 issues one FP64 warp instruction per 16 cycles and SM (64 issue slots),
// and a correctly rounded FP64 divide is about ten of them; the integer and
// FP32 pipes are nearly idle beside it.  Here the significands are divided as
// integers, schoolbook fashion in three digits of 22, 20 and 12 bits, each
// estimated in FP32 from one hardware reciprocal (square root: reciprocal
// square root) seed and corrected through the exact integer remainder, which
// always fits 64 bits (the products wrap around harmlessly).  About 80 issue
// slots and no FP64 operation.
//
// Correctness needs of the seed y only |y fb - 1| < 2^-21 (fb the leading 24
// bits of b, truncated): the first digit is then within 5 units, the second
// within 2.5, the third within 0.51, and the sign of the last remainder says
// on which side of it the exact result lies.  A quotient or a square root of
// 53-bit significands is never half way between two, so rounding the floor
// with two guard bits is round-to-nearest-even.
//
// Zeros, subnormals, infinities, NaN and results outside the normal range take
// the same digits with integer code before and after them: bit for bit the IEEE
// results as well, without the call and the second division routine that the
// compiler's own quotient would put into every loop that divides.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define WENO_HD __host__ __device__ __forceinline__
#else
#include <cmath>
#define WENO_HD inline
#endif

namespace weno {
namespace rn64 {

#ifdef __CUDA_ARCH__
WENO_HD int to_int(float x) { return __float2int_rn(x); }
WENO_HD float as_float(uint32_t b) { return __uint_as_float(b); }
WENO_HD int leading_zeros(uint64_t x) { return __clzll((long long)x); }
#else
WENO_HD int to_int(float x) { return (int)lrintf(x); }
WENO_HD float as_float(uint32_t b) {
  float f;
  __builtin_memcpy(&f, &b, 4);
  return f;
}
WENO_HD int leading_zeros(uint64_t x) { return __builtin_clzll(x); }
#endif

constexpr uint64_t kSign = 0x8000000000000000ull, kInf = 0x7ff0000000000000ull, kNaN = 0x7ff8000000000000ull;

WENO_HD uint32_t biased_exp(uint64_t x) { return (uint32_t)(x >> 52) & 0x7ffu; }
// Significand of a normal number, in [2^52, 2^53).
WENO_HD uint64_t significand(uint64_t x) { return (x & 0xfffffffffffffull) | 0x10000000000000ull; }
// The leading 24 bits of a significand, truncated, as a float of biased exponent fexp.
WENO_HD float leading(uint64_t m, uint32_t fexp) {
  return as_float((fexp << 23) | ((uint32_t)(m >> 29) & 0x7fffffu));
}

// Normal operands whose quotient is a normal number away from the ends.
WENO_HD bool div_in_range(uint64_t a, uint64_t b) {
  const uint32_t ea = biased_exp(a), eb = biased_exp(b);
  return ea - 1u < 2046u && eb - 1u < 2046u && ea - eb + 1000u <= 2000u;
}

// floor(2^54 ma / mb) of two significands, in (2^53, 2^55); y approximates
// 1 / leading(mb, 127); `inexact`: a remainder is left.
WENO_HD uint64_t div_digits(uint64_t ma, uint64_t mb, float y, bool& inexact) {
  // digits in units of 2^-22, 2^-42, 2^-54
  const int q1 = to_int(leading(ma, 127u + 22u) * y);
  const uint64_t r1 = (ma << 22) - (uint64_t)(uint32_t)q1 * mb;
  const int q2 = to_int((float)(int)((int64_t)r1 >> 26) * (y * 0x1p-6f));
  const uint64_t r2 = (r1 << 20) - (uint64_t)(int64_t)q2 * mb;
  const int q3 = to_int((float)(int)((int64_t)r2 >> 26) * (y * 0x1p-14f));
  const uint64_t r3 = (r2 << 12) - (uint64_t)(int64_t)q3 * mb;
  inexact = r3 != 0;
  return ((uint64_t)(uint32_t)q1 << 32) + (uint64_t)((int64_t)q2 * 4096 + q3) - (r3 >> 63);
}

// Bits of RN(a / b); rcp(x) approximates 1 / x for x in [1, 2).
template <class Rcp>
WENO_HD uint64_t div(uint64_t a, uint64_t b, Rcp rcp) {
  const bool normal = div_in_range(a, b);
  const uint64_t sign = (a ^ b) & kSign;
  uint64_t ma = significand(a), mb = significand(b);
  int ed = (int)biased_exp(a) - (int)biased_exp(b);
  if (!normal) {
    const uint64_t ua = a & ~kSign, ub = b & ~kSign;
    if (ua > kInf || ub > kInf) return kNaN;
    if (ua == 0 || ub == kInf) return (ub == 0 || ua == kInf) ? kNaN : sign;
    if (ub == 0 || ua == kInf) return sign | kInf;
    if (biased_exp(a) == 0) {
      const int sh = leading_zeros(ua) - 11;
      ma = ua << sh;
      ed += 1 - sh;
    }
    if (biased_exp(b) == 0) {
      const int sh = leading_zeros(ub) - 11;
      mb = ub << sh;
      ed -= 1 - sh;
    }
  }
  bool inexact;
  const uint64_t Q = div_digits(ma, mb, rcp(leading(mb, 127u)), inexact);
  const uint32_t s = (uint32_t)(Q >> 54);  // quotient of the significands >= 1
  const int e = ed + 1022 + (int)s;        // biased exponent
  if (!normal && (e < 1 || e > 2046)) {
    if (e > 2046) return sign | kInf;
    const int sh = (int)s + 2 - e;  // bits below the last place of a subnormal result
    if (sh > 60) return sign;
    const uint64_t R = Q >> sh, rem = Q & ((1ull << sh) - 1), half = 1ull << (sh - 1);
    return sign | (R + (rem > half || (rem == half && (inexact || (R & 1))) ? 1 : 0));
  }
  const uint64_t R = (Q + (1u + s)) >> (1u + s);  // no ties: see above
  return sign | (((uint64_t)(uint32_t)(e - 1) << 52) + R);
}

// Bits of RN(sqrt(x)); rsq(m) approximates 1 / sqrt(m) for m in [1, 4).
template <class Rsqrt>
WENO_HD uint64_t sqrt(uint64_t x, Rsqrt rsq) {
  uint64_t sig = significand(x);
  int ex = (int)biased_exp(x);
  if (ex - 1 >= 2046 || ex == 0 || (x & kSign)) {
    if ((x & ~kSign) == 0 || x == kInf) return x;
    if ((x & kSign) || x > kInf) return kNaN;
    const int sh = leading_zeros(x) - 11;
    sig = x << sh;
    ex = 1 - sh;
  }
  const int odd = (ex + 1) & 1;
  const uint64_t m = sig << odd;  // in [1, 4), units of 2^-52
  const float y = rsq(leading(sig, 127u + (uint32_t)odd));
  // s in [1, 2): digits in units of 2^-22, 2^-42, 2^-54
  const int s1 = to_int(leading(sig, 127u + (uint32_t)odd) * (y * 0x1p22f));
  const int64_t r1 = (int64_t)(m - (((uint64_t)(uint32_t)s1 * (uint32_t)s1) << 8));
  const int s2 = to_int((float)(int)(r1 >> 4) * (y * 0x1p-7f));
  const uint64_t S2 = ((uint64_t)(uint32_t)s1 << 20) + (uint64_t)(int64_t)s2;
  const int64_t r2 = (int64_t)((m << 32) - S2 * S2);
  const int s3 = to_int((float)(int)(r2 >> 16) * (y * 0x1p-15f));
  const uint64_t S3 = (S2 << 12) + (uint64_t)(int64_t)s3;
  const uint64_t r3 = (m << 56) - S3 * S3;
  const uint64_t R = (S3 - (r3 >> 63) + 2u) >> 2;
  const int e = (ex - odd + 1023) >> 1;  // biased exponent of the root
  return ((uint64_t)(uint32_t)(e - 1) << 52) + R;
}

}  // namespace rn64
}  // namespace weno
