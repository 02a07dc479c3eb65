// f64: a double whose operations are spelled for GB300's FP64 pipe.
//
// * Sums and products are fused multiply-adds (opaque64.cuh): same bits, 16
//   cycles of the pipe instead of 19.
// * Comparisons, minima and maxima are integer operations on the bits.
// * Quotients and square roots are the integer forms of rn64.cuh, correctly
//   rounded: about 80 issue slots against the 640 that ten FP64 instructions take.
//
// In a translation unit with WENO_F64_CONTRACT (the FAST ones) a product is a
// proxy, as in f32x2.cuh, and a * b + c becomes one FMA; without it every
// operation rounds on its own, in the order written.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

#include "opaque64.cuh"
#include "rn64.cuh"

namespace weno {
inline namespace WENO_TU_NS {

__device__ __forceinline__ float rcp_seed(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float rsqrt_seed(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// x 2^K: an integer addition to the exponent for zeros and for normal numbers
// whose result is normal, the multiplication otherwise.
template <int K>
__device__ __forceinline__ double xscale(double x) {
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const uint32_t e = hi & 0x7ff00000u;
  constexpr uint32_t lo_e = K < 0 ? (uint32_t)(1 - K) << 20 : 1u << 20;       // smallest exponent field taken
  constexpr uint32_t hi_e = K > 0 ? (uint32_t)(2046 - K) << 20 : 2046u << 20;  // largest
  if (e - lo_e <= hi_e - lo_e) return __hiloint2double((int)(hi + (uint32_t)(K * (1 << 20))), (int)lo);
  if (((hi << 1) | lo) == 0u) return x;
  return xmul(x, K >= 0 ? (double)(1u << (K >= 0 ? K : 0)) : 1.0 / (double)(1u << (K < 0 ? -K : 0)));
}

__device__ __forceinline__ double xdiv(double a, double b) {
  return __longlong_as_double((long long)rn64::div((uint64_t)__double_as_longlong(a), (uint64_t)__double_as_longlong(b),
                                                   [](float x) { return rcp_seed(x); }));
}
__device__ __forceinline__ double xsqrt(double x) {
  return __longlong_as_double(
      (long long)rn64::sqrt((uint64_t)__double_as_longlong(x), [](float m) { return rsqrt_seed(m); }));
}

// The type and its functions live in their own namespace (as df64's): argument-
// dependent lookup finds them for f64 arguments, while unqualified calls on
// floats and doubles still reach the CUDA math functions.
namespace xf {

struct f64 {
  double v;
  f64() = default;
  __host__ __device__ constexpr f64(double x) : v(x) {}
  __host__ __device__ explicit operator double() const { return v; }
  __host__ __device__ explicit operator float() const { return (float)v; }
};

__device__ __forceinline__ long long f64_bits(f64 x) { return __double_as_longlong(x.v); }
__device__ __forceinline__ f64 operator-(f64 a) { return f64(-a.v); }
__device__ __forceinline__ f64 operator+(f64 a, f64 b) { return f64(xadd(a.v, b.v)); }
__device__ __forceinline__ f64 operator-(f64 a, f64 b) { return f64(xadd(a.v, -b.v)); }
__device__ __forceinline__ f64 operator/(f64 a, f64 b) { return f64(xdiv(a.v, b.v)); }
__device__ __forceinline__ f64 fma(f64 a, f64 b, f64 c) { return f64(__fma_rn(a.v, b.v, c.v)); }

#ifdef WENO_F64_CONTRACT
struct f64_prod {
  double a, b;
  __device__ __forceinline__ operator f64() const { return f64(xmul(a, b)); }
  __device__ __forceinline__ double val() const { return xmul(a, b); }
};
__device__ __forceinline__ f64_prod operator*(f64 a, f64 b) { return f64_prod{a.v, b.v}; }
__device__ __forceinline__ f64_prod operator*(f64_prod p, f64 b) { return f64_prod{p.val(), b.v}; }
__device__ __forceinline__ f64_prod operator*(f64 a, f64_prod p) { return f64_prod{a.v, p.val()}; }
__device__ __forceinline__ f64_prod operator*(f64_prod p, f64_prod q) { return f64_prod{p.val(), q.val()}; }
__device__ __forceinline__ f64 operator+(f64_prod p, f64 c) { return f64(__fma_rn(p.a, p.b, c.v)); }
__device__ __forceinline__ f64 operator+(f64 c, f64_prod p) { return f64(__fma_rn(p.a, p.b, c.v)); }
__device__ __forceinline__ f64 operator+(f64_prod p, f64_prod q) { return f64(__fma_rn(p.a, p.b, q.val())); }
__device__ __forceinline__ f64 operator-(f64_prod p, f64 c) { return f64(__fma_rn(p.a, p.b, -c.v)); }
__device__ __forceinline__ f64 operator-(f64 c, f64_prod p) { return f64(__fma_rn(-p.a, p.b, c.v)); }
__device__ __forceinline__ f64 operator-(f64_prod p, f64_prod q) { return f64(__fma_rn(p.a, p.b, -q.val())); }
__device__ __forceinline__ f64_prod operator-(f64_prod p) { return f64_prod{-p.a, p.b}; }
__device__ __forceinline__ f64 operator/(f64_prod p, f64 b) { return f64(xdiv(p.val(), b.v)); }
#else
__device__ __forceinline__ f64 operator*(f64 a, f64 b) { return f64(xmul(a.v, b.v)); }
#endif

// Comparisons on the bits: key() orders all numbers as signed integers, both
// zeros at 0; a NaN compares false.
__device__ __forceinline__ long long f64_key(f64 x) {
  const long long s = f64_bits(x);
  return s < 0 ? (long long)(0x8000000000000000ull - (unsigned long long)s) : s;
}
__device__ __forceinline__ bool f64_isnan(f64 x) {
  return (f64_bits(x) & 0x7fffffffffffffffll) > 0x7ff0000000000000ll;
}
__device__ __forceinline__ bool operator<(f64 a, f64 b) {
  return f64_key(a) < f64_key(b) && !f64_isnan(a) && !f64_isnan(b);
}
__device__ __forceinline__ bool operator<=(f64 a, f64 b) {
  return f64_key(a) <= f64_key(b) && !f64_isnan(a) && !f64_isnan(b);
}
__device__ __forceinline__ bool operator>(f64 a, f64 b) { return b < a; }
__device__ __forceinline__ bool operator>=(f64 a, f64 b) { return b <= a; }
__device__ __forceinline__ bool operator==(f64 a, f64 b) { return a.v == b.v; }
__device__ __forceinline__ bool operator!=(f64 a, f64 b) {
  return f64_key(a) != f64_key(b) || f64_isnan(a) || f64_isnan(b);
}
// maxNum / minNum: a NaN operand yields the other one; max(+0, -0) = +0.
__device__ __forceinline__ f64 fmax(f64 a, f64 b) {
  const long long x = f64_bits(a), y = f64_bits(b);
  const long long kx = x ^ ((x >> 63) & 0x7fffffffffffffffll), ky = y ^ ((y >> 63) & 0x7fffffffffffffffll);
  return (f64_isnan(b) || (kx > ky && !f64_isnan(a))) ? a : b;
}
__device__ __forceinline__ f64 fmin(f64 a, f64 b) {
  const long long x = f64_bits(a), y = f64_bits(b);
  const long long kx = x ^ ((x >> 63) & 0x7fffffffffffffffll), ky = y ^ ((y >> 63) & 0x7fffffffffffffffll);
  return (f64_isnan(b) || (kx < ky && !f64_isnan(a))) ? a : b;
}
__device__ __forceinline__ f64 fabs(f64 a) { return f64(::fabs(a.v)); }
__device__ __forceinline__ f64 copysign(f64 m, f64 s) { return f64(::copysign(m.v, s.v)); }
__device__ __forceinline__ f64 sqrt(f64 x) { return f64(xsqrt(x.v)); }

}  // namespace xf
using xf::f64;
using xf::f64_bits;

// The device arithmetic type of a host scalar type.
template <class T>
struct dev_type {
  using type = T;
};
template <>
struct dev_type<double> {
  using type = f64;
};
template <class T>
using dev_t = typename dev_type<T>::type;

}  // inline namespace WENO_TU_NS
}  // namespace weno
