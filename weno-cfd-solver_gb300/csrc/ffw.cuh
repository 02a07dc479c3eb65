// WENO5 weights of the FAST FP64 kernels on the FP32 pipe.
//
// One FP64 warp instruction takes 16 cycles of an SM, in which the FP32 and
// integer pipes can issue 64; forming the non-linear weights took most of the 69
// FP64 operations per field and face (and of the 40 per Gauss pair).  The weights
// multiply first differences of the field, so they need not be formed in FP64:
// here the indicators, their inverse squares and the weights are float pairs
// (hi + lo), and come back as doubles; 19 FP64 operations
// per field and face remain (14 per Gauss pair).
//
// Around a cell with first differences d0, d1 on its left and d2, d3 on its right
//   0.75 beta of (d2, d3) = (13 (d3 - d2)^2 + 3 (d3 - 3 d2)^2) / 16
//   0.75 beta of (d1, d2) = (13 (d2 - d1)^2 + 3 (d1 + d2)^2) / 16
//   0.75 beta of (d0, d1) = (13 (d1 - d0)^2 + 3 (d0 - 3 d1)^2) / 16
// (the Jiang-Shu indicators, weno.rs:223-230, in first differences; sums of
// squares, so nothing cancels).
//
// Accuracy, against extended precision: the weights are within 2^-44 of their sum (the
// largest error seen over the covered range is 2^-45.0).
// Face values come out no further off than with weights formed in FP64 and
// normalised by the reciprocal of relative error 2^-41 that served before (root
// mean square over 3 million stencils: smooth data 5.4e-17 against 7.2e-17, a jump
// of 1.3 with noise 7.0e-17 against 8.8e-17, random data in [0.05, 3] 1.54e-15
// against 1.60e-15).
//
// Mirror-image stencils (d_m -> -d_{3-m}) give mirror-image face states, as the
// reference's do: the state at the other face is formed by the same operations on the
// mirrored values.  The two values of a Gauss pair are not each other's mirror to the
// last bit (nor are the reference's: its sums run in the order of the stencils).
//
// Range: differences below 2^22 (smaller than 2^-70 count as zero) and an epsilon in
// [2^-48, 2^40); callers take the FP64 weights otherwise.  The lower end keeps the low
// part of the reciprocal of the weights' sum, eps^2 / 2^24, a normal float: at 2^-58 it
// has three bits left and the weights of a smooth stencil are off by 2^-27 of their sum
// (2^-43 at 2^-50, 2^-45 from 2^-48 on).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace weno {
namespace ffw {

struct ff {
  float h, l;
};

__device__ __forceinline__ ff quick_two_sum(float a, float b) {  // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return ff{s, __fadd_rn(b, -__fadd_rn(s, -a))};
}
__device__ __forceinline__ ff add(ff a, ff b) {
  const float s = __fadd_rn(a.h, b.h);
  const float bb = __fadd_rn(s, -a.h);
  const float e = __fadd_rn(__fadd_rn(a.h, -__fadd_rn(s, -bb)), __fadd_rn(b.h, -bb));
  return quick_two_sum(s, __fadd_rn(e, __fadd_rn(a.l, b.l)));
}
__device__ __forceinline__ ff neg(ff a) { return ff{-a.h, -a.l}; }
__device__ __forceinline__ ff mul(ff a, ff b) {
  const float p = __fmul_rn(a.h, b.h);
  const float e = __fmaf_rn(a.l, b.h, __fmaf_rn(a.h, b.l, __fmaf_rn(a.h, b.h, -p)));
  return quick_two_sum(p, e);
}
__device__ __forceinline__ ff sq(ff a) {
  const float p = __fmul_rn(a.h, a.h);
  const float e = __fmaf_rn(__fadd_rn(a.h, a.h), a.l, __fmaf_rn(a.h, a.h, -p));
  return quick_two_sum(p, e);
}
// c a for a float c
__device__ __forceinline__ ff scale(float c, ff a) {
  const float p = __fmul_rn(c, a.h);
  return quick_two_sum(p, __fmaf_rn(c, a.l, __fmaf_rn(c, a.h, -p)));
}
__device__ __forceinline__ ff pow2(float c, ff a) { return ff{__fmul_rn(c, a.h), __fmul_rn(c, a.l)}; }  // c a power of two
__device__ __forceinline__ ff rcp(ff a) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a.h));
  const float r = __fmaf_rn(-a.l, y, __fmaf_rn(-a.h, y, 1.0f));
  return quick_two_sum(y, __fmul_rn(y, __fmaf_rn(r, r, r)));
}
__host__ __device__ constexpr ff constant(double c) { return ff{(float)c, (float)(c - (double)(float)c)}; }

// A double as a float pair, on its bits; below 2^-70 it is zero.
__device__ __forceinline__ ff from_double(double d) {
  const uint32_t hi = (uint32_t)__double2hiint(d), lo = (uint32_t)__double2loint(d);
  // head: the fraction rounded to 23 bits (a carry runs into the exponent), and
  // the exponent rebiased by its bit 7
  const uint64_t r = (((uint64_t)hi << 32) | lo) + 0x10000000u;
  const uint32_t h = (((uint32_t)(r >> 29) & 0x7fffffffu) ^ 0x40000000u) | (hi & 0x80000000u);
  // rest: the low 29 bits as a signed number of units of 2^(exponent - 52)
  const float rest = (float)((int32_t)(lo << 3) >> 3);
  const uint32_t unit = (((hi << 3) & 0x7f800000u) ^ 0x40000000u) - (52u << 23);
  const float l = __fmul_rn(rest, __uint_as_float(unit | (hi & 0x80000000u)));
  const bool tiny = (hi & 0x7fffffffu) < ((1023u - 70u) << 20);
  return ff{tiny ? 0.0f : __uint_as_float(h), tiny ? 0.0f : l};
}

// A non-negative float pair as a double, exact (anything below 2^-75 is only
// that small): the low part is made positive, so that adding it to the head's
// significand as an integer stays within the head's binade.
__device__ __forceinline__ double to_double(ff a) {
  const bool below = a.l < 0.0f;
  const uint32_t hb = __float_as_uint(a.h) - (below ? 1u : 0u);
  const float l = below ? __fadd_rn(a.l, __fadd_rn(a.h, -__uint_as_float(hb))) : a.l;
  const uint32_t li = __float2uint_rz(__fmul_rn(l, __uint_as_float((306u << 23) - (hb & 0x7f800000u))));
  const uint64_t bits = (((uint64_t)hb) << 29) + ((uint64_t)896 << 52) + li;
  return __longlong_as_double((long long)bits);
}

// Whether the float pairs cover differences whose largest high word (sign
// cleared) is dmax with the epsilon eps.
__device__ __forceinline__ uint32_t magnitude(double d) { return (uint32_t)__double2hiint(d) & 0x7fffffffu; }
__device__ __forceinline__ bool covers(uint32_t dmax, double eps) {
  return dmax < ((1023u + 22u) << 20) &&
         (uint32_t)__double2hiint(eps) - ((1023u - 48u) << 20) < ((48u + 40u) << 20);
}

// The same for float pairs.
__device__ __forceinline__ bool covers_pair(float dmax, float eps) {
  return dmax < 0x1p22f && eps >= 0x1p-48f && eps < 0x1p40f;
}

// 0.75 eps.
__device__ __forceinline__ ff eps75(double eps) { return scale(0.75f, from_double(eps)); }

// 1/(0.75 (eps + beta))^2 of the one-sided stencil with near difference y and
// far difference x, and of the central one.
__device__ __forceinline__ ff inv_sq(ff e) { return sq(rcp(e)); }
__device__ __forceinline__ ff curvature(ff a, ff b) { return scale(0.8125f, sq(add(b, neg(a)))); }  // 13/16 (b - a)^2
__device__ __forceinline__ ff side(ff y, ff x, ff w) {
  return inv_sq(add(add(scale(0.1875f, sq(add(x, scale(-3.0f, y)))), curvature(y, x)), w));
}
__device__ __forceinline__ ff centre(ff a, ff b, ff w) {
  return inv_sq(add(add(scale(0.1875f, sq(add(a, b))), curvature(a, b)), w));
}

// k w_j of three weights a_j (heads comparable, a sum over them r^-1), with the
// largest formed as k less the other two: the weights then sum to k to 2^-50 and
// an error of the two smaller ones only multiplies the difference of their
// candidates to the largest one's.
__device__ __forceinline__ void take(ff a, double& c) { c = to_double(a); }
__device__ __forceinline__ void take(ff a, ff& c) { c = a; }
template <class C>  // double, or ff for the df64 kernels
__device__ __forceinline__ void normalised(ff a0, ff a1, ff a2, ff r, ff k, C& c0, C& c1, C& c2) {
  const bool m0 = a0.h > a1.h && a0.h > a2.h, m2 = !m0 && a2.h > a1.h;  // largest: 0, 2 or else 1
  const ff x = mul(ff{m0 ? a1.h : a0.h, m0 ? a1.l : a0.l}, r);  // a1 where 0 is the largest, else a0
  const ff y = mul(ff{m2 ? a1.h : a2.h, m2 ? a1.l : a2.l}, r);  // a1 where 2 is the largest, else a2
  C cx, cy, cm;
  take(x, cx);
  take(y, cy);
  take(add(add(k, neg(x)), neg(y)), cm);
  c0 = m0 ? cm : cx;
  c1 = m0 ? cx : (m2 ? cy : cm);
  c2 = m2 ? cm : cy;
}

// 2 c for a positive normal c.
__device__ __forceinline__ double twice(double c) {
  return __hiloint2double(__double2hiint(c) + (1 << 20), __double2loint(c));
}

// w/6 of a face state from the inverse squares of the stencil reaching over the
// face (linear weight .3), the central one (.6) and the one on the other side (.1).
template <class C>
__device__ __forceinline__ void face_weights(ff q_near, ff q_mid, ff q_far, C& c_near, C& c_mid, C& c_far) {
  constexpr ff sixth = constant(1.0 / 6.0);
  const ff a0 = scale(3.0f, q_near), a1 = pow2(2.0f, scale(3.0f, q_mid));
  const ff r = mul(sixth, rcp(add(add(a0, a1), q_far)));
  normalised(a0, a1, q_far, r, sixth, c_near, c_mid, c_far);
}

// S w of one Gauss point from the inverse squares of the stencils on its side, in the
// middle and on the other side; r0, r2 are the outer linear weights over the central one.
template <class C>
__device__ __forceinline__ void gauss_weights(ff q0, ff q1, ff q2, ff r0, ff r2, ff S, C& c0, C& c1, C& c2) {
  const ff a0 = mul(r0, q0), a2 = mul(r2, q2);
  const ff r = mul(S, rcp(add(add(a0, a2), q1)));
  normalised(a0, q1, a2, r, S, c0, c1, c2);
}

}  // namespace ffw
}  // namespace weno
