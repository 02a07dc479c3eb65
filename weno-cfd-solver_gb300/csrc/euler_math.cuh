// Device arithmetic of the 2D Euler finite-volume residual.
//
// Every function follows the reference's Rust core (weno_ext/src/utils.rs,
// weno.rs, riemann.rs) and is templated on
//   T    -- f64 (a double whose operations are spelled for the FP64 pipe,
//           f64.cuh), float or df64, the arithmetic type;
//   FAST -- false: the reference's operation order, so that a translation unit
//           compiled with --fmad=false reproduces the Rust IEEE-754 doubles bit
//           for bit; true: the same mathematics with fewer FP64 operations and
//           FMA contraction, checked against the oracle by tolerance.
//
// GB300 executes FP64 at 1/64 of the FP32 rate and every FP64 kernel here is bound
// by that pipe, so both arithmetics are written to need few of its slots rather
// than little memory traffic: additions and products issue as FMAs (16 cycles a
// warp and SM where DADD and DMUL take 19), comparisons, divisions and square
// roots run on the integer pipe (rn64.cuh), and the FAST WENO weights run on the
// FP32 pipe as float pairs (ffw.cuh).
#pragma once

#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>

#ifndef WENO_TU_NS
#error "WENO_TU_NS names the translation unit's inline namespace (tu_exact or tu_fast)"
#endif

#include "df64.cuh"
#include "f32x2.cuh"
#include "f64.cuh"
#include "ffw.cuh"
#include "fp64_fast.cuh"

namespace weno {
// Each translation unit compiles its kernels into its own inline namespace, so
// the --fmad=false and --fmad=true builds of the same template never share a
// symbol (the linker would otherwise keep only one of them).
inline namespace WENO_TU_NS {

// utils.rs:3-6
constexpr double kEps = 1e-12;              // DEFAULT_EPS, RHO_MIN and P_MIN; also the default WENO epsilon
                                            // `weps` (weno.rs:223), which callers may change
constexpr double kSqrt3_12 = 0.1443375673;  // truncated literal, not sqrt(3)/12
// weno.rs:270 / weno.rs:292 (Gauss-point linear weights, 10 digits)
constexpr double kGqA0 = 0.1928406937, kGqA1 = 0.6111111111, kGqA2 = 0.1960481952;
constexpr double kC13 = 13.0 / 12.0;
// The non-linear weights d_k/(eps+b_k)^2 / sum are unchanged when every
// eps+b_k is multiplied by the same factor; the FAST forms use 4 (eps+b_k) =
// 4 eps + (13/3) D^2 + s^2, two fused multiply-adds per indicator.
constexpr double kC43 = 13.0 / 3.0;

// Arithmetic kinds: native double takes the common-denominator WENO form (its
// exponent range is ample); float and df64 (float exponent range) take the
// reciprocal form.
template <class T>
constexpr bool is_native_f64 = std::is_same<T, f64>::value;
template <class T>
constexpr bool is_f32 = std::is_same<T, float>::value;

template <class T>
__device__ __forceinline__ T vmax(T a, T b) { return fmax(a, b); }
template <class T>
__device__ __forceinline__ T vmin(T a, T b) { return fmin(a, b); }
// a*b + c as one FMA where the type has one (the FAST forms that must round
// the same way in two kernels spell it out).
template <class T>
__device__ __forceinline__ T mul_add(T a, T b, T c) {
  if constexpr (is_native_f64<T> || is_f32<T>) return fma(a, b, c);
  else return a * b + c;
}

// max(x, c) against a non-negative bound.  FAST native double reads the operands'
// bits as signed 64-bit integers: for non-negative doubles that order is the numeric
// order, and every value with the sign bit set (negatives, -0) reads below any
// non-negative bound, so the result is max(x, c) for every non-NaN x, in one integer
// compare (an f64's general compare orders the bits of both signs and looks for
// NaN).  A NaN x with the sign bit clear passes through where fmax would return the
// bound; NaN propagates through the neighbouring arithmetic either way.
template <class T, bool FAST>
__device__ __forceinline__ T cmax(T x, T c) {
  if constexpr (FAST && is_native_f64<T>) return f64_bits(x) > f64_bits(c) ? x : c;
  else return vmax(x, c);
}
// x 2^K of the exact forms: an integer operation on an f64's exponent.
template <int K, class T>
__device__ __forceinline__ T mul_pow2(T x) {
  if constexpr (is_native_f64<T>) return T(xscale<K>(x.v));
  else return x * T(K >= 0 ? (double)(1 << (K >= 0 ? K : 0)) : 1.0 / (double)(1 << (K < 0 ? -K : 0)));
}

template <class T>
__device__ __forceinline__ T half(T x) { return mul_pow2<-1>(x); }

// v[k] and v[k] = x for a run-time k without leaving registers.  The FP64 and df64
// kernels loop over the four fields: unrolled, their integer divisions (exact) or
// float-pair weights (FAST) would not fit the instruction cache, and FP64 or issue
// slots are their bound, not the latency of one warp.
template <class T>
constexpr int kFieldUnroll = is_f32<T> ? 4 : 1;
template <class T>
__device__ __forceinline__ T pick4(const T v[4], int k) {
  const T a = (k & 1) ? v[1] : v[0], b = (k & 1) ? v[3] : v[2];
  return (k & 2) ? b : a;
}
template <class T>
__device__ __forceinline__ void pick_row(const T M[4][4], int r, T row[4]) {
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    const T col[4] = {M[0][c], M[1][c], M[2][c], M[3][c]};
    row[c] = pick4(col, r);
  }
}
template <class T>
__device__ __forceinline__ void put4(T v[4], int k, T x) {
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = k == i ? x : v[i];
}

// a / b: the IEEE quotient except in FAST float (the SFU path).  For an f64 the
// correctly rounded integer forms of rn64.cuh: no FP64 slot, where the seeded
// Newton forms of fp64_fast.cuh take three to six (64 issue slots each).
template <class T, bool FAST>
__device__ __forceinline__ T qdiv(T a, T b) {
  if constexpr (FAST && is_f32<T>) return __fdividef(a, b);
  else return a / b;
}
// 1 / b.  FAST float: the hardware reciprocal itself, for arguments that are never
// subnormal (clamped densities, guarded denominators, spacings): __fdividef(1, b)
// gives the same bits there but carries four instructions for subnormal b.
template <class T, bool FAST>
__device__ __forceinline__ T qrcp(T b) {
  if constexpr (FAST && is_f32<T>) return rcp_seed(b);
  else return T(1.0) / b;
}
// 1 / e^2 of the float weights.  For a vanishing e, 2^-123 keeps six times the sum of
// three of them, a denominator, below 2^126, from which on the fast division gives
// zero (the slope was lost, and the scheme first order, where e was below 1e-19); the
// weights become the linear ones there.  It is below half a unit of the square of any
// e above 1e-15.
constexpr float kSquareFloor = 0x1p-123f;
__device__ __forceinline__ float inv_square(float e) { return rcp_seed(__fmaf_rn(e, e, kSquareFloor)); }
__device__ __forceinline__ f32x2 inv_square(f32x2 e) {
  const float2 s = __ffma2_rn(e.v, e.v, make_float2(kSquareFloor, kSquareFloor));
  return f32x2(rcp_seed(s.x), rcp_seed(s.y));
}
__device__ __forceinline__ df64 inv_square(df64 e) { return df64(1.0) / (e * e); }
// sqrt(x), 1/sqrt(x) and 1/x of the FAST forms (x > 0).  An f64 takes the integer
// root and reciprocal and one product; float (CUDA's rsqrtf, within 2 ulp) and
// df64 one reciprocal square root r, x r and r r.
template <class T>
__device__ __forceinline__ void roots(T x, T& root, T& inv_root, T& inv) {
  if constexpr (is_native_f64<T>) {
    root = sqrt(x);
    inv = T(1.0) / x;
    inv_root = root * inv;
  } else {
    if constexpr (is_f32<T>) inv_root = rsqrtf(x);
    else inv_root = T(1.0) / sqrt(x);
    root = x * inv_root;
    inv = inv_root * inv_root;
  }
}

// a*b + c*d with both products rounded on their own (never contracted into an
// FMA).  For mirror-image arguments (c*d = -(a*b) exactly) the sum is +0.0, as
// the reference's separately rounded products give; a fused form would leave
// the first product's rounding error, a tiny value of either sign.  Used where
// a sign decides a branch: the Roe-averaged normal velocity and the HLLC star
// speed at a reflecting wall, where the reference flux jumps from F_L to F_R as
// that sign changes (when the Roe sound speed is zero, e.g. a state whose
// energy has gone negative).
template <class T>
__device__ __forceinline__ T sum_prod_rn(T a, T b, T c, T d) {
  if constexpr (is_native_f64<T>) return T(xadd(xmul(a.v, b.v), xmul(c.v, d.v)));
  else if constexpr (is_f32<T>) return __fadd_rn(__fmul_rn(a, b), __fmul_rn(c, d));
  else return a * b + c * d;
}

// ---------------------------------------------------------------------------
// Conserved state helpers (utils.rs:9-35, utils.rs:74-109)
// ---------------------------------------------------------------------------
// The kinetic energy term 0.5 rho (u^2 + v^2) of a pressure, with u = m/rho and
// v = n/rho for the (clamped) density rho: the reference's form, or in FAST the
// same quantity as 0.5 (m u + n v) (rho u = m), two operations fewer.
template <class T, bool FAST>
__device__ __forceinline__ T half_rho_speed2(T rho, T m, T n, T u, T v) {
  if constexpr (FAST) return T(0.5) * (m * u + n * v);
  else return mul_pow2<-1>(rho) * (u * u + v * v);
}

// Euler flux normal to x (Y = false) or y (Y = true), utils.rs:74-109.
template <class T, bool FAST, bool Y>
__device__ __forceinline__ void euler_flux(const T q[4], T gamma, T f[4]) {
  const T rho = cmax<T, FAST>(q[0], T(kEps));
  T u, v;
  if constexpr (FAST) {
    const T r = qrcp<T, FAST>(rho);
    u = q[1] * r;
    v = q[2] * r;
  } else {
    u = q[1] / rho;
    v = q[2] / rho;
  }
  const T p = (gamma - T(1.0)) * (q[3] - half_rho_speed2<T, FAST>(rho, q[1], q[2], u, v));
  if constexpr (!Y) {
    f[0] = q[1];
    f[1] = q[1] * u + p;
    f[2] = q[2] * u;
    f[3] = u * (q[3] + p);
  } else {
    f[0] = q[2];
    f[1] = q[1] * v;
    f[2] = q[2] * v + p;
    f[3] = v * (q[3] + p);
  }
}

// Two Euler fluxes (utils.rs:74-109).
template <class T, bool FAST, bool Y>
__device__ __forceinline__ void euler_flux_pair(const T qa[4], const T qb[4], T gamma, T fa[4], T fb[4]) {
  euler_flux<T, FAST, Y>(qa, gamma, fa);
  euler_flux<T, FAST, Y>(qb, gamma, fb);
}

// The sum of the two fluxes of a Gauss pair (FAST).  An f64 adds the products as
// FMAs: with m, n the momenta along and across the face normal,
// sum (m, m u + p, n u, u (E + p)).
template <class T, bool Y>
__device__ __forceinline__ void euler_flux_sum(const T qa[4], const T qb[4], T gamma, T f[4]) {
  if constexpr (is_native_f64<T>) {
    constexpr int M = Y ? 2 : 1, N = Y ? 1 : 2;
    const T ia = T(1.0) / cmax<T, true>(qa[0], T(kEps)), ib = T(1.0) / cmax<T, true>(qb[0], T(kEps));
    const T ua = qa[M] * ia, ub = qb[M] * ib, va = qa[N] * ia, vb = qb[N] * ib;
    const T g = gamma - T(1.0);
    const T pa = g * (qa[3] - T(0.5) * (qa[M] * ua + qa[N] * va)), pb = g * (qb[3] - T(0.5) * (qb[M] * ub + qb[N] * vb));
    f[0] = qa[M] + qb[M];
    f[M] = qa[M] * ua + (qb[M] * ub + (pa + pb));
    f[N] = qa[N] * ua + qb[N] * ub;
    f[3] = ua * (qa[3] + pa) + ub * (qb[3] + pb);
  } else {
    T f1[4], f2[4];
    euler_flux_pair<T, true, Y>(qa, qb, gamma, f1, f2);
#pragma unroll
    for (int k = 0; k < 4; ++k) f[k] = f1[k] + f2[k];
  }
}

// utils.rs:9-35 con2primi_local for one cell.
template <class T, bool FAST>
__device__ __forceinline__ void con2prim(T q0, T q1, T q2, T q3, T gamma, T& p, T& a, T& rho, T& u, T& v, T& h) {
  rho = cmax<T, FAST>(q0, T(kEps));
  if constexpr (FAST) {
    const T r = qrcp<T, FAST>(rho);
    u = q1 * r;
    v = q2 * r;
    p = cmax<T, FAST>((gamma - T(1.0)) * (q3 - half_rho_speed2<T, FAST>(rho, q1, q2, u, v)), T(kEps));
    a = sqrt(T(gamma * p * r));
    h = (q3 + p) * r;
  } else {
    u = q1 / rho;
    v = q2 / rho;
    p = vmax<T>((gamma - T(1.0)) * (q3 - T(0.5) * rho * (u * u + v * v)), T(kEps));
    a = sqrt(gamma * p / rho);
    h = (q3 + p) / rho;
  }
}

// Pressure of con2primi (clamped density and pressure) -- the quantity the
// shock sensor averages (riemann.rs:421-430).
template <class T, bool FAST>
__device__ __forceinline__ T clamped_pressure(const T q[4], T gamma) {
  const T rho = cmax<T, FAST>(q[0], T(kEps));
  T u, v;
  if constexpr (FAST) {
    const T r = qrcp<T, FAST>(rho);
    u = q[1] * r;
    v = q[2] * r;
  } else {
    u = q[1] / rho;
    v = q[2] / rho;
  }
  return cmax<T, FAST>((gamma - T(1.0)) * (q[3] - half_rho_speed2<T, FAST>(rho, q[1], q[2], u, v)), T(kEps));
}

// ---------------------------------------------------------------------------
// WENO5-JS (weno.rs:214-257) and the 2-point Gauss-quadrature pair
// (weno.rs:262-303).
// ---------------------------------------------------------------------------
// Jiang-Shu indicators of the stencils (u2,u3,u4), (u1,u2,u3), (u0,u1,u2) in the
// reference's operation order.
template <class T>
__device__ __forceinline__ void js_betas(T u0, T u1, T u2, T u3, T u4, T& b0, T& b1, T& b2) {
  T t, s;
  t = u2 - mul_pow2<1>(u3) + u4;
  s = T(3.0) * u2 - mul_pow2<2>(u3) + u4;
  b0 = T(kC13) * (t * t) + mul_pow2<-2>(T(s * s));
  t = u1 - mul_pow2<1>(u2) + u3;
  s = u1 - u3;
  b1 = T(kC13) * (t * t) + mul_pow2<-2>(T(s * s));
  t = u0 - mul_pow2<1>(u1) + u2;
  s = u0 - mul_pow2<2>(u1) + T(3.0) * u2;
  b2 = T(kC13) * (t * t) + mul_pow2<-2>(T(s * s));
}

// Biased exponent of the largest of three positive doubles, from integer
// operations on the high words (no FP64 slot).
__device__ __forceinline__ int max_biased_exp3(f64 a, f64 b, f64 c) {
  const int ea = (__double2hiint(a.v) >> 20) & 0x7ff;
  const int eb = (__double2hiint(b.v) >> 20) & 0x7ff;
  const int ec = (__double2hiint(c.v) >> 20) & 0x7ff;
  return max(ea, max(eb, ec));
}

// Brings (eps + beta_k) into the range where the products of the
// common-denominator weights neither overflow nor lose the dominant weight.
// For a largest value within [2^-W, 2^W] (every practical stencil) nothing is
// done; otherwise all three are scaled by the same power of two that puts the
// largest into [0.5, 1) (exact).  NaN and infinity pass through.  W = 200 for
// the fourth-power products of the WENO5 weights, 120 for the Gauss-point
// pair, whose shared reciprocal takes an eighth-power product.
template <int W = 200>
__device__ __forceinline__ void weno_range(f64& e0, f64& e1, f64& e2) {
  const int em = max_biased_exp3(e0, e1, e2);
  if (em >= 1023 - W && em <= 1023 + W) return;
  if (em == 0x7ff || em == 0) return;
  int b = 2045 - em;
  if (b < 1) b = 1;
  const f64 sc = f64(__hiloint2double(b << 20, 0));
  e0 = e0 * sc;
  e1 = e1 * sc;
  e2 = e2 * sc;
}

// The same for the reciprocal weights of df64, which has the float exponent range: the
// smallest (eps + beta_k), at least 2^-126, is brought into [1, 2) and the others are
// held at 2^30, where a weight is below 2^-58 of the largest one's and drops out of
// the 48 bits.  Without it 1/(eps + beta)^2 overflowed for an epsilon below 2^-63 in
// a uniform flow (the shear field's is eps rho^2: rho below 2.5e-6) and vanished in
// all three for differences above 2^31, and the face state was NaN.
__device__ __forceinline__ df64 weno_scaled(df64 e, float scale) {
  const float h = e.hi * scale;
  if (h < 1.0f) return df64(1.0f, 0.0f);
  return h > 0x1p30f ? df64(0x1p30f, 0.0f) : df64(h, e.lo * scale);
}
__device__ __forceinline__ void weno_range(df64& e0, df64& e1, df64& e2) {
  const float low = fminf(fmaxf(fminf(fminf(e0.hi, e1.hi), e2.hi), 0x1p-126f), 0x1p126f);
  const float scale = __uint_as_float((254u << 23) - (__float_as_uint(low) & 0x7f800000u));  // 2^-(exponent of low)
  e0 = weno_scaled(e0, scale);
  e1 = weno_scaled(e1, scale);
  e2 = weno_scaled(e2, scale);
}

// Non-linear weighting of three candidate values with linear weights d in FAST
// float and df64 (whose float exponent range rules out products of fourth
// powers): reciprocals.  FAST native double uses weno_nd instead.
template <class T>
__device__ __forceinline__ T weno_combine(T e0, T e1, T e2, T d0, T d1, T d2, T p0, T p1, T p2, T scale) {
  static_assert(!is_native_f64<T>, "FAST double takes the common-denominator form (weno_nd)");
  if constexpr (std::is_same<T, df64>::value) weno_range(e0, e1, e2);
  const T a0 = d0 * inv_square(e0);
  const T a1 = d1 * inv_square(e1);
  const T a2 = d2 * inv_square(e2);
  const T num = a0 * p0 + a1 * p1 + a2 * p2;
  return qdiv<T, true>(num, (a0 + a1 + a2) * scale);
}

// The exact weights, a_k = d_k/(eps+b_k)^2 and w_k = a_k/sum, applied to the
// candidates: w0 p0 + w1 p1 + w2 p2, from the squares (passed in a_k).  The three divisions of each kind share
// one piece of code (a loop): FP64 is the bound, not the latency of one warp,
// and integer divisions unrolled at every use would not fit the instruction cache.
// U = 3 unrolls them, for the kernels that one warp's latency bounds.
template <class T, int U = 1>
__device__ __forceinline__ T weno_combine_exact(T a0, T a1, T a2, T d0, T d1, T d2, T p0, T p1, T p2) {
#pragma unroll(U)
  for (int k = 0; k < 3; ++k) {  // rotates (d, a) so that every k divides the front pair
    const T q = d0 / a0;
    a0 = a1, a1 = a2, a2 = q;
    d0 = d1, d1 = d2;
  }
  const T sum = a0 + a1 + a2;
#pragma unroll(U)
  for (int k = 0; k < 3; ++k) {
    const T w = a0 / sum;
    a0 = a1, a1 = a2, a2 = w;
  }
  return a0 * p0 + a1 * p1 + a2 * p2;
}

// FAST native double: the weights in a common-denominator form,
// d_k prod_{j != k} (eps+b_j)^2, returned as numerator and denominator so that
// a caller can share one divide between two reconstructions; the (eps+b_k)
// are first brought into a safe range (weno_range), so the products neither
// overflow nor lose the dominant weight whatever the magnitude of the values.
__device__ __forceinline__ void weno_nd_products(f64 e0, f64 e1, f64 e2, f64& P0, f64& P1, f64& P2) {
  weno_range(e0, e1, e2);
  const f64 s0 = e0 * e0, s1 = e1 * e1, s2 = e2 * e2;
  P0 = s1 * s2;
  P1 = s0 * s2;
  P2 = s0 * s1;
}
// Numerator and denominator of the weighted slope from the products, linear
// weights (3, 6, 1) (the reference's 0.3, 0.6, 0.1 scaled by 10), each
// operation spelled out: two reconstructions that share the products (the
// same three stencils seen from both sides of a cell) round exactly as two
// separate evaluations would.
__device__ __forceinline__ void weno_nd_combine(f64 P0, f64 P1, f64 P2, f64 g0, f64 g1, f64 g2, f64& num,
                                                f64& den) {
  const f64 c0 = 3.0 * P0, c1 = 6.0 * P1;
  num = fma(P2, g2, fma(c1, g1, c0 * g0));
  den = (c0 + c1) + P2;
}

// x = x0 + a/(k b) and y = y0 + c/(k d) with one divide, 1/(k b d), when b d is
// a normal number well inside the double range (tested on its exponent bits, no
// FP64 slot); otherwise two divides.
__device__ __forceinline__ void div_pair(f64 a, f64 b, f64 c, f64 d, f64& x, f64& y, f64 k, f64 x0, f64 y0) {
  const f64 bd = b * d;
  const int e = (__double2hiint(bd.v) >> 20) & 0x7ff;
  if (e > 64 && e < 1983) {
    const f64 inv = f64(f64fast::rcp2(f64(bd * k).v));  // scales the slopes only
    x = fma(a * d, inv, x0);
    y = fma(c * b, inv, y0);
  } else {
    x = x0 + a / (b * k);
    y = y0 + c / (d * k);
  }
}

// weno.rs:214-257, exact: the left-biased value at the right face of u2 and the
// right-biased one at the left face of u3, the reference's operations.  The
// right stencils are the left ones shifted by a cell, so one loop body serves both.
template <class T, int U = 1>
__device__ __forceinline__ void weno5_lr_exact(const T u[6], T weps, T& left, T& right) {
  // candidate polynomials (x6): two are shared by the two sides
  const T f1 = -u[4] + T(5.0) * u[3] + mul_pow2<1>(u[2]);
  const T f2 = -u[1] + T(5.0) * u[2] + mul_pow2<1>(u[3]);
#pragma unroll(U == 1 ? 1 : 2)
  for (int side = 0; side < 2; ++side) {
    const T v0 = side ? u[1] : u[0], v1 = side ? u[2] : u[1], v2 = side ? u[3] : u[2], v3 = side ? u[4] : u[3],
            v4 = side ? u[5] : u[4];
    T b0, b1, b2;
    js_betas(v0, v1, v2, v3, v4, b0, b1, b2);
    // 2 u0 - 7 u1 + 11 u2 (left, third candidate), 2 u5 - 7 u4 + 11 u3 (right, first)
    const T g = mul_pow2<1>(side ? u[5] : u[0]) - T(7.0) * (side ? u[4] : u[1]) + T(11.0) * v2;
    const T e0 = weps + b0, e1 = weps + b1, e2 = weps + b2;
    const T r = weno_combine_exact<T, U>(e0 * e0, e1 * e1, e2 * e2, side ? T(0.1) : T(0.3), T(0.6),
                                         side ? T(0.3) : T(0.1), side ? g : f1, side ? f1 : f2, side ? f2 : g) /
                T(6.0);
    left = side ? left : r;
    right = r;
  }
}

// Largest high word (sign cleared) of differences, for ffw::covers.
__device__ __forceinline__ uint32_t max_magnitude(f64 a, f64 b) { return max(ffw::magnitude(a.v), ffw::magnitude(b.v)); }
__device__ __forceinline__ uint32_t max_magnitude(uint32_t a, uint32_t b, f64 c) {
  return max(max(a, b), ffw::magnitude(c.v));
}

// u plus (sg = 1) or minus the weighted slope of a cell's face state: near and
// mid differences dn (across the face), dm and far ones df (behind the cell), fn
// (beyond the face).
__device__ __forceinline__ f64 face_slope(f64 dn, f64 fn, f64 dm, f64 df, double c_near, double c_mid, double c_far) {
  // candidates less the cell's value (x6): 4 dn - fn, 2 dn + dm, 5 dm - 2 df
  return fma(f64(c_near), fma(f64(4.0), dn, -fn),
             fma(f64(c_mid), fma(f64(2.0), dn, dm), f64(xmul(ffw::twice(c_far), fma(f64(2.5), dm, -df).v))));
}

// Both states of one field at the face between u2 and u3 with float-pair weights
// (ffw.cuh): 19 FP64 operations, where the FP64 weights below take 69.
__device__ __forceinline__ void weno5_lr_ffw(f64 u2, f64 u3, f64 d0, f64 d1, f64 d2, f64 d3, f64 d4, f64 weps,
                                             f64& left, f64& right) {
  const ffw::ff w = ffw::eps75(weps.v);
  const ffw::ff f0 = ffw::from_double(d0.v), f1 = ffw::from_double(d1.v), f2 = ffw::from_double(d2.v),
                f3 = ffw::from_double(d3.v), f4 = ffw::from_double(d4.v);
  double cn, cm, cf;
  ffw::face_weights(ffw::side(f2, f3, w), ffw::centre(f1, f2, w), ffw::side(f1, f0, w), cn, cm, cf);
  left = u2 + face_slope(d2, d3, d1, d0, cn, cm, cf);
  ffw::face_weights(ffw::side(f2, f1, w), ffw::centre(f2, f3, w), ffw::side(f3, f4, w), cn, cm, cf);
  right = u3 - face_slope(d2, d1, d3, d4, cn, cm, cf);
}

// The same in df64, whose values already are float pairs.
__device__ __forceinline__ ffw::ff as_pair(df64 a) { return ffw::ff{a.hi, a.lo}; }
__device__ __forceinline__ df64 from_pair(ffw::ff a) { return df64(a.h, a.l); }
__device__ __forceinline__ df64 scaled(float c, df64 a) { return df64(c * a.hi, c * a.lo); }  // c a power of two
__device__ __forceinline__ float max_head(df64 a, df64 b, df64 c, df64 d) {
  return fmaxf(fmaxf(fabsf(a.hi), fabsf(b.hi)), fmaxf(fabsf(c.hi), fabsf(d.hi)));
}
__device__ __forceinline__ df64 face_slope(df64 dn, df64 fn, df64 dm, df64 df, ffw::ff c_near, ffw::ff c_mid,
                                           ffw::ff c_far) {
  return from_pair(c_near) * (scaled(4.0f, dn) - fn) +
         (from_pair(c_mid) * (scaled(2.0f, dn) + dm) + from_pair(ffw::pow2(2.0f, c_far)) * (df64(2.5f, 0.0f) * dm - df));
}
__device__ __forceinline__ void weno5_lr_ffw(df64 u2, df64 u3, df64 d0, df64 d1, df64 d2, df64 d3, df64 d4, df64 weps,
                                             df64& left, df64& right) {
  const ffw::ff w = ffw::scale(0.75f, as_pair(weps));
  const ffw::ff f0 = as_pair(d0), f1 = as_pair(d1), f2 = as_pair(d2), f3 = as_pair(d3), f4 = as_pair(d4);
  ffw::ff cn, cm, cf;
  ffw::face_weights(ffw::side(f2, f3, w), ffw::centre(f1, f2, w), ffw::side(f1, f0, w), cn, cm, cf);
  left = u2 + face_slope(d2, d3, d1, d0, cn, cm, cf);
  ffw::face_weights(ffw::side(f2, f1, w), ffw::centre(f2, f3, w), ffw::side(f3, f4, w), cn, cm, cf);
  right = u3 - face_slope(d2, d1, d3, d4, cn, cm, cf);
}

// Both reconstructions of one field at one face (the right stencil is the left
// one shifted by a cell), FAST: native double shares one divide
// between the two; float and df64 take reciprocal weights.
template <class T>
__device__ __forceinline__ void weno5_lr_fast(T u0, T u1, T u2, T u3, T u4, T u5, T weps, T& left, T& right) {
  // first differences d_m = u_{m+1} - u_m, second differences D_m = d_m - d_{m-1}
  // (centred on u_m), shared by the two stencils; each Jiang-Shu indicator is
  // 13/12 D^2 + 1/4 s^2 with s a combination of two first differences.
  const T d0 = u1 - u0, d1 = u2 - u1, d2 = u3 - u2, d3 = u4 - u3, d4 = u5 - u4;
  if constexpr (is_native_f64<T>) {
    if (ffw::covers(max_magnitude(max_magnitude(d0, d1), max_magnitude(d2, d3), d4), weps.v)) {
      weno5_lr_ffw(u2, u3, d0, d1, d2, d3, d4, weps, left, right);
      return;
    }
  }
  if constexpr (std::is_same<T, df64>::value) {
    if (ffw::covers_pair(fmaxf(max_head(d0, d1, d2, d3), fabsf(d4.hi)), weps.hi)) {
      weno5_lr_ffw(u2, u3, d0, d1, d2, d3, d4, weps, left, right);
      return;
    }
  }
  const T D1 = d1 - d0, D2 = d2 - d1, D3 = d3 - d2, D4 = d4 - d3;
  // indicators scaled by 4 (see kC43): 4 eps + (13/3) D^2 + s^2
  const T w4 = T(4.0) * weps;
  const T C1 = T(kC43) * D1 * D1 + w4, C2 = T(kC43) * D2 * D2 + w4, C3 = T(kC43) * D3 * D3 + w4,
          C4 = T(kC43) * D4 * D4 + w4;
  const T sl0 = d3 - T(3.0) * d2, sl1 = d1 + d2, sl2 = T(3.0) * d1 - d0;  // left:  stencils 2-4, 1-3, 0-2
  const T sr0 = d4 - T(3.0) * d3, sr1 = d2 + d3, sr2 = T(3.0) * d2 - d1;  // right: stencils 3-5, 2-4, 1-3
  const T el0 = sl0 * sl0 + C3, el1 = sl1 * sl1 + C2, el2 = sl2 * sl2 + C1;
  const T er0 = sr0 * sr0 + C4, er1 = sr1 * sr1 + C3, er2 = sr2 * sr2 + C2;
  // Candidate polynomials (x6) less six times the centre value, from the same
  // differences: left 6 u2 + (4 d2 - d3, d1 + 2 d2, 5 d1 - 2 d0), right 6 u3 +
  // (d1 - 4 d2, -(2 d2 + d3), 2 d4 - 5 d3); each face state is its centre value
  // plus the weighted slope / 6 (no 6 u2 formed and cancelled).
  const T gl0 = d2 - sl0, gl1 = sl1 + d2, gl2 = T(2.0) * sl2 - d1;
  const T gr2 = -d2 - sr2, gr1 = -d2 - sr1, gr0 = T(2.0) * sr0 + d3;
  // The right reconstruction takes its stencils in the mirror order of the left
  // one (1-3, 2-4, 3-5 against 2-4, 1-3, 0-2), so that for mirror-image inputs
  // (u_k -> u_{5-k}, as across a reflecting wall: d_m -> -d_{4-m}) it performs
  // the left one's operations on bit-identical values and the two face states
  // are exact mirrors, as in the reference's arithmetic.
  if constexpr (is_native_f64<T>) {
    // linear weights scaled by 10 -- (3, 6, 1) -- and the 1/6 of the candidate
    // polynomials applied once to the shared divide
    f64 P0, P1, P2, nl, dl, nr, dr;
    weno_nd_products(el0, el1, el2, P0, P1, P2);
    weno_nd_combine(P0, P1, P2, gl0, gl1, gl2, nl, dl);
    weno_nd_products(er2, er1, er0, P0, P1, P2);
    weno_nd_combine(P0, P1, P2, gr2, gr1, gr0, nr, dr);
    div_pair(nl, dl, nr, dr, left, right, 6.0, u2, u3);
  } else {
    left = u2 + weno_combine<T>(el0, el1, el2, T(0.3), T(0.6), T(0.1), gl0, gl1, gl2, T(6.0));
    right = u3 + weno_combine<T>(er2, er1, er0, T(0.3), T(0.6), T(0.1), gr2, gr1, gr0, T(6.0));
  }
}

// Both face states of one cell u[2] of a field from its five cells, component-wise
// pass 1: `lf` at its left face, `rf` at its right face.  The operations are those
// of weno5_lr_fast seen from the cell (indicators and weight products once for
// both states), odd under the mirror image of the stencil.
template <class T>
__device__ __forceinline__ void weno5_cell_fast(const T u[5], T weps, T& lf, T& rf) {
  const T d0 = u[1] - u[0], d1 = u[2] - u[1], d2 = u[3] - u[2], d3 = u[4] - u[3];
  if constexpr (is_native_f64<T>) {
    if (ffw::covers(max(max_magnitude(d0, d1), max_magnitude(d2, d3)), weps.v)) {
      const ffw::ff w = ffw::eps75(weps.v);
      const ffw::ff f0 = ffw::from_double(d0.v), f1 = ffw::from_double(d1.v), f2 = ffw::from_double(d2.v),
                    f3 = ffw::from_double(d3.v);
      const ffw::ff qr = ffw::side(f2, f3, w), qm = ffw::centre(f1, f2, w), ql = ffw::side(f1, f0, w);
      double cn, cm, cf;
      ffw::face_weights(qr, qm, ql, cn, cm, cf);
      rf = u[2] + face_slope(d2, d3, d1, d0, cn, cm, cf);
      ffw::face_weights(ql, qm, qr, cn, cm, cf);
      lf = u[2] - face_slope(d1, d0, d2, d3, cn, cm, cf);
      return;
    }
  }
  const T D1 = d1 - d0, D2 = d2 - d1, D3 = d3 - d2;
  const T w4 = T(4.0) * weps;
  const T sr = d3 - T(3.0) * d2, sm = d1 + d2, sl = T(3.0) * d1 - d0;
  const T er = sr * sr + (T(kC43) * D3 * D3 + w4), em = sm * sm + (T(kC43) * D2 * D2 + w4),
          el = sl * sl + (T(kC43) * D1 * D1 + w4);
  // slopes (x6) of the stencils reaching over the face, central and behind the cell
  const T rn = d2 - sr, rm = sm + d2, rr = T(2.0) * sl - d1;
  const T ln = d1 + sl, lm = sm + d1, ll = -d2 - T(2.0) * sr;
  if constexpr (is_native_f64<T>) {
    T Pr, Pm, Pl, nr, dr, nl, dl;
    weno_nd_products(er, em, el, Pr, Pm, Pl);
    weno_nd_combine(Pr, Pm, Pl, rn, rm, rr, nr, dr);
    weno_nd_combine(Pl, Pm, Pr, ln, lm, ll, nl, dl);
    div_pair(nr, dr, -nl, dl, rf, lf, 6.0, u[2], u[2]);
  } else {
    const T ar = inv_square(er), am = inv_square(em), al = inv_square(el);
    const T r0 = T(0.3) * ar, m0 = T(0.6) * am, l0 = T(0.1) * al, l1 = T(0.3) * al, r1 = T(0.1) * ar;
    rf = u[2] + qdiv<T, true>(r0 * rn + m0 * rm + l0 * rr, (r0 + m0 + l0) * T(6.0));
    lf = u[2] - qdiv<T, true>(l1 * ln + m0 * lm + r1 * ll, (l1 + m0 + r1) * T(6.0));
  }
}

// The same in the reference's operations (weno.rs:214-257): the left-biased state
// at the right face and the right-biased one at the left face share the indicators.
template <class T>
__device__ __forceinline__ void weno5_cell_exact(const T u[5], T weps, T& lf, T& rf) {
  T b0, b1, b2;
  js_betas(u[0], u[1], u[2], u[3], u[4], b0, b1, b2);
  const T e0 = weps + b0, e1 = weps + b1, e2 = weps + b2;
  const T s0 = e0 * e0, s1 = e1 * e1, s2 = e2 * e2;
  const T fu = T(5.0) * u[2], el = T(11.0) * u[2], two = mul_pow2<1>(u[2]);
#pragma unroll 1
  for (int side = 0; side < 2; ++side) {  // left face (right-biased), then right face
    // -u4 + 5 u3 + 2 u2, -u1 + 5 u2 + 2 u3, 2 u0 - 7 u1 + 11 u2 at the right face;
    // 2 u4 - 7 u3 + 11 u2, -u3 + 5 u2 + 2 u1, -u0 + 5 u1 + 2 u2 at the left one
    const T a = side ? u[4] : u[0], b = side ? u[3] : u[1], c = side ? u[1] : u[3], d = side ? u[0] : u[4];
    const T near = -a + T(5.0) * b + two;
    const T mid = -c + fu + mul_pow2<1>(b);
    const T far = mul_pow2<1>(d) - T(7.0) * c + el;
    const T r = weno_combine_exact<T>(s0, s1, s2, side ? T(0.3) : T(0.1), T(0.6), side ? T(0.1) : T(0.3),
                                      side ? near : far, mid, side ? far : near) /
                T(6.0);
    lf = side ? lf : r;
    rf = r;
  }
}

// FAST float: the four fields' left/right reconstructions as two packed pairs
// (fields 0,1 and 2,3) on the FP32x2 instructions; field 2 takes weps2.
__device__ __forceinline__ void weno5_lr_fast_f32_pairs(const float c[6][4], float weps, float left[4],
                                                        float right[4], float weps2) {
#pragma unroll
  for (int f = 0; f < 4; f += 2) {
    f32x2 l, r;
    weno5_lr_fast<f32x2>(f32x2(c[0][f], c[0][f + 1]), f32x2(c[1][f], c[1][f + 1]), f32x2(c[2][f], c[2][f + 1]),
                         f32x2(c[3][f], c[3][f + 1]), f32x2(c[4][f], c[4][f + 1]), f32x2(c[5][f], c[5][f + 1]),
                         f == 0 ? f32x2(weps) : f32x2(weps2, weps), l, r);
    left[f] = l.v.x;
    left[f + 1] = l.v.y;
    right[f] = r.v.x;
    right[f + 1] = r.v.y;
  }
}

// weno.rs:262-303: both Gauss-point values from one 5-cell stencil.  The
// smoothness indicators are shared (the reference recomputes identical values).
// FAST Gauss-point pair from the centre value, the slopes h_k of the three
// candidate polynomials and the (scaled) indicators f_k: native double in the
// common-denominator form, float and df64 with reciprocals.  The candidates
// are q2 +- S h_k, so each weighted value is q2 plus S times a weighted slope.
template <class T>
__device__ __forceinline__ void gq_weights(T q2, T h0, T h1, T h2, T f0, T f1, T f2, T& ra, T& rb) {
  const T S = T(kSqrt3_12);
  if constexpr (is_native_f64<T>) {
    weno_range<120>(f0, f1, f2);
    const f64 s0 = f0 * f0, s1 = f1 * f1, s2 = f2 * f2;
    const f64 P0 = s1 * s2, P1 = s0 * s2, P2 = s0 * s1;
    // linear weights divided by the centre one (a common factor): point a
    // weighs (r0 P0, P1, r2 P2), point b the mirror (r2 P0, P1, r0 P2)
    constexpr double r0 = kGqA0 / kGqA1, r2 = kGqA2 / kGqA1;
    const f64 u0 = P0 * h0, u1 = P1 * h1, u2 = P2 * h2;
    const f64 sa = fma(r0, P0, fma(r2, P2, P1)), sb = fma(r2, P0, fma(r0, P2, P1));
    const f64 t = S * f64(f64fast::rcp2(f64(sa * sb).v));  // scales the weighted slopes only
    // point a: candidates (q2 + S h0, q2 - S h1, q2 - S h2); point b: the mirror
    ra = fma(r0, u0, fma(-r2, u2, -u1)) * (sb * t) + q2;
    rb = fma(r0, u2, fma(-r2, u0, u1)) * (sa * t) + q2;
  } else {
    if constexpr (std::is_same<T, df64>::value) weno_range(f0, f1, f2);
    const T r0 = inv_square(f0), r1 = inv_square(f1), r2 = inv_square(f2);
    const T ca0 = T(kGqA0 / kGqA1) * r0, ca1 = r1, ca2 = T(kGqA2 / kGqA1) * r2;
    const T cb0 = T(kGqA2 / kGqA1) * r0, cb2 = T(kGqA0 / kGqA1) * r2;
    ra = qdiv<T, true>((ca0 * h0 - ca1 * h1 - ca2 * h2) * S, ca0 + ca1 + ca2) + q2;
    rb = qdiv<T, true>((ca1 * h1 + cb2 * h2 - cb0 * h0) * S, cb0 + ca1 + cb2) + q2;
  }
}

// The Gauss-point pair of one cell with first differences d0, d1 | d2, d3 (their
// float pairs f), float-pair weights.
__device__ __forceinline__ void gq_ffw(f64 q, f64 d0, f64 d1, f64 d2, f64 d3, ffw::ff f0, ffw::ff f1, ffw::ff f2,
                                       ffw::ff f3, ffw::ff w, f64& ra, f64& rb) {
  constexpr ffw::ff r0 = ffw::constant(kGqA0 / kGqA1), r2 = ffw::constant(kGqA2 / kGqA1), S = ffw::constant(kSqrt3_12);
  const ffw::ff qr = ffw::side(f2, f3, w), qm = ffw::centre(f1, f2, w), ql = ffw::side(f1, f0, w);
  const f64 hr = fma(f64(-3.0), d2, d3), hm = d1 + d2, hl = fma(f64(3.0), d1, -d0);
  double cr, cm, cl;
  ffw::gauss_weights(qr, qm, ql, r0, r2, S, cr, cm, cl);
  ra = q + fma(f64(cr), hr, fma(f64(-cm), hm, f64(xmul(-cl, hl.v))));
  ffw::gauss_weights(qr, qm, ql, r2, r0, S, cr, cm, cl);
  rb = q + fma(f64(-cr), hr, fma(f64(cm), hm, f64(xmul(cl, hl.v))));
}

__device__ __forceinline__ void gq_ffw(df64 q, df64 d0, df64 d1, df64 d2, df64 d3, df64 weps, df64& ra, df64& rb) {
  constexpr ffw::ff r0 = ffw::constant(kGqA0 / kGqA1), r2 = ffw::constant(kGqA2 / kGqA1), S = ffw::constant(kSqrt3_12);
  const ffw::ff w = ffw::scale(0.75f, as_pair(weps)), f0 = as_pair(d0), f1 = as_pair(d1), f2 = as_pair(d2), f3 = as_pair(d3);
  const ffw::ff qr = ffw::side(f2, f3, w), qm = ffw::centre(f1, f2, w), ql = ffw::side(f1, f0, w);
  const df64 three(3.0f, 0.0f), hr = d3 - three * d2, hm = d1 + d2, hl = three * d1 - d0;
  ffw::ff cr, cm, cl;
  ffw::gauss_weights(qr, qm, ql, r0, r2, S, cr, cm, cl);
  ra = q + (from_pair(cr) * hr - (from_pair(cm) * hm + from_pair(cl) * hl));
  ffw::gauss_weights(qr, qm, ql, r2, r0, S, cr, cm, cl);
  rb = q - (from_pair(cr) * hr - (from_pair(cm) * hm + from_pair(cl) * hl));
}

// Two neighbouring 5-cell stencils (q0..q4 and q1..q5), FAST: both
// Gauss-point pairs, sharing the first and second differences.
template <class T>
__device__ __forceinline__ void weno5_gq_two(T q0, T q1, T q2, T q3, T q4, T q5, T weps, T& raA, T& rbA, T& raB,
                                             T& rbB) {
  const T d0 = q1 - q0, d1 = q2 - q1, d2 = q3 - q2, d3 = q4 - q3, d4 = q5 - q4;
  if constexpr (is_native_f64<T>) {
    if (ffw::covers(max_magnitude(max_magnitude(d0, d1), max_magnitude(d2, d3), d4), weps.v)) {
      const ffw::ff w = ffw::eps75(weps.v);
      const ffw::ff f0 = ffw::from_double(d0.v), f1 = ffw::from_double(d1.v), f2 = ffw::from_double(d2.v),
                    f3 = ffw::from_double(d3.v), f4 = ffw::from_double(d4.v);
      gq_ffw(q2, d0, d1, d2, d3, f0, f1, f2, f3, w, raA, rbA);
      gq_ffw(q3, d1, d2, d3, d4, f1, f2, f3, f4, w, raB, rbB);
      return;
    }
  }
  const T D1 = d1 - d0, D2 = d2 - d1, D3 = d3 - d2, D4 = d4 - d3;
  const T w4 = T(4.0) * weps;
  const T C1 = T(kC43) * D1 * D1 + w4, C2 = T(kC43) * D2 * D2 + w4, C3 = T(kC43) * D3 * D3 + w4,
          C4 = T(kC43) * D4 * D4 + w4;
  const T hA0 = d3 - T(3.0) * d2, hA1 = d1 + d2, hA2 = T(3.0) * d1 - d0;
  const T hB0 = d4 - T(3.0) * d3, hB1 = d2 + d3, hB2 = T(3.0) * d2 - d1;
  gq_weights<T>(q2, hA0, hA1, hA2, hA0 * hA0 + C3, hA1 * hA1 + C2, hA2 * hA2 + C1, raA, rbA);
  gq_weights<T>(q3, hB0, hB1, hB2, hB0 * hB0 + C4, hB1 * hB1 + C3, hB2 * hB2 + C2, raB, rbB);
}

template <class T, bool FAST, int U = 1>
__device__ __forceinline__ void weno5_gq_pair(T q0, T q1, T q2, T q3, T q4, T& ra, T& rb, T weps) {
  const T S = T(kSqrt3_12);
  if constexpr (FAST) {
    // difference form (as in weno5_lr_fast): the one-sided indicator terms are
    // the polynomial slopes g0, g2 and the centred one is g1/S
    const T d0 = q1 - q0, d1 = q2 - q1, d2 = q3 - q2, d3 = q4 - q3;
    if constexpr (is_native_f64<T>) {
      if (ffw::covers(max(max_magnitude(d0, d1), max_magnitude(d2, d3)), weps.v)) {
        gq_ffw(q2, d0, d1, d2, d3, ffw::from_double(d0.v), ffw::from_double(d1.v), ffw::from_double(d2.v),
               ffw::from_double(d3.v), ffw::eps75(weps.v), ra, rb);
        return;
      }
    }
    if constexpr (std::is_same<T, df64>::value) {
      if (ffw::covers_pair(max_head(d0, d1, d2, d3), weps.hi)) {
        gq_ffw(q2, d0, d1, d2, d3, weps, ra, rb);
        return;
      }
    }
    const T D1 = d1 - d0, D2 = d2 - d1, D3 = d3 - d2;
    const T h0 = d3 - T(3.0) * d2;  // 3 q2 - 4 q3 + q4
    const T h1 = d1 + d2;           // q3 - q1
    const T h2 = T(3.0) * d1 - d0;  // 3 q2 - 4 q1 + q0
    // indicators scaled by 4 (see kC43): 4 eps + (13/3) D^2 + h^2
    const T w4 = T(4.0) * weps;
    const T f0 = h0 * h0 + (T(kC43) * D3 * D3 + w4);
    const T f1 = h1 * h1 + (T(kC43) * D2 * D2 + w4);
    const T f2 = h2 * h2 + (T(kC43) * D1 * D1 + w4);
    gq_weights<T>(q2, h0, h1, h2, f0, f1, f2, ra, rb);
  } else {
    T b0, b1, b2;
    js_betas(q0, q1, q2, q3, q4, b0, b1, b2);
    const T e0 = weps + b0, e1 = weps + b1, e2 = weps + b2;
    const T s0 = e0 * e0, s1 = e1 * e1, s2 = e2 * e2;
    const T g0 = (T(3.0) * q2 - mul_pow2<2>(q3) + q4) * S;
    const T g2 = (T(3.0) * q2 - mul_pow2<2>(q1) + q0) * S;
    // point a: q2 + g0, q2 - (q3 - q1) S, q2 - g2; point b: the mirror (negation
    // is exact: -q1 + q3 and q1 - q3 are opposite)
    const T g1 = (-q1 + q3) * S;
#pragma unroll(U == 1 ? 1 : 2)
    for (int pt = 0; pt < 2; ++pt) {
      const T r = weno_combine_exact<T, U>(s0, s1, s2, pt ? T(kGqA2) : T(kGqA0), T(kGqA1), pt ? T(kGqA0) : T(kGqA2),
                                        q2 + (pt ? -g0 : g0), q2 - (pt ? -g1 : g1), q2 - (pt ? -g2 : g2));
      ra = pt ? ra : r;
      rb = r;
    }
  }
}

// ---------------------------------------------------------------------------
// Characteristic projection (weno.rs:13-205)
// ---------------------------------------------------------------------------
// FAST Roe-average inputs of one cell: with r = 1/sqrt(rho) (one reciprocal
// square root), sqrt(rho) = rho r, 1/rho = r r, sqrt(rho) u = m r and
// sqrt(rho) v = n r; E + p with the clamped pressure.
template <class T>
struct RoeSide {
  T sq, r, i, a, b, ep;  // sqrt(rho), 1/sqrt(rho), 1/rho, m r, n r, E + p
};

template <class T>
__device__ __forceinline__ RoeSide<T> roe_side(const T u[4], T gamma) {
  RoeSide<T> s;
  roots(vmax(u[0], T(kEps)), s.sq, s.r, s.i);
  // kinetic energy (m^2 + n^2) / (2 rho): the velocities themselves are not needed
  const T p = vmax<T>((gamma - T(1.0)) * (u[3] - T(0.5) * ((u[1] * u[1] + u[2] * u[2]) * s.i)), T(kEps));
  s.a = u[1] * s.r;
  s.b = u[2] * s.r;
  s.ep = u[3] + p;
  return s;
}

// Roe average of the face between sides L and R (weno.rs:13-52), FAST: m_l,
// n_l are the left cell's momenta.  Also returns 1/c_roe and 1/rho_roe (ic,
// irho) for the eigenvectors; 1/rho_roe = r_l r_r.
template <class T>
__device__ __forceinline__ void roe_face(const RoeSide<T>& L, const RoeSide<T>& R, T m_l, T n_l, T gamma,
                                         T& rho_roe, T& u_roe, T& v_roe, T& h_roe, T& c_roe, T& ic, T& irho) {
  const T id = qrcp<T, true>(L.sq + R.sq);
  u_roe = mul_add<T>(m_l, L.r, R.a) * id;
  v_roe = mul_add<T>(n_l, L.r, R.b) * id;
  h_roe = mul_add<T>(L.ep, L.r, R.ep * R.r) * id;
  const T kin = T(0.5) * (u_roe * u_roe + v_roe * v_roe);
  const T c2 = vmax<T>((gamma - T(1.0)) * (h_roe - kin), T(kEps) * vmax<T>(L.i, R.i));
  if constexpr (is_native_f64<T>) {
    c_roe = sqrt(c2);
    ic = T(1.0) / c_roe;
  } else {
    T i;
    roots(c2, c_roe, ic, i);
  }
  rho_roe = L.sq * R.sq;
  irho = L.r * R.r;
}

// Roe average of two conserved cells, weno.rs:13-52 (FAST: roe_side and
// roe_face, two reciprocal square roots, one divide and one more reciprocal
// square root for c).
template <class T, bool FAST>
__device__ __forceinline__ void roe_avg(const T ul[4], const T ur[4], T gamma, T& rho_roe, T& u_roe, T& v_roe,
                                        T& h_roe, T& c_roe, T& ic, T& irho) {
  if constexpr (FAST) {
    roe_face(roe_side(ul, gamma), roe_side(ur, gamma), ul[1], ul[2], gamma, rho_roe, u_roe, v_roe, h_roe, c_roe, ic,
             irho);
  } else {
    (void)ic;
    (void)irho;
    const T rho_l = vmax(ul[0], T(kEps));
    const T rho_r = vmax(ur[0], T(kEps));
    const T sqrt_l = sqrt(rho_l);
    const T sqrt_r = sqrt(rho_r);
    const T denom = sqrt_l + sqrt_r;
    const T u_l = ul[1] / rho_l, v_l = ul[2] / rho_l;
    const T u_r = ur[1] / rho_r, v_r = ur[2] / rho_r;
    const T p_l = vmax<T>((gamma - T(1.0)) * (ul[3] - T(0.5) * rho_l * (u_l * u_l + v_l * v_l)), T(kEps));
    const T p_r = vmax<T>((gamma - T(1.0)) * (ur[3] - T(0.5) * rho_r * (u_r * u_r + v_r * v_r)), T(kEps));
    const T h_l = (ul[3] + p_l) / rho_l;
    const T h_r = (ur[3] + p_r) / rho_r;
    u_roe = (sqrt_l * u_l + sqrt_r * u_r) / denom;
    v_roe = (sqrt_l * v_l + sqrt_r * v_r) / denom;
    h_roe = (sqrt_l * h_l + sqrt_r * h_r) / denom;
    const T kin = T(0.5) * (u_roe * u_roe + v_roe * v_roe);
    const T c2 = vmax<T>((gamma - T(1.0)) * (h_roe - kin), T(kEps) / vmin(rho_l, rho_r));
    c_roe = sqrt(c2);
    rho_roe = sqrt_l * sqrt_r;
  }
}

// Left eigenvectors, weno.rs:76-107 (x) and weno.rs:136-167 (y), in the
// reference's operation order (FAST callers use CharScalars / project_left).
template <class T, bool Y>
__device__ __forceinline__ void left_eig(T rho, T u, T v, T c, T gamma, T L[4][4]) {
  const T g1 = gamma - T(1.0);
  const T kin = T(0.5) * (u * u + v * v);
  const T vn = Y ? v : u;
  const T rc = rho * c;
  const T inv_rc = T(1.0) / rc;
  const T inv_c2 = T(1.0) / (c * c);
  const T a = g1 * kin / (mul_pow2<1>(c) * c);
  const T b = vn / mul_pow2<1>(c);
  const T gu = mul_pow2<-1>(T(-g1 * u * inv_c2));
  const T gv = mul_pow2<-1>(T(-g1 * v * inv_c2));
  const T gg = mul_pow2<-1>(T(g1 * inv_c2));
  const T hr = T(0.5) * inv_rc;
  L[0][0] = a + b;
  L[3][0] = a - b;
  if constexpr (!Y) {
    L[0][1] = gu - hr; L[0][2] = gv; L[0][3] = gg;
    L[3][1] = gu + hr; L[3][2] = gv; L[3][3] = gg;
    L[2][0] = -v / rho; L[2][1] = T(0.0); L[2][2] = T(1.0) / rho; L[2][3] = T(0.0);
  } else {
    L[0][1] = gu; L[0][2] = gv - hr; L[0][3] = gg;
    L[3][1] = gu; L[3][2] = gv + hr; L[3][3] = gg;
    L[2][0] = -u / rho; L[2][1] = T(1.0) / rho; L[2][2] = T(0.0); L[2][3] = T(0.0);
  }
  L[1][0] = T(1.0) - g1 * kin * inv_c2;
  L[1][1] = g1 * u * inv_c2;
  L[1][2] = g1 * v * inv_c2;
  L[1][3] = -g1 * inv_c2;
}

// Right eigenvectors, weno.rs:113-131 (x) and weno.rs:171-189 (y).
template <class T, bool Y>
__device__ __forceinline__ void right_eig(T rho, T u, T v, T h, T c, T R[4][4]) {
  const T kin = T(0.5) * (u * u + v * v);
  R[0][0] = T(1.0); R[0][1] = T(1.0); R[0][2] = T(0.0); R[0][3] = T(1.0);
  if constexpr (!Y) {
    R[1][0] = u - c; R[1][1] = u; R[1][2] = T(0.0); R[1][3] = u + c;
    R[2][0] = v; R[2][1] = v; R[2][2] = rho; R[2][3] = v;
    R[3][0] = h - u * c; R[3][1] = kin; R[3][2] = rho * v; R[3][3] = h + u * c;
  } else {
    R[1][0] = u; R[1][1] = u; R[1][2] = rho; R[1][3] = u;
    R[2][0] = v - c; R[2][1] = v; R[2][2] = T(0.0); R[2][3] = v + c;
    R[3][0] = h - v * c; R[3][1] = kin; R[3][2] = rho * u; R[3][3] = h + v * c;
  }
}

// weno.rs:197-205 mat4_vec4: every product accumulated from 0.0 in column
// order, as the reference does (FAST callers use project_left / project_right).
// 0.0 + x is x except for x = -0, which becomes +0: an integer select.
template <class T>
__device__ __forceinline__ T from_zero(T x) {
  if constexpr (is_native_f64<T>) return f64_bits(x) == (long long)0x8000000000000000ull ? T(0.0) : x;
  else return T(0.0) + x;
}
template <class T>
__device__ __forceinline__ T row_vec4(const T row[4], const T x[4]) {
  T acc = from_zero<T>(row[0] * x[0]);
#pragma unroll
  for (int c = 1; c < 4; ++c) acc = acc + row[c] * x[c];
  return acc;
}
template <class T>
__device__ __forceinline__ void mat4_vec4(const T M[4][4], const T x[4], T out[4]) {
#pragma unroll
  for (int r = 0; r < 4; ++r) out[r] = row_vec4<T>(M[r], x);
}

// FAST products with the eigenvector matrices of weno.rs:76-189, written from
// their structure instead of a 4x4 product.  With G = (gamma-1)/c^2,
// kin = (u^2+v^2)/2, b = u_n/(2c), hr = 1/(2 rho c) and Z = kin q0 - u q1 - v q2 + q3:
//   L q = ( G Z/2 + (b q0 - hr q_n),  q0 - G Z,  (q_t - u_t q0)/rho,  G Z/2 - (b q0 - hr q_n) )
// (n the normal and t the tangential momentum index), and with s = w0+w1+w3:
//   R w = ( s,  u s + [c (w3-w0) | rho w2],  v s + [rho w2 | c (w3-w0)],  R3 . w ).
// The shear field is carried as rho w2 = q_t - u_t q0: WENO5 is homogeneous
// when its epsilon scales with the square of the field (the indicators are
// quadratic, the candidates linear), so reconstructing rho w2 with
// eps rho^2 gives rho times the reconstruction of w2, which is what R needs;
// the 1/rho of L and the rho of R drop out.
template <class T>
struct CharScalars {
  T u, v, c, rho, kin, G, G2, b, hr, h;
};

template <class T, bool Y>
__device__ __forceinline__ void project_parts(const CharScalars<T>& k, const T q[4], T& Z, T& Yv) {
  Z = (k.kin * q[0] + q[3]) - k.u * q[1] - k.v * q[2];
  Yv = k.b * q[0] - k.hr * q[Y ? 2 : 1];
}
template <class T, bool Y>
__device__ __forceinline__ CharScalars<T> char_scalars(T rho, T u, T v, T h, T c, T ic, T irho, T gamma) {
  CharScalars<T> k;
  k.u = u;
  k.v = v;
  k.c = c;
  k.rho = rho;
  k.h = h;
  k.kin = T(0.5) * (u * u + v * v);
  k.G = (gamma - T(1.0)) * (ic * ic);
  k.G2 = T(0.5) * k.G;
  const T ich = T(0.5) * ic;
  k.b = (Y ? v : u) * ich;
  k.hr = ich * irho;
  return k;
}
// Field f of a cell from its parts: G2 Z + Yv, q0 - G Z, q_t - u_t q0, G2 Z - Yv
// as one product and one addend.
template <class T, bool Y>
__device__ __forceinline__ T char_field(const CharScalars<T>& k, const T q[4], T Z, T Yv, int f) {
  const T A = f == 1 ? -k.G : (f == 2 ? -(Y ? k.u : k.v) : k.G2);
  const T X = f == 2 ? q[0] : Z;
  const T B = f == 0 ? Yv : (f == 1 ? q[0] : (f == 2 ? q[Y ? 1 : 2] : -Yv));
  return mul_add<T>(A, X, B);
}
template <class T, bool Y>
__device__ __forceinline__ void project_left(const CharScalars<T>& k, const T q[4], T w[4]) {
  // Z from q3 upwards and G Z / 2 +- Yv as one FMA each: nine operations
  T Z, Yv;
  project_parts<T, Y>(k, q, Z, Yv);
  w[0] = k.G2 * Z + Yv;
  w[1] = q[0] - k.G * Z;
  w[2] = q[Y ? 1 : 2] - (Y ? k.u : k.v) * q[0];  // rho w2
  w[3] = k.G2 * Z - Yv;
}
template <class T, bool Y>
__device__ __forceinline__ void project_right(const CharScalars<T>& k, const T w[4], T out[4]) {
  const T s = w[0] + w[1] + w[3];
  const T d = w[3] - w[0];
  const T un = Y ? k.v : k.u;
  out[0] = s;
  if constexpr (!Y) {
    out[1] = k.u * s + k.c * d;
    out[2] = k.v * s + w[2];
  } else {
    out[1] = k.u * s + w[2];
    out[2] = k.v * s + k.c * d;
  }
  out[3] = (k.h - un * k.c) * w[0] + k.kin * w[1] + (Y ? k.u : k.v) * w[2] + (k.h + un * k.c) * w[3];
}

// A double as the nearest-below float for a screening test: zero below the float
// range, NaN (which fails every comparison) above it.
__device__ __forceinline__ float screen_float(f64 x) {
  const uint32_t hi = (uint32_t)__double2hiint(x.v), e = hi & 0x7ff00000u;
  const uint32_t m = (__funnelshift_l((uint32_t)__double2loint(x.v), hi, 3) & 0x7fffffffu) ^ 0x40000000u;
  const float f = __uint_as_float(m | (hi & 0x80000000u));
  return e < (897u << 20) ? 0.0f : (e > (1150u << 20) ? __uint_as_float(0x7fffffffu) : f);
}
// Whether the density is positive and the pressure test E rho - |m|^2/2 >=
// eps rho / (gamma - 1) passes by 4e-6 of E rho (the float forms are within
// 5e-7 of it, and 3e-6 E rho exceeds the bound): the limiter has nothing to do.
__device__ __forceinline__ bool clearly_positive(const f64 q[4], f64 gamma) {
  const float r = screen_float(q[0]), m = screen_float(q[1]), n = screen_float(q[2]), e = screen_float(q[3]);
  const float er = e * r;
  return r > 1e-9f && e > 1e-3f && er - 0.5f * (m * m + n * n) > 4e-6f * er && gamma > f64(1.001);
}

// weno.rs:312-315 pressure ; weno.rs:327-352 Zhang-Shu limiter toward `ub`.
template <class T, bool FAST>
__device__ __forceinline__ T pp_pressure(const T q[4], T gamma) {
  if (q[0] <= T(0.0)) return T(0.0);
  return (gamma - T(1.0)) * (q[3] - qdiv<T, FAST>(T(0.5) * (q[1] * q[1] + q[2] * q[2]), q[0]));
}
template <class T, bool FAST>
__device__ __forceinline__ void pp_limit(T q[4], const T ub[4], T gamma) {
  // FAST native double: a float test, off the FP64 pipe, settles nearly every face
  if constexpr (FAST && is_native_f64<T>) {
    if (clearly_positive(q, gamma)) return;
  }
  if (q[0] < T(kEps)) {
    const T rho_bar = vmax(ub[0], T(kEps));
    const T theta = vmax<T>(vmin<T>(qdiv<T, FAST>(rho_bar - T(kEps), rho_bar - q[0]), T(1.0)), T(0.0));
#pragma unroll
    for (int k = 0; k < 4; ++k) q[k] = theta * (q[k] - ub[k]) + ub[k];
  }
  if constexpr (FAST) {
    // p < eps  <=>  (gamma-1)(E rho - |m|^2/2) < eps rho for rho > 0 (pp_pressure
    // is 0 for rho <= 0): the divide is only needed when the limiter acts.
    if (q[0] > T(0.0) &&
        !((gamma - T(1.0)) * (q[3] * q[0] - T(0.5) * (q[1] * q[1] + q[2] * q[2])) < T(kEps) * q[0]))
      return;
  }
  const T p_q = pp_pressure<T, FAST>(q, gamma);
  if (p_q < T(kEps)) {
    const T p_bar = vmax<T>(pp_pressure<T, FAST>(ub, gamma), T(kEps));
    const T theta = vmax<T>(vmin<T>(qdiv<T, FAST>(p_bar - T(kEps), p_bar - p_q), T(1.0)), T(0.0));
#pragma unroll
    for (int k = 0; k < 4; ++k) q[k] = theta * (q[k] - ub[k]) + ub[k];
  }
}

// ---------------------------------------------------------------------------
// Pass 1: normal-direction reconstruction of the two states at the interface
// between stencil cells 2 and 3 (weno.rs:390-454 characteristic,
// weno.rs:654-717 component-wise).  c[0..5] are the six cells along the normal.
// ---------------------------------------------------------------------------
template <class T, bool FAST, bool Y, bool CHAR>
__device__ __forceinline__ void pass1_face(const T c[6][4], T gamma, T ql[4], T qr[4], T weps) {
  if constexpr (!CHAR && FAST && is_f32<T>) {
    weno5_lr_fast_f32_pairs(c, weps, ql, qr, weps);
  } else if constexpr (!CHAR) {
#pragma unroll(kFieldUnroll<T>)
    for (int k = 0; k < 4; ++k) {
      T u[6], l, r;
#pragma unroll
      for (int s = 0; s < 6; ++s) u[s] = pick4(c[s], k);
      if constexpr (FAST) weno5_lr_fast<T>(u[0], u[1], u[2], u[3], u[4], u[5], weps, l, r);
      else weno5_lr_exact<T>(u, weps, l, r);
      put4(ql, k, l);
      put4(qr, k, r);
    }
  } else {
    T rho_a, u_a, v_a, h_a, c_a, ic_a = T(0.0), irho_a = T(0.0);
    roe_avg<T, FAST>(c[2], c[3], gamma, rho_a, u_a, v_a, h_a, c_a, ic_a, irho_a);
    // The reference projects cells 0..4 for the left state and 1..5 for the
    // right state with the same matrix (both faces use the Roe average of
    // cells 2|3), so six projections cover both.
    T chl[4], chr[4];
    if constexpr (FAST) {
      const CharScalars<T> k = char_scalars<T, Y>(rho_a, u_a, v_a, h_a, c_a, ic_a, irho_a, gamma);
      const T weps2 = weps * (rho_a * rho_a);  // epsilon of the shear field rho w2
      if constexpr (!is_f32<T>) {
        T Z[6], Yv[6];
#pragma unroll
        for (int s = 0; s < 6; ++s) project_parts<T, Y>(k, c[s], Z[s], Yv[s]);
#pragma unroll 1
        for (int f = 0; f < 4; ++f) {
          T w[6], l, r;
#pragma unroll
          for (int s = 0; s < 6; ++s) w[s] = char_field<T, Y>(k, c[s], Z[s], Yv[s], f);
          weno5_lr_fast<T>(w[0], w[1], w[2], w[3], w[4], w[5], f == 2 ? weps2 : weps, l, r);
          put4(chl, f, l);
          put4(chr, f, r);
        }
      } else {
        T w[6][4];
#pragma unroll
        for (int s = 0; s < 6; ++s) project_left<T, Y>(k, c[s], w[s]);
        weno5_lr_fast_f32_pairs(w, weps, chl, chr, weps2);
      }
      project_right<T, Y>(k, chl, ql);
      project_right<T, Y>(k, chr, qr);
    } else {
      T Lm[4][4];
      left_eig<T, Y>(rho_a, u_a, v_a, c_a, gamma, Lm);
#pragma unroll 1
      for (int f = 0; f < 4; ++f) {
        // characteristic field f of the six cells: row f of L times the cells
        T row[4], w[6], l, r;
        pick_row(Lm, f, row);
#pragma unroll
        for (int s = 0; s < 6; ++s) w[s] = row_vec4<T>(row, c[s]);
        weno5_lr_exact<T>(w, weps, l, r);
        put4(chl, f, l);
        put4(chr, f, r);
      }
      T Rm[4][4];
      right_eig<T, Y>(rho_a, u_a, v_a, h_a, c_a, Rm);
      mat4_vec4<T>(Rm, chl, ql);
      mat4_vec4<T>(Rm, chr, qr);
    }
    pp_limit<T, FAST>(ql, c[2], gamma);
    pp_limit<T, FAST>(qr, c[3], gamma);
  }
}

// Pass 1 of one face by the four lanes of a quad, lane f reconstructing field f:
// the operations of pass1_face, each on one lane only (the Roe average on all
// four), and the fields exchanged by shuffles.  Returns component f of q_l and
// q_r.  All 32 lanes of the warp call it.
template <class T>
__device__ __forceinline__ T quad_get(T x, int lane) {
  return T(__shfl_sync(0xffffffffu, x.v, lane, 4));
}
template <class T>
__device__ __forceinline__ void quad_gather(T x, T v[4]) {
#pragma unroll
  for (int k = 0; k < 4; ++k) v[k] = quad_get(x, k);
}
template <class T, bool FAST, bool Y, bool CHAR>
__device__ __forceinline__ void pass1_face_quad(const T c[6][4], int f, T gamma, T& ql_f, T& qr_f, T weps) {
  T w[6];
  if constexpr (!CHAR) {
#pragma unroll
    for (int s = 0; s < 6; ++s) w[s] = pick4(c[s], f);
    if constexpr (FAST) weno5_lr_fast<T>(w[0], w[1], w[2], w[3], w[4], w[5], weps, ql_f, qr_f);
    else weno5_lr_exact<T, 3>(w, weps, ql_f, qr_f);
  } else {
    T rho_a, u_a, v_a, h_a, c_a, ic_a = T(0.0), irho_a = T(0.0);
    roe_avg<T, FAST>(c[2], c[3], gamma, rho_a, u_a, v_a, h_a, c_a, ic_a, irho_a);
    T l, r, chl[4], chr[4], ql[4], qr[4];
    if constexpr (FAST) {
      const CharScalars<T> k = char_scalars<T, Y>(rho_a, u_a, v_a, h_a, c_a, ic_a, irho_a, gamma);
#pragma unroll
      for (int s = 0; s < 6; ++s) {
        T Z, Yv;
        project_parts<T, Y>(k, c[s], Z, Yv);
        w[s] = char_field<T, Y>(k, c[s], Z, Yv, f);
      }
      weno5_lr_fast<T>(w[0], w[1], w[2], w[3], w[4], w[5], f == 2 ? T(weps * (rho_a * rho_a)) : weps, l, r);
      quad_gather(l, chl);
      quad_gather(r, chr);
      project_right<T, Y>(k, chl, ql);
      project_right<T, Y>(k, chr, qr);
    } else {
      T M[4][4], row[4];
      left_eig<T, Y>(rho_a, u_a, v_a, c_a, gamma, M);
      pick_row(M, f, row);
#pragma unroll
      for (int s = 0; s < 6; ++s) w[s] = row_vec4<T>(row, c[s]);
      weno5_lr_exact<T, 3>(w, weps, l, r);
      quad_gather(l, chl);
      quad_gather(r, chr);
      right_eig<T, Y>(rho_a, u_a, v_a, h_a, c_a, M);
      pick_row(M, f, row);
      quad_gather(row_vec4<T>(row, chl), ql);
      quad_gather(row_vec4<T>(row, chr), qr);
    }
    pp_limit<T, FAST>(ql, c[2], gamma);
    pp_limit<T, FAST>(qr, c[3], gamma);
    ql_f = pick4(ql, f);
    qr_f = pick4(qr, f);
  }
}

// ---------------------------------------------------------------------------
// Interface Riemann solvers (riemann.rs:6-349).  Inputs are the face-averaged
// states and fluxes; `ql`/`qr` are the raw (unclamped) states.
// ---------------------------------------------------------------------------
template <class T, bool FAST, bool Y>
struct RiemannPre {
  T ql0, qr0, u_l, v_l, u_r, v_r, p_l, p_r, s_l, s_r, un_l, un_r;
};

// S = 2 (FAST): ql, qr are twice the face states (the sums of the two Gauss-point
// values, which saves the halving multiplies); the clamps then take 2 eps, so
// densities and pressures are exactly twice the clamped values and every
// velocity, enthalpy and wave speed is a ratio that the factor leaves alone.
template <class T, bool FAST, bool Y, int S = 1>
__device__ __forceinline__ RiemannPre<T, FAST, Y> riemann_pre(const T ql[4], const T qr[4], T gamma) {
  static_assert(S == 1 || FAST, "doubled states are a FAST form");
  RiemannPre<T, FAST, Y> r;
  r.ql0 = cmax<T, FAST>(ql[0], T(kEps * S));
  r.qr0 = cmax<T, FAST>(qr[0], T(kEps * S));
  T h_l, h_r, u_t, v_t, h_t;
  T sl = T(0.0), sr = T(0.0), rsl = T(0.0), rsr = T(0.0), il = T(0.0), ir = T(0.0);  // FAST: sqrt(rho), 1/sqrt(rho), 1/rho
  if constexpr (!FAST) {
    r.u_l = ql[1] / r.ql0; r.v_l = ql[2] / r.ql0;
    r.u_r = qr[1] / r.qr0; r.v_r = qr[2] / r.qr0;
  } else {
    roots(r.ql0, sl, rsl, il);
    roots(r.qr0, sr, rsr, ir);
    r.u_l = ql[1] * il; r.v_l = ql[2] * il;
    r.u_r = qr[1] * ir; r.v_r = qr[2] * ir;
  }
  // FAST: sqrt(rho)*u = q1/sqrt(rho) and sqrt(rho)*h = (E+p)/sqrt(rho); the
  // kinetic energy is (m^2 + n^2) / (2 rho), without the velocities.
  if constexpr (!FAST) {
    r.p_l = (gamma - T(1.0)) * (ql[3] - half_rho_speed2<T, FAST>(r.ql0, ql[1], ql[2], r.u_l, r.v_l));
    r.p_r = (gamma - T(1.0)) * (qr[3] - half_rho_speed2<T, FAST>(r.qr0, qr[1], qr[2], r.u_r, r.v_r));
  } else {
    r.p_l = (gamma - T(1.0)) * (ql[3] - T(0.5) * ((ql[1] * ql[1] + ql[2] * ql[2]) * il));
    r.p_r = (gamma - T(1.0)) * (qr[3] - T(0.5) * ((qr[1] * qr[1] + qr[2] * qr[2]) * ir));
  }
  r.p_l = cmax<T, FAST>(r.p_l, T(kEps * S));
  r.p_r = cmax<T, FAST>(r.p_r, T(kEps * S));
  if constexpr (!FAST) {
    const T srl = sqrt(r.ql0), srr = sqrt(r.qr0);
    const T denom_r = srl + srr;
    h_l = (ql[3] + r.p_l) / r.ql0;
    h_r = (qr[3] + r.p_r) / r.qr0;
    u_t = (srl * r.u_l + srr * r.u_r) / denom_r;
    v_t = (srl * r.v_l + srr * r.v_r) / denom_r;
    h_t = (srl * h_l + srr * h_r) / denom_r;
  } else {
    // sqrt(rho) = rho r and sqrt(rho)*h = (E+p) r with r = 1/sqrt(rho) per side.
    const T id = qrcp<T, FAST>(sl + sr);
    u_t = sum_prod_rn<T>(ql[1], rsl, qr[1], rsr) * id;
    v_t = sum_prod_rn<T>(ql[2], rsl, qr[2], rsr) * id;
    h_t = ((ql[3] + r.p_l) * rsl + (qr[3] + r.p_r) * rsr) * id;
  }
  const T tmp = h_t - T(0.5) * (u_t * u_t + v_t * v_t);
  const T a_t = sqrt(cmax<T, FAST>((gamma - T(1.0)) * tmp, T(0.0)));
  const T un_t = Y ? v_t : u_t;
  r.un_l = Y ? r.v_l : r.u_l;
  r.un_r = Y ? r.v_r : r.u_r;
  r.s_l = un_t - a_t;
  r.s_r = un_t + a_t;
  return r;
}

template <class T, bool FAST>
__device__ __forceinline__ T guard_denom(T d) {
  bool small;
  if constexpr (FAST && is_native_f64<T>)
    small = (f64_bits(d) & 0x7fffffffffffffffLL) < __double_as_longlong(kEps);
  else
    small = fabs(d) < T(kEps);
  if (small) d = copysign(T(kEps), d) + T(kEps);
  return d;
}

// riemann.rs:191-349 HLLE.  S = 2: states and fluxes are doubled (riemann_pre),
// the flux is halved on the way out.
template <class T, bool FAST, bool Y, int S = 1>
__device__ __forceinline__ void hlle_flux(const RiemannPre<T, FAST, Y>& r, const T ql[4], const T fl[4],
                                          const T qr[4], const T fr[4], T F[4]) {
  const T denom = guard_denom<T, FAST>(r.s_r - r.s_l);
  if (r.s_l >= T(0.0)) {
#pragma unroll
    for (int k = 0; k < 4; ++k) F[k] = S == 1 ? fl[k] : T(0.5) * fl[k];
  } else if (r.s_r < T(0.0)) {
#pragma unroll
    for (int k = 0; k < 4; ++k) F[k] = S == 1 ? fr[k] : T(0.5) * fr[k];
  } else {
    const T qlv[4] = {r.ql0, ql[1], ql[2], ql[3]};
    const T qrv[4] = {r.qr0, qr[1], qr[2], qr[3]};
    const T srsl = r.s_r * r.s_l;
    if constexpr (!FAST) {
#pragma unroll
      for (int k = 0; k < 4; ++k) F[k] = r.s_r * fl[k] - r.s_l * fr[k] + srsl * (qrv[k] - qlv[k]);
#pragma unroll 1
      for (int k = 0; k < 4; ++k) {  // one division in the code, F rotating past it
        const T f = F[0] / denom;
        F[0] = F[1], F[1] = F[2], F[2] = F[3], F[3] = f;
      }
    } else {
      const T id = qrcp<T, FAST>(S == 1 ? denom : T(S) * denom);
#pragma unroll
      for (int k = 0; k < 4; ++k) F[k] = (r.s_r * fl[k] - r.s_l * fr[k] + srsl * (qrv[k] - qlv[k])) * id;
    }
  }
}

// riemann.rs:6-189 HLLC
template <class T, bool FAST, bool Y>
__device__ __forceinline__ void hllc_flux(const RiemannPre<T, FAST, Y>& r, const T ql[4], const T fl[4],
                                          const T qr[4], const T fr[4], T F[4]) {
  if (r.s_l >= T(0.0)) {
#pragma unroll
    for (int k = 0; k < 4; ++k) F[k] = fl[k];
    return;
  }
  const T denom = guard_denom<T, FAST>(r.ql0 * (r.s_l - r.un_l) - r.qr0 * (r.s_r - r.un_r));
  // FAST: the two momentum terms rounded on their own, so mirror-image states give
  // S* = +0.0 exactly, as the reference's arithmetic does
  const T s_star = FAST ? qdiv<T, FAST>((r.p_r - r.p_l) + sum_prod_rn<T>(r.ql0 * r.un_l, r.s_l - r.un_l,
                                                                           -(r.qr0 * r.un_r), r.s_r - r.un_r),
                                        denom)
                        : qdiv<T, FAST>(r.p_r - r.p_l + r.ql0 * r.un_l * (r.s_l - r.un_l) -
                                            r.qr0 * r.un_r * (r.s_r - r.un_r),
                                        denom);
  if (r.s_l < T(0.0) && s_star >= T(0.0)) {
    // left star state
    const T m_l = r.ql0 * (r.s_l - r.un_l);
    const T coeff = qdiv<T, FAST>(m_l, r.s_l - s_star);
    const T e_spec = qdiv<T, FAST>(ql[3], r.ql0);
    const T e_star = e_spec + (s_star - r.un_l) * (s_star + qdiv<T, FAST>(r.p_l, m_l));
    T qs[4];
    qs[0] = coeff;
    qs[1] = Y ? coeff * r.u_l : coeff * s_star;
    qs[2] = Y ? coeff * s_star : coeff * r.v_l;
    qs[3] = coeff * e_star;
#pragma unroll
    for (int k = 0; k < 4; ++k) F[k] = fl[k] + r.s_l * (qs[k] - ql[k]);
  } else if (s_star < T(0.0) && r.s_r > T(0.0)) {
    const T m_r = r.qr0 * (r.s_r - r.un_r);
    const T coeff = qdiv<T, FAST>(m_r, r.s_r - s_star);
    const T e_spec = qdiv<T, FAST>(qr[3], r.qr0);
    const T e_star = e_spec + (s_star - r.un_r) * (s_star + qdiv<T, FAST>(r.p_r, m_r));
    T qs[4];
    qs[0] = coeff;
    qs[1] = Y ? coeff * r.u_r : coeff * s_star;
    qs[2] = Y ? coeff * s_star : coeff * r.v_r;
    qs[3] = coeff * e_star;
#pragma unroll
    for (int k = 0; k < 4; ++k) F[k] = fr[k] + r.s_r * (qs[k] - qr[k]);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) F[k] = fr[k];
  }
}

// riemann.rs:394-405: blend weight from the normalised pressure gradient.
template <class T, bool FAST>
__device__ __forceinline__ T sensor_weight(T dpdx, T dpdy, T p, T jp_lo, T jp_hi) {
  const T grad = sqrt(T(dpdx * dpdx + dpdy * dpdy));
  const T jp = qdiv<T, FAST>(grad, vmax(p, T(kEps)));
  if (jp <= jp_lo) return T(1.0);
  if (jp >= jp_hi) return T(0.0);
  return T(1.0) - qdiv<T, FAST>(jp - jp_lo, jp_hi - jp_lo);
}

}  // inline namespace WENO_TU_NS
}  // namespace weno
