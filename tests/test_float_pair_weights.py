"""The float-pair WENO weights of the FAST FP64 kernels (csrc/ffw.cuh), compiled for the host and
compared with extended precision.

Tolerance, from the error bounds of float-pair arithmetic (u = 2^-24: conversion 0.5 u^2, sum 3 u^2,
product 5 u^2, reciprocal 4 u^2): an indicator is within 16 u^2, its inverse square within 45 u^2, a
weight, whose normalisation adds the error of the sum of the three and of one reciprocal and product,
within 110 u^2 < 2^-41 of itself.  The largest weight is formed as the constant less the other two and
inherits their absolute errors.  The conversion back to double is exact for what is representable.
"""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "weno-cfd-solver_gb300", "csrc", "ffw.cuh")

SOURCE = r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#define __device__
#define __host__
#define __forceinline__ inline
static inline float __fadd_rn(float a, float b) { return a + b; }
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
template <class A, class B> static A cast(B b) { A a; static_assert(sizeof a == sizeof b, ""); memcpy(&a, &b, sizeof a); return a; }
static inline int __double2hiint(double d) { return (int)(cast<uint64_t>(d) >> 32); }
static inline int __double2loint(double d) { return (int)cast<uint64_t>(d); }
static inline double __hiloint2double(int h, int l) { return cast<double>(((uint64_t)(uint32_t)h << 32) | (uint32_t)l); }
static inline float __uint_as_float(uint32_t u) { return cast<float>(u); }
static inline uint32_t __float_as_uint(float f) { return cast<uint32_t>(f); }
static inline double __longlong_as_double(long long u) { return cast<double>(u); }
static inline uint32_t __float2uint_rz(float f) { return !(f > 0) ? 0 : f >= 4294967296.f ? 0xffffffffu : (uint32_t)f; }
#include "ffw_host.h"
using namespace weno::ffw;
typedef long double L;
int main(int, char** av) {
  const int kind = atoi(av[1]);
  std::mt19937_64 g(3 + kind);
  std::uniform_real_distribution<double> U(-1, 1);
  const L tol = ldexpl(1, -41);
  for (long i = 0; i < 200000; ++i) {
    double d[4], eps = kind == 4 ? 0x1p-57 : kind == 5 ? 0x1p39 : 1e-12;
    for (double& x : d) x = U(g);
    if (kind == 1) for (double& x : d) x = ldexp(x, -(int)(g() %% 60));
    if (kind == 2) for (double& x : d) x = (g() & 1) ? 0.0 : x;
    if (kind == 3) for (double& x : d) x = ldexp(x, 27);
    if (kind == 5) for (double& x : d) x = ldexp(x, 20);
    if (kind == 6) { d[0] *= 1e-9, d[1] *= 1e-9; }       // a jump beyond the cell
    if (kind == 7) { d[1] = d[0] * (1 + 1e-7 * U(g)), d[2] = d[1], d[3] = d[2] * (1 - 1e-7); }  // almost linear
    if (kind == 8) for (double& x : d) x = ldexp(x, 22);  // the largest covered
    uint32_t dmax = 0;
    for (double x : d) dmax = magnitude(x) > dmax ? magnitude(x) : dmax;
    if (!covers(dmax, eps)) continue;  // callers take the FP64 weights
    ff f[4], w = eps75(eps);
    for (int k = 0; k < 4; ++k) f[k] = from_double(d[k]);
    const L x[4] = {d[0], d[1], d[2], d[3]}, E = eps;
    const L b0 = 13 * (x[3] - x[2]) * (x[3] - x[2]) / 12 + (x[3] - 3 * x[2]) * (x[3] - 3 * x[2]) / 4,
            b1 = 13 * (x[2] - x[1]) * (x[2] - x[1]) / 12 + (x[2] + x[1]) * (x[2] + x[1]) / 4,
            b2 = 13 * (x[1] - x[0]) * (x[1] - x[0]) / 12 + (x[0] - 3 * x[1]) * (x[0] - 3 * x[1]) / 4;
    const ff q0 = side(f[2], f[3], w), q1 = centre(f[1], f[2], w), q2 = side(f[1], f[0], w);
    double c[3];
    auto check = [&](const L* lin, L k) {
      const L a[3] = {lin[0] / ((E + b0) * (E + b0)), lin[1] / ((E + b1) * (E + b1)), lin[2] / ((E + b2) * (E + b2))};
      const L s = a[0] + a[1] + a[2];
      for (int j = 0; j < 3; ++j) {
        const L want = k * a[j] / s, big = want > k / 3 - tol ? k : want;
        if (fabsl(c[j] - want) > tol * big + 0x1p-75L) {
          printf("weight %%d of (%%a %%a %%a %%a): %%a, off by %%Lg\n", j, d[0], d[1], d[2], d[3], c[j], c[j] - want);
          exit(1);
        }
      }
    };
    face_weights(q0, q1, q2, c[0], c[1], c[2]);
    const L face[3] = {0.3L, 0.6L, 0.1L}, gp[3] = {0.1928406937L, 0.6111111111L, 0.1960481952L};
    check(face, 1 / 6.0L);
    gauss_weights(q0, q1, q2, constant(0.1928406937 / 0.6111111111), constant(0.1960481952 / 0.6111111111),
                  constant(0.1443375673), c[0], c[1], c[2]);
    check(gp, 0.1443375673L);
    // the mirror image has the mirrored weights, bit for bit
    double m[3], n[3];
    face_weights(q0, q1, q2, m[0], m[1], m[2]);
    const ff g0 = neg(f[3]), g1 = neg(f[2]), g2 = neg(f[1]), g3 = neg(f[0]);
    face_weights(side(g1, g0, w), centre(g1, g2, w), side(g2, g3, w), n[0], n[1], n[2]);
    if (m[0] != n[0] || m[1] != n[1] || m[2] != n[2]) return printf("mirror image differs\n"), 1;
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("ffw")
    text = open(HEADER).read().replace("#include <cuda_runtime.h>", "")
    seed = 'asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a.h));'
    assert seed in text
    (d / "ffw_host.h").write_text(text.replace(seed, "y = 1.0f / a.h; y = __uint_as_float(__float_as_uint(y) + 1u);"))
    (d / "ffw.cpp").write_text(SOURCE.replace("%%", "%"))
    exe = d / "ffw"
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", str(d / "ffw.cpp"), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("kind", range(9))
def test_weights_against_extended_precision(harness, kind):
    r = subprocess.run([harness, str(kind)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
