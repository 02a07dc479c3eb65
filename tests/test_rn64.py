"""The integer FP64 quotient and square root of the exact kernels (csrc/rn64.cuh), compiled for the
host and compared bit for bit with the IEEE operations: ordinary significands, all-ones and
near-half-way ones, zeros, subnormal operands and results, infinities and NaN, with the hardware
seed replaced by one that is up to 4 units (reciprocal; 2 for the square root) in the last place off.
"""

import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
HEADER = os.path.join(ROOT, "weno-cfd-solver_gb300", "csrc", "rn64.cuh")

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include "%s"
namespace R = weno::rn64;
static uint64_t bits(double x) { uint64_t b; memcpy(&b, &x, 8); return b; }
static double dbl(uint64_t b) { double x; memcpy(&x, &b, 8); return x; }
static float off(float y, int k) { uint32_t u; memcpy(&u, &y, 4); u += k; memcpy(&y, &u, 4); return y; }
static bool same(uint64_t r, double w) { return r == bits(w) || (dbl(r) != dbl(r) && w != w); }
int main(int, char** av) {
  const int kind = atoi(av[1]);
  const uint64_t M = 0xfffffffffffffull, S = 0x8000000000000000ull;
  std::mt19937_64 g(7 + kind);
  auto with_exp = [&](uint64_t x, int e) { return (x & (S | M)) | ((uint64_t)e << 52); };
  for (long i = 0; i < 400000; ++i) {
    uint64_t a = g(), b = g();
    if (kind < 4) a = with_exp(a, 523 + g() %% 1000), b = with_exp(b, 523 + g() %% 1000);
    if (kind == 1) b |= (g() & 1) ? M : 0xffffffff00000ull, a |= (g() & 1) ? M : 0;
    if (kind == 2) a = (a & ~M) | ((b + g() %% 9 - 4) & M);
    if (kind == 3) {  // a within half a unit of b times a 53-bit number
      const double q = dbl(with_exp(a, 1023) & ~S), d = dbl(with_exp(b, 1023) & ~S);
      a = bits(q * d), b = bits(d);
    }
    if (kind == 4) a = (a & (S | M)) >> (g() %% 53), b = (g() & 1) ? b : (b & M) >> (g() %% 53);
    if (kind == 5) a = with_exp(a, 1 + g() %% 60), b = with_exp(b, 1010 + g() %% 60);
    if (kind == 6) a = with_exp(a, 1 + g() %% 60), b = with_exp(b & S, 1010 + g() %% 60);  // ties
    if (kind == 7) {
      const uint64_t sp[] = {0, S, 0x7ff0000000000000ull, 0xfff0000000000000ull, 0x7ff8000000000000ull, 1, M + 1, ~S >> 1};
      if (g() & 1) a = sp[g() %% 8];
      if (g() & 1) b = sp[g() %% 8];
    }
    const int k = (int)(g() %% 9) - 4;
    const uint64_t r = R::div(a, b, [&](float x) { return off(1.0f / x, k); });
    if (!same(r, dbl(a) / dbl(b))) return printf("div %%a %%a -> %%a\n", dbl(a), dbl(b), dbl(r)), 1;
    uint64_t x = (i & 1) ? a : a & ~S;
    if (kind == 3) x = bits(dbl(with_exp(a, 1023) & ~S) * dbl(with_exp(a, 1023) & ~S));
    const uint64_t q = R::sqrt(x, [&](float m) { return off(1.0f / sqrtf(m), k / 2); });
    if (!same(q, std::sqrt(dbl(x)))) return printf("sqrt %%a -> %%a\n", dbl(x), dbl(q)), 1;
  }
  return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("rn64")
    src, exe = d / "rn64.cpp", d / "rn64"
    src.write_text(SOURCE % HEADER)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", str(src), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("kind", range(8))
def test_matches_ieee(harness, kind):
    r = subprocess.run([harness, str(kind)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
