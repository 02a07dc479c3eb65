"""The float-pair WENO weights (csrc/ffw.cuh) at the ends of the epsilons and differences they cover, compiled
for the host: where a smooth stencil's indicators are small beside the epsilon, the sum of the weights before
normalisation is of the order of 1 / epsilon^2, and the low part of its reciprocal has to stay a normal float.

Bound: every weight within 2^-44 of the sum of the three (the largest error seen over these data is 2^-45.0).
"""

import subprocess

import pytest

from test_float_pair_weights import HEADER, SOURCE

MAIN = r"""
int main(int, char** av) {
  const int le = atoi(av[1]);
  std::mt19937_64 g(3 + le);
  std::uniform_real_distribution<double> U(-1, 1);
  const L tol = ldexpl(1, -44);
  long n = 0;
  for (long i = 0; i < 200000; ++i) {
    double d[4], eps = ldexp(1 + 0.99 * fabs(U(g)), le);
    // differences well below, around and far above the root of the epsilon, and up to 2^22
    const int s = (int)(g() % 5), sh = s == 0 ? le / 2 - 6 : s == 1 ? le / 2 : s == 2 ? -(int)(g() % 40) : s == 3 ? 0 : 22;
    for (double& x : d) x = ldexp(U(g), sh - (s == 2 ? (int)(g() % 20) : 0));
    uint32_t dmax = 0;
    for (double x : d) dmax = magnitude(x) > dmax ? magnitude(x) : dmax;
    if (!covers(dmax, eps)) continue;
    if (!covers_pair(0x1p21f, (float)eps)) return printf("the two rules differ at %a\n", eps), 1;
    ++n;
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
      const L s3 = a[0] + a[1] + a[2];
      for (int j = 0; j < 3; ++j)
        if (!(fabsl(c[j] - k * a[j] / s3) <= tol * k)) {
          printf("eps %a, weight %d of (%a %a %a %a): 2^%Lf of the sum off\n", eps, j, d[0], d[1], d[2], d[3],
                 log2l(fabsl(c[j] / k - a[j] / s3)));
          exit(1);
        }
    };
    const L face[3] = {0.3L, 0.6L, 0.1L}, gp[3] = {0.1928406937L, 0.6111111111L, 0.1960481952L};
    face_weights(q0, q1, q2, c[0], c[1], c[2]);
    check(face, 1 / 6.0L);
    gauss_weights(q0, q1, q2, constant(0.1928406937 / 0.6111111111), constant(0.1960481952 / 0.6111111111),
                  constant(0.1443375673), c[0], c[1], c[2]);
    check(gp, 0.1443375673L);
  }
  printf("%ld\n", n);
  return 0;
}
"""


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    d = tmp_path_factory.mktemp("ffw_eps")
    text = open(HEADER).read().replace("#include <cuda_runtime.h>", "")
    seed = 'asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(a.h));'
    assert seed in text
    (d / "ffw_host.h").write_text(text.replace(seed, "y = 1.0f / a.h; y = __uint_as_float(__float_as_uint(y) + 1u);"))
    (d / "ffw.cpp").write_text(SOURCE[:SOURCE.index("int main(")].replace("%%", "%") + MAIN)
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", str(d / "ffw.cpp"), "-o", str(d / "ffw")],
                   check=True)
    return str(d / "ffw")


@pytest.mark.parametrize("log2_eps", [-59, -58, -56, -52, -50, -49, -48, -47, -44, -40, -20, 0, 20, 38, 39, 40])
def test_weights_over_the_covered_epsilons(harness, log2_eps):
    r = subprocess.run([harness, str(log2_eps)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
    if -48 <= log2_eps < 40:
        assert int(r.stdout) > 100000  # covered, not left to the FP64 weights
