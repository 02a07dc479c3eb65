"""Face workspace addresses of the staged batch (csrc/solve_desc.h, the code the kernels use), compiled
for the host: every plane of every face array lies inside the solve's block and where 64-bit arithmetic
puts it, for solves whose planes pass 2^31 elements (15,500^2 with the sensor blend in FP64: 100 GB).
"""

import os
import re
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "weno-cfd-solver_gb300", "csrc")

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include "%s"
using namespace weno;
int main(int, char** av) {
  SolveDesc d{};
  const int lq = atoi(av[3]), nf = atoi(av[4]);
  d.nx = atoi(av[1]);
  d.ny = atoi(av[2]);
  d.ld = (d.ny + lq - 1) / lq * lq;
  printf("%%lld\n", staged_layout(d, lq, nf));
  // address of the last value of plane k as the kernels form it, in elements
  auto at = [](int k, auto stride, auto e) { return (long long)(&plane_value((char*)0 + 1, k, stride, e) - ((char*)0 + 1)); };
  for (int k = 0; k < 8; ++k) {
    printf("p1x %%d %%lld %%lld\n", k, at(k, d.s_p1x, p1x_elem(d, 0, 0)), at(k, d.s_p1x, p1x_elem(d, d.nx, d.ny + 3)));
    printf("p1y %%d %%lld %%lld\n", k, at(k, d.s_p1y, p1y_elem(d, 0, 0)), at(k, d.s_p1y, p1y_elem(d, d.nx + 3, d.ny)));
  }
  for (int k = 0; k < nf; ++k) {
    printf("fx %%d %%lld %%lld\n", k, at(k, d.s_fx, fx_elem(d, 0, 0)), at(k, d.s_fx, fx_elem(d, d.nx, d.ny - 1)));
    printf("fy %%d %%lld %%lld\n", k, at(k, d.s_fy, fy_elem(d, 0, 0)), at(k, d.s_fy, fy_elem(d, d.nx - 1, d.ny)));
  }
}
"""


@pytest.fixture(scope="module")
def layout(tmp_path_factory):
    d = tmp_path_factory.mktemp("layout")
    (d / "layout.cpp").write_text(SOURCE % os.path.join(CSRC, "solve_desc.h"))
    subprocess.run(["g++", "-O1", "-std=c++17", str(d / "layout.cpp"), "-o", str(d / "layout")], check=True)
    return str(d / "layout")


@pytest.mark.parametrize("nx,ny,lq,nf", [(3, 3, 2, 4), (7, 5, 4, 9), (64, 1023, 2, 9), (15500, 15500, 2, 9),
                                         (15501, 15451, 4, 9), (24001, 24000, 2, 4), (26800, 26751, 2, 4),
                                         (3, 20000000, 2, 9), (46000, 46001, 4, 4)])
def test_every_plane_in_its_place(layout, nx, ny, lq, nf):
    out = subprocess.run([layout, str(nx), str(ny), str(lq), str(nf)], capture_output=True, text=True, check=True)
    lines = out.stdout.split("\n")
    total = int(lines[0])
    up = lambda x, q: -(-x // q) * q  # noqa: E731
    ld, lx, ly = up(ny, lq), up(ny + 4, lq), up(ny + 1, lq)
    arrays, pos = {}, 0  # name -> (offset, plane stride, last element of a plane)
    for name, planes, rows, pitch, last_col in (("p1x", 8, nx + 1, lx, ny + 3), ("p1y", 8, nx + 4, ly, ny),
                                                ("fx", nf, nx + 1, ld, ny - 1), ("fy", nf, nx, ly, ny)):
        stride = up(rows * pitch, 64)
        arrays[name] = (pos, stride, (rows - 1) * pitch + last_col)
        pos += planes * stride
    assert total == pos
    seen = 0
    for line in filter(None, lines[1:]):
        name, k, first, last = line.split()
        off, stride, end = arrays[name]
        assert int(first) == off + int(k) * stride
        assert int(last) == off + int(k) * stride + end < total
        seen += 1
    assert seen == 16 + 2 * nf


def test_kernels_keep_64_bit_strides():
    """No workspace stride is narrowed on its way into the staged kernels' indices."""
    text = open(os.path.join(CSRC, "batch_kernels.cuh")).read()
    staged = text[text.index("k_staged_pass1"):]
    assert not re.search(r"\(int\)\s*(ks\b|d\.s_|\(x \? d\.s_)", staged)
    assert not re.search(r"\bfi \* d\.l", staged)
