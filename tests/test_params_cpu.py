"""Kernel parameters that the marches index with unclamped: every position inside the
volume has to give an entry of the cell tables, for the field's cells and the map's."""
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
CUDA = "/usr/local/cuda/include"
SRC = r"""
#include <cstdio>
#include <cstdlib>
#include "beams_params.h"
using namespace beams;
// floor of the product that the marches take toward zero, or -1 when it is none
static double entry(double x, float f) {
  const double p = x * (double)f;  // exact: two floats
  return p >= 0.0 && p < 8388608.0 ? std::floor(p) : -1.0;
}
int main(int, char** a) {
  const float org = strtof(a[1], 0), h = strtof(a[2], 0);
  const int n = atoi(a[3]), M = atoi(a[4]);
  ExactGeo g;
  std::memset(&g, 0, sizeof(g));
  for (int d = 0; d < 3; ++d) {
    g.n[d] = n;
    g.org[d] = org;
    g.h[d] = h;
    g.invh[d] = 1.f / h;
    g.minp[d] = org + h * 0.f;
    g.maxp[d] = org + h * (float)(n - 1);
    g.bmin[d] = g.minp[d];
    g.bmax[d] = g.maxp[d];
    g.pd[d] = M + 1;
    g.morig[d] = g.minp[d];
    g.msp[d] = (float)(g.bmax[d] - g.bmin[d]) / (float)M;
    g.minv[d] = 1.f / g.msp[d];
  }
  geo_loop_constants(g, true);
  int bad = 0;
  for (int i = 0; i <= 4096; ++i) {
    float p = i == 4096 ? g.maxp[0] : g.minp[0] + (float)(i / 4096.0 * ((double)g.maxp[0] - g.minp[0]));
    if (!(p >= g.minp[0] && p <= g.maxp[0])) continue;
    const float x = p - g.org[0], y = p - g.morig[0];
    const double c = entry(x, g.seed[0]), m = entry(y, g.minv[0]);
    bad += !(c >= 0 && c <= n - 1) + !(m >= 0 && m <= M);
  }
  std::printf("%d\n", bad);
  return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("params")
    (d / "t.cpp").write_text(SRC)
    p = subprocess.run(["g++", "-std=c++17", "-O1", "-ffp-contract=off", "-I", CUDA, "-I",
                        str(ROOT / "pilot_b200" / "csrc"), str(d / "t.cpp"), "-o", str(d / "t")],
                       capture_output=True, text=True)
    assert p.returncode == 0, p.stderr
    return d / "t"


@pytest.mark.parametrize("org,h,n,m", [(0, 1, 129, 128), (-3.7, 0.013, 200, 2047), (5e5, 1, 200, 100), (3e7, 1, 160, 77),
                                       (3.3e7, 0.5, 64, 300), (1e6, 1e-3, 10, 16), (0, 1e-38, 2, 2047),
                                       (0, 1e-38, 2, 1), (0, 2.2e-39, 3, 128), (0, 1e-40, 64, 128), (0, 1e-45, 2, 2),
                                       (1e18, 1e15, 100, 100), (0, 1e17, 100, 2047)])
def test_positions_inside_index_the_tables(program, org, h, n, m):
    p = subprocess.run([str(program), repr(org), repr(h), str(n), str(m)], capture_output=True, text=True)
    assert p.returncode == 0 and p.stdout.strip() == "0", p.stdout
