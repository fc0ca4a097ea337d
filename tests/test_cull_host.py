"""The distance test of the adjoint's Gaussian pair sweep (lddmm_b200/csrc/cull.h), compiled
here: for random tiles and blocks whose momenta differ by many powers of ten from point to
point, and for every row of the tile by itself, all blocks that the test skips together add
no more than it allows.  Zero, infinite and NaN weights and boxes are never skipped wrongly."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

HARNESS = r'''
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "cull.h"
using namespace lddmm;
int main() {
  std::mt19937 rng(7);
  std::uniform_real_distribution<double> U(0.0, 1.0);
  long skipped = 0;
  for (int trial = 0; trial < 200000; ++trial) {
    const int n = 128, nblk = 1 + (int)(U(rng) * 300);
    const float diag2 = (float)std::pow(10.0, -3.0 + 4.0 * U(rng));
    std::vector<double> u(n), r(n);
    const int kind = trial % 4;  // even; log-uniform; one point of u; one point of r
    double UI = 0.0, RI = 0.0;
    for (int i = 0; i < n; ++i) {
      u[i] = std::pow(10.0, kind == 0 ? 0.0 : -8.0 * U(rng)) * (kind == 2 && i ? 1e-7 : 1.0);
      r[i] = std::pow(10.0, kind == 0 ? 0.0 : -8.0 * U(rng)) * (kind == 3 && i ? 1e-7 : 1.0);
      UI += u[i];
      RI += r[i];
    }
    const AdjointCut cut = adjoint_cut(diag2, nblk, (float)UI, (float)RI);
    const double UB = std::pow(10.0, 4.0 - 12.0 * U(rng)), RB = std::pow(10.0, 4.0 - 12.0 * U(rng));
    const double g = 10.0 * U(rng);
    if (!adjoint_skips(cut, (float)(g * g), (float)UB, (float)RB)) continue;
    ++skipped;
    const double K = std::exp2(-g * g), e = std::exp2(-26.0 - diag2) / nblk * 1.001;
    const double d = std::sqrt(diag2) / 4.0;
    if (K * UB > e * UI) return 1;
    for (int i = 0; i < n; ++i)
      for (double m : {u[i] + r[i], u[i], 0.0})  // |m_i| is between | |u| - |r| | and |u| + |r|
        if (K * g * (m * RB + r[i] * UB) > e * d * (m * RI + r[i] * UI)) return 2;
  }
  if (skipped < 20000) return 3;
  const float inf = INFINITY, nan = NAN;
  const AdjointCut c = adjoint_cut(1.0f, 4, 1.0f, 1.0f);
  if (!adjoint_skips(c, 60.0f, 1.0f, 0.0f) || adjoint_skips(c, 60.0f, inf, 1.0f) ||
      adjoint_skips(c, 60.0f, 1.0f, inf) || adjoint_skips(c, nan, 1.0f, 1.0f) ||
      adjoint_skips(c, 0.0f, 0.0f, 0.0f))
    return 4;
  for (float bad : {0.0f, inf, nan})  // the tile's own weight: nothing of weight is skipped
    if (adjoint_skips(adjoint_cut(1.0f, 4, bad, 1.0f), 60.0f, 1.0f, 1.0f) ||
        adjoint_skips(adjoint_cut(1.0f, 4, 1.0f, bad), 60.0f, 1.0f, 1.0f))
      return 5;
  if (adjoint_skips(adjoint_cut(0.0f, 4, 1.0f, 1.0f), 60.0f, 1.0f, 1.0f)) return 6;
  return 0;
}
'''


@pytest.mark.skipif(shutil.which("g++") is None, reason="no host compiler")
def test_adjoint_distance_test_row_by_row(tmp_path):
    src, exe = tmp_path / "cull.cpp", tmp_path / "cull"
    src.write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", os.path.join(ROOT, "lddmm_b200", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    assert subprocess.run([str(exe)]).returncode == 0
