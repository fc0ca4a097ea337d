"""Host plan of the persistent sweeps' 64-row tiles (plan_sweeps in lddmm_b200/csrc/plan.h) as a
context makes it, for two CTAs on each of 148 SMs: every (tile, j) entry is covered exactly once
and in part order, cuts leave at least 32 entries, and where one CTA per SM is preferred the
plan does not exceed the SMs."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

HARNESS = r'''
#include <cstdio>
#include <cstdlib>
#include <vector>
#include <vector_types.h>
#include <vector_functions.h>
#include "plan.h"
using namespace lddmm;
int main(int argc, char **argv) {
  std::vector<PairDesc> hpd(argc - 1);
  std::vector<int2> units;
  for (int p = 0; p + 1 < argc; ++p) {
    hpd[p].Npad = (std::atoi(argv[p + 1]) + 63) / 64 * 64;
    for (int t = 0; t < hpd[p].Npad / 64; ++t) units.push_back(make_int2(p, t));
  }
  const HostPlan two = plan_sweeps(units, hpd, 296), h = plan_sweeps(units, hpd, 296, 148);
  const int ctas = (int)h.cta_seg.size() - 1;
  if (ctas > 296 || h.cta_seg.back() != (int)h.segs.size()) return 1;
  std::vector<int> end(units.size(), 0), part(units.size(), 0);
  long long share = 0, share2 = 0;
  for (int k = 0; k < ctas; ++k) {
    long long s = 0;
    for (int q = h.cta_seg[k]; q < h.cta_seg[k + 1]; ++q) {
      const int4 g = h.segs[q];
      if (g.y != end[g.x] || g.z <= g.y || g.w != part[g.x]) return 2;
      if (g.z - g.y < kMinSeg && g.z - g.y < hpd[units[g.x].x].Npad) return 3;
      end[g.x] = g.z;
      ++part[g.x];
      s += g.z - g.y + kSegCost;
    }
    share = std::max(share, s);
  }
  for (size_t k = 0; k + 1 < two.cta_seg.size(); ++k) {
    long long s = 0;
    for (int q = two.cta_seg[k]; q < two.cta_seg[k + 1]; ++q)
      s += two.segs[q].z - two.segs[q].y + kSegCost;
    share2 = std::max(share2, s);
  }
  int slots = 0;
  for (size_t u = 0; u < units.size(); ++u) {
    if (end[u] != hpd[units[u].x].Npad || h.unit_parts[u].x != part[u] || part[u] > 11) return 4;
    if (part[u] > 1) {
      if (h.unit_parts[u].y != slots) return 5;
      slots += part[u];
    }
  }
  if (slots != h.slots) return 6;
  // one CTA per SM: chosen for balance, never at the price of more than two shares of the other
  if (ctas <= 148 && (int)two.cta_seg.size() - 1 > 148 && share > 2 * share2) return 7;
  std::printf("%d\n", ctas);
  return 0;
}
'''


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    inc = next((p for p in ("/usr/local/cuda/include",) if os.path.isdir(p)), None)
    if shutil.which("g++") is None or inc is None:
        pytest.skip("no host compiler or CUDA headers")
    d = tmp_path_factory.mktemp("plan")
    (d / "plan.cpp").write_text(HARNESS)
    subprocess.run(["g++", "-O2", "-std=c++17", "-I", inc, "-I",
                    os.path.join(ROOT, "lddmm_b200", "csrc"), str(d / "plan.cpp"), "-o",
                    str(d / "plan")], check=True)
    return str(d / "plan")


@pytest.mark.parametrize("sizes,one_per_sm", [
    ((5,), None), ((64,), None), ((642,), None), ((1200,), True), ((1800,), None),
    ((2562,), None), ((5000,), None), ((9473,), None), ((64, 9001, 513), None),
    (tuple(200 + 5 * k for k in range(130)), None)])
def test_tile_plans(exe, sizes, one_per_sm):
    r = subprocess.run([exe, *map(str, sizes)], capture_output=True, text=True)
    assert r.returncode == 0, r.returncode
    if one_per_sm:
        assert int(r.stdout) <= 148
