"""The streaming GEMMs' ranges (csrc/stream_plan.cuh, compiled for the host): a range longer than the equal one is whole slabs or
divides one, and is taken only where it costs no more than a cut."""
import os
import subprocess

from conftest import ROOT

MAIN = r"""
#include <cstdio>
#include "stream_plan.cuh"
int main() {
  const int ctas[] = {7, 148, 160};
  for (int c : ctas)
    for (int groups = 1; groups <= 32; ++groups)
      for (int units = 0; units <= 40 * groups * (c == 7 ? 1 : 16); units += groups)
        printf("%d %d %d %d\n", units, groups, c, b200moe::stream_range(units, groups, c));
  printf("%d\n", b200moe::kCutCost);
}
"""


def test_longer_ranges_cut_no_slab_unevenly(tmp_path):
    src, exe = tmp_path / "plan.cpp", tmp_path / "plan"
    src.write_text(MAIN)
    subprocess.run(["g++", "-O1", "-std=c++17", "-I", os.path.join(ROOT, "fused_moe_b200", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    lines = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split("\n")
    cost = int(lines[-2])
    seen = set()
    for line in lines[:-2]:
        units, groups, ctas, got = map(int, line.split())
        per = -(-units // ctas)
        even = next((s for s in range(per, per + groups + 1) if s and (s % groups == 0 or groups % s == 0)), 0) if per else 0
        assert got == (even if even - per <= cost else per), (units, groups, ctas, got)
        assert got * ctas >= units
        seen.add((groups, per))
    assert {(28, 5), (28, 8), (28, 9), (5, 2), (28, 15), (32, 17)} <= seen
