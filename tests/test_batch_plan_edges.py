"""The batch's strip counts (csrc/fd_batch_plan.h) where there is nothing to plan: no CTA,
no member, members without bands."""
import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DRIVER = r"""
#include <cstdio>
#include "fd_batch_plan.h"
int main() {
  const fd::BatchShape none, one{{96}, {2}}, left_out{{96, 33}, {0, 0}};
  for (int grid : {0, -1, 760})
    for (const fd::BatchShape* s : {&none, &one, &left_out}) {
      for (int n : fd::plan_strips(*s, 32, grid)) std::printf("%d ", n);
      std::printf("| ");
    }
  return 0;
}
"""


def test_nothing_to_plan(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    (tmp_path / "p.cpp").write_text(DRIVER)
    exe = str(tmp_path / "p")
    subprocess.run([cxx, "-std=c++17", "-O0", "-I", os.path.join(REPO, "fingering_dynamics_gb300", "csrc"), "-o", exe,
                    str(tmp_path / "p.cpp")], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    groups = [g.split() for g in out.split("|")[:-1]]
    assert groups[:6] == [[], ["3"], ["3", "2"]] * 2  # without a CTA: as tall as allowed
    assert groups[6] == [] and groups[8] == ["3", "2"] and int(groups[7][0]) >= 3
