"""The batch's strip counts (csrc/fd_batch_plan.h), compiled with the host C++
compiler: strips never exceed the caller's height nor fall below the shortest,
members that are left out stay so, and the greedy schedule never ends later
than with strips as tall as allowed."""
import os
import random
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include "fd_batch_plan.h"
int main(int argc, char** argv) {
  const int rows = std::atoi(argv[1]), grid = std::atoi(argv[2]);
  fd::BatchShape s;
  std::vector<int> base;
  for (int i = 3; i + 1 < argc; i += 2) {
    s.height.push_back(std::atoi(argv[i]));
    s.bands.push_back(std::atoi(argv[i + 1]));
    base.push_back((s.height.back() + rows - 1) / rows);
  }
  const std::vector<int> p = fd::plan_strips(s, rows, grid);
  std::printf("%lld %lld", fd::batch_makespan(s, base, grid), fd::batch_makespan(s, p, grid));
  for (size_t i = 0; i < p.size(); ++i) std::printf(" %d", fd::strip_rows(s.height[i], p[i]));
  return 0;
}
"""


@pytest.fixture(scope="module")
def plan(tmp_path_factory):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("plan")
    (d / "p.cpp").write_text(DRIVER)
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(REPO, "fingering_dynamics_gb300", "csrc"),
                    str(d / "p.cpp"), "-o", str(d / "p")], check=True)

    def run(rows, grid, members):
        args = [str(v) for m in members for v in m]
        out = subprocess.run([str(d / "p"), str(rows), str(grid), *args], check=True, capture_output=True, text=True)
        v = [int(x) for x in out.stdout.split()]
        return v[0], v[1], v[2:]
    return run


def test_small_batches_fill_the_grid(plan):
    before, after, rows = plan(32, 760, [(256, 4)] * 8)  # 256 tiles of 32 rows on 760 CTAs
    assert before == 36 and after <= 16 and max(rows) <= 12


def test_one_row_lattices_and_left_out_members(plan):
    assert plan(32, 760, [(3, 1)])[2] == [3]
    assert plan(1, 4, [(5, 1)])[2] == [1]
    before, after, rows = plan(32, 10, [(64, 0), (64, 2)])
    assert after <= before and rows[0] == 32  # no bands: not cut further


@pytest.mark.parametrize("seed", range(12))
def test_random_batches(plan, seed):
    rng = random.Random(seed)
    members = [(rng.choice((3, 37, 128, 256, 512)), rng.choice((0, 1, 2, 4, 8, 16))) for _ in range(rng.randint(1, 60))]
    rows, grid = rng.choice((1, 8, 16, 32, 64, 1000)), rng.choice((1, 100, 608, 760, 1064))
    before, after, got = plan(rows, grid, members)
    assert after <= before
    for (h, _), r in zip(members, got):
        assert 1 <= r <= min(rows, h) and (r >= min(4, rows, h) or r == -(-h // -(-h // rows)))
