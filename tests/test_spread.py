"""Lanes that a launch gives paths to (csrc/spread.h), compiled for the host:
with room for `room' paths in flight, at most that many lanes run, and no
fewer than the paths there are; no two warps of a launch differ by more than
one lane.  No GPU needed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <algorithm>
#include <cstdio>
#include "spread.h"

int main()
{
  const uint64_t warps[] = {1, 3, 592, 1184, 2368}, room[] = {1, 31, 37, 592, 1500, 2000, 3000, 18944, 37888, 75776, 151552},
                 left[] = {0, 1, 100, 1183, 1184, 1185, 3000, 40000, 2097152, 1ull << 40};
  int bad = 0;
  for(uint64_t w : warps) for(uint64_t r : room) for(uint64_t l : left) {
    uint64_t sum = 0, least = 32, most = 0, mixed = 0;
    for(uint64_t i = 0; i < w; ++i) {
      const uint64_t n = hg::warp_lanes(i, w, r, l);
      sum += n;
      least = std::min(least, n);
      most = std::max(most, n);
      mixed += hg::warp_lanes(i, w, r, i % 2 ? l : l / 2); /* another warp's view of the queue */
    }
    if(sum > r || sum < std::min(std::min(l, r), 32 * w) || most - least > 1 || mixed > r) {
      std::printf("warps %llu room %llu left %llu: %llu lanes, %llu to %llu a warp\n", (unsigned long long)w,
                  (unsigned long long)r, (unsigned long long)l, (unsigned long long)sum, (unsigned long long)least,
                  (unsigned long long)most);
      ++bad;
    }
  }
  return bad != 0;
}
"""


def test_lanes_fill_the_room(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "spread.cpp").write_text(SRC)
    exe = tmp_path / "spread"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I",
                    os.path.join(ROOT, "htrdr_kmin_b200", "csrc"), str(tmp_path / "spread.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout[-2000:]
