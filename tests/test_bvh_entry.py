"""A stacked node of a mesh traversal (csrc/bvh_entry.h), compiled for the host:
any node or triangle index of 32 bits and any leaf's triangle count come back,
the entry distance within a millionth part.  No GPU needed."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include "bvh_entry.h"

int main()
{
  const uint32_t first[] = {0, 1, (1u << 29) - 1, 1u << 29, (1u << 29) + 5, 3000000001u, 0xFFFFFFFFu};
  const float enter[] = {-1e-3f, 0.f, 1e-30f, 0.37f, 1.f, 1234.5f, 3e8f, 1e9f, INFINITY};
  for(uint32_t f : first) for(uint32_t c = 0; c <= 4; ++c) for(float t : enter) {
    uint32_t bits;
    std::memcpy(&bits, &t, 4);
    const hg::BvhEntry e = hg::bvh_entry(f, c, bits);
    const uint32_t back = hg::bvh_enter_bits(e);
    float u;
    std::memcpy(&u, &back, 4);
    const bool near = std::isinf(t) ? u == t : std::fabs(u - t) <= 1e-6f * std::fabs(t) + 1e-37f;
    if(e.first != f || hg::bvh_count(e) != c || !near) {
      std::printf("%u %u %g: %u %u %g\n", f, c, t, e.first, hg::bvh_count(e), u);
      return 1;
    }
  }
  return 0;
}
"""


def test_entry_keeps_what_it_is_given(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no C++ compiler")
    (tmp_path / "entry.cpp").write_text(SRC)
    exe = tmp_path / "entry"
    subprocess.run(["g++", "-std=c++17", "-Wall", "-Wextra", "-Werror", "-I",
                    os.path.join(ROOT, "htrdr_kmin_b200", "csrc"), str(tmp_path / "entry.cpp"), "-o", str(exe)],
                   check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
