"""The fixed-point reciprocal (hg_rcp.cuh) against the division, on the CPU: every
bit, over random and boundary significands and exponents, with the
single-precision seed off by up to two units."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r'''
#include <cstdio>
#include <random>
#include "hg_rcp.cuh"
using namespace hg;
static long bad = 0, count = 0;
static void check(uint64_t b) {
  if (!rcp_in_range(b)) return;
  const uint64_t want = rcp_bits(1.0 / rcp_double(b));
  const uint32_t seed = rcp_seed(0x3f800000u | ((uint32_t)(b >> 29) & 0x7fffffu));
  for (int d = -2; d <= 2; ++d) {
    if (seed + d > 0x3f800000u) continue;
    ++count;
    if (rcp_bits(rcp_from_seed(b, seed + d)) != want) ++bad;
  }
}
int main() {
  std::mt19937_64 g(7);
  for (int i = 0; i < 1000000; ++i) check(g());
  for (int i = 0; i < 300000; ++i) {
    const uint64_t e = (uint64_t)(1 + g() % 2043) << 52;
    check(e | (g() & 0xffff));
    check(e | (0xfffffffffffffull - (g() & 0xffff)));
    check(e | ((g() & 0x7fffff) << 29));
    check(e | ((g() & 0x7fffff) << 29) | 0x1fffffff);
  }
  for (uint64_t e = 1; e <= 2043; ++e)
    for (uint64_t m : {0ull, 1ull, 0x8000000000000ull, 0xfffffffffffffull}) {
      check((e << 52) | m);
      check((1ull << 63) | (e << 52) | m);
    }
  std::printf("%ld %ld\n", count, bad);
  return 0;
}
'''


def test_fixed_point_reciprocal_is_the_division(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    src = tmp_path / "rcp.cpp"
    src.write_text(PROGRAM)
    exe = tmp_path / "rcp"
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "hams-mrel_gb300", "csrc"), str(src), "-o", str(exe)],
                   check=True)
    count, bad = map(int, subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split())
    assert count > 5_000_000 and bad == 0
