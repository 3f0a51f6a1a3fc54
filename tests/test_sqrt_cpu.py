"""The square roots and reciprocal square roots from a single-precision seed
(hg_rcp.cuh) against extended precision, on the CPU, the seed off by up to two
units either way as the device's approximation may be (its relative error is
below 2^-22)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

PROGRAM = r'''
#include <cmath>
#include <cstdio>
#include <random>
#include <string.h>
#include "hg_rcp.cuh"
using namespace hg;
typedef long double ld;
static double ulps(double got, ld want) {
  int e;
  std::frexp((double)want, &e);
  return (double)(std::fabs((ld)got - want) / std::ldexp((ld)1, e - 53));
}
int main() {
  std::mt19937_64 g(11);
  double worst[3] = {0, 0, 0};
  long inexact = 0, count = 0, fallback = 0;
  for (int i = 0; i < 3000000; ++i) {
    double x;
    const int kind = i % 4;
    if (kind == 0) x = std::ldexp(1.0 + (g() >> 12) * 0x1p-52, (int)(g() % 240) - 120);
    else if (kind == 1) x = std::ldexp((double)(g() >> 40), (int)(g() % 100) - 60);
    else if (kind == 2) { const double r = (double)(g() >> 38) * std::ldexp(1.0, (int)(g() % 60) - 40); x = r * r; }  // exact squares
    else x = std::ldexp(1.0 + (double)(g() % 64) * 0x1p-52 * ((g() & 1) ? 1 : -1), (int)(g() % 200) - 100);
    if (!(x > 0)) continue;
    if (!rsqrt_in_range(x)) { ++fallback; continue; }
    const ld s = sqrtl((ld)x);
    const float seed = rsqrt_seed((float)x);
    for (int d = -2; d <= 2; ++d) {
      uint32_t b;
      memcpy(&b, &seed, 4);
      b += d;
      float f;
      memcpy(&f, &b, 4);
      const double y = rsqrt_from_seed(x, f), q = sqrt_from_seed(x, f), r = root_of(x, y);
      ++count;
      worst[0] = std::fmax(worst[0], ulps(y, 1 / s));
      worst[1] = std::fmax(worst[1], ulps(q, s));
      worst[2] = std::fmax(worst[2], ulps(r, s));
      if (kind == 2 && (q != (double)s || r != (double)s)) ++inexact;
    }
  }
  // outside the range the library's root
  const double ends[] = {0.0, 5e-324, 1e-300, 0x1p-123, 0x1p123, 1e300, INFINITY};
  int same = 1;
  for (double x : ends) same = same && !rsqrt_in_range(x) && sqrt_near(x) == std::sqrt(x) && rsqrt_near(x) == 1.0 / std::sqrt(x);
  std::printf("%.6f %.6f %.6f %ld %ld %d\n", worst[0], worst[1], worst[2], inexact, count, same);
  return 0;
}
'''


def test_roots_from_a_seed(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    src, exe = tmp_path / "sqrt.cpp", tmp_path / "sqrt"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-I", os.path.join(ROOT, "hams-mrel_gb300", "csrc"),
                    str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout.split()
    rs, sq, root = map(float, out[:3])
    # the reciprocal: the step's last rounding, and half the rounding of x y in e: at most 1 unit together, with the
    # cubed seed error 5/16 (3 2^-23)^3 2^53 below 2^-11; the roots: the last rounding alone, the residual of a value
    # right to 2^-43 (or one unit) leaving less than 2^-30
    assert rs <= 1.01 and sq <= 0.5 + 2.0 ** -20 and root <= 0.5 + 2.0 ** -20
    assert int(out[3]) == 0 and int(out[4]) > 10_000_000 and out[5] == "1"
