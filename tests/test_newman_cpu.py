"""Newman's panel integral in the fused form (newman_pair, hg_green.cuh,
compiled for the host) where it can take a wrong turn: panels so small or so
large that an edge's complex number leaves the product's range and the angles
are added one by one, and points above, beside, in the plane of and in line
with the edges, where the sum of the angles is next to a multiple of 2 pi."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r'''
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include "hg_green.cuh"
using namespace hg;
typedef long double ld;

template <class T> void newman(const double* pr, const double* f, T o[4]) {
  T c[3] = {0, 0, 0};
  for (int a = 0; a < 3; ++a)
    for (int k = 0; k < 3; ++k) c[a] += (T)pr[PR_UI + 3 * a + k] * ((T)f[k] - pr[PR_PO + k]);
  const T x = c[0], y = c[1], z = c[2];
  const int nv = (int)pr[PR_NCN];
  T st = 0, sx = 0, sy = 0, sz = 0;
  for (int e = 0; e < nv; ++e) {
    const int n = (e + 1) % nv;
    const T k1 = pr[PR_KSI + e] - x, e1 = pr[PR_ETA + e] - y, k2 = pr[PR_KSI + n] - x, e2 = pr[PR_ETA + n] - y, l = pr[PR_L + e];
    const T dk = (T)pr[PR_KSI + n] - pr[PR_KSI + e], de = (T)pr[PR_ETA + n] - pr[PR_ETA + e];
    if (nv == 4 && l < (T)1e-8) continue;
    const T r1 = sqrt(k1 * k1 + e1 * e1 + z * z), r2 = sqrt(k2 * k2 + e2 * e2 + z * z);
    const T b1 = de * (k1 * k1 + z * z) - dk * k1 * e1, a1 = r1 * z * dk, b2 = de * (k2 * k2 + z * z) - dk * k2 * e2, a2 = r2 * z * dk;
    if (!(std::abs(z) < (T)1e-6)) sz += atan2(b1 * a2 - b2 * a1, a1 * a2 + b1 * b2);
    const T s = r1 + r2;
    if (std::abs(s - l) < (T)1e-6) continue;
    const T lg = log((s + l) / (s - l));
    sx -= de / l * lg;
    sy += dk / l * lg;
    st -= (de * k1 - dk * e1) / l * lg;
  }
  const T sg = nv == 3 ? 1 : -1;
  o[0] = sg * (st - z * sz);
  for (int k = 0; k < 3; ++k) o[1 + k] = sg * (pr[PR_UI + k] * sx + pr[PR_UJ + k] * sy + pr[PR_UK + k] * sz);
}

int main(int c, char** v) {
  const double size = std::atof(v[1]);
  const int nv = std::atoi(v[2]);
  std::mt19937_64 gen(3);
  auto uni = [&](double a, double b) { return std::uniform_real_distribution<double>(a, b)(gen); };
  double worst[2] = {0, 0}, grad[2] = {0, 0};  // ours, the formula's in double
  for (int k = 0; k < 40000; ++k) {
    // the panel in its own frame, the frame's axes those of space: the point's place relative to the edges is exact
    double pr[PR_SIZE] = {};
    pr[PR_UI] = pr[PR_UJ + 1] = pr[PR_UK + 2] = 1.0;
    pr[PR_NCN] = nv;
    const double sx[4] = {1, -1, -1, 1}, sy[4] = {1, 1, -1, -1};
    for (int e = 0; e < nv; ++e) {
      pr[PR_KSI + e] = size * (sx[e] * uni(0.2, 0.6));
      pr[PR_ETA + e] = size * (sy[e] * uni(0.2, 0.6));
      if (k % 5 == 0) { pr[PR_KSI + e] = size * 0.5 * sx[e]; pr[PR_ETA + e] = size * 0.5 * sy[e]; }  // edges along the axes
    }
    for (int e = 0; e < nv; ++e) {
      const int n = (e + 1) % nv;
      pr[PR_L + e] = std::hypot(pr[PR_KSI + n] - pr[PR_KSI + e], pr[PR_ETA + n] - pr[PR_ETA + e]);
    }
    const int e = k % nv, n = (e + 1) % nv;
    const double low = 2e-6 * std::fmax(1.0, size);  // just out of the plane
    double t = uni(-2, 3), f[3], z = size * std::pow(10.0, uni(-3, 1));
    switch (k % 6) {
      case 0: f[0] = uni(-.1, .1) * size; f[1] = uni(-.1, .1) * size; break;                                       // above the panel
      case 1: f[0] = uni(-3, 3) * size; f[1] = uni(-3, 3) * size; break;                                           // anywhere
      case 2: case 3:                                                                                             // above an edge's line
        f[0] = pr[PR_KSI + e] + t * (pr[PR_KSI + n] - pr[PR_KSI + e]);
        f[1] = pr[PR_ETA + e] + t * (pr[PR_ETA + n] - pr[PR_ETA + e]);
        break;
      case 4: f[0] = pr[PR_KSI + e]; f[1] = pr[PR_ETA + e]; break;                                                 // above a vertex
      default: f[0] = uni(-.2, .2) * size; f[1] = uni(-3, 3) * size;                                               // inside or beside
    }
    f[2] = (k % 12 < 6 ? z : low) * (k & 64 ? 1 : -1);
    if (std::fabs(f[2]) < 1e-6) f[2] = std::copysign(1.5e-6, f[2]);
    if (k % 31 == 0) f[2] = 0.0;                                                                                  // in the plane
    double o[2][4];
    ld x[4];
    newman_pair(pr, f[0], f[1], f[2], o[0][0], o[0][1], o[0][2], o[0][3]);
    newman<double>(pr, f, o[1]);
    newman<ld>(pr, f, x);
    for (int w = 0; w < 2; ++w) {
      worst[w] = std::fmax(worst[w], std::fabs((double)(o[w][0] - x[0])) / std::fmax(size, std::fabs(f[2])));
      for (int q = 1; q < 4; ++q) grad[w] = std::fmax(grad[w], std::fabs((double)(o[w][q] - x[q])));
    }
  }
  std::printf("%.3e %.3e %.3e %.3e\n", worst[0], worst[1], grad[0], grad[1]);
  return 0;
}
'''


@pytest.fixture(scope="module")
def errors(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    d = tmp_path_factory.mktemp("newman")
    src, exe = d / "newman.cpp", d / "newman"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-w", "-I", os.path.join(ROOT, "hams-mrel_gb300", "csrc"),
                    "-I", os.path.join(CUDA, "include"), str(src), "-o", str(exe)], check=True)
    return lambda *a: map(float, subprocess.run([str(exe), *map(str, a)], check=True, capture_output=True,
                                                text=True).stdout.split())


# An edge's number is of the order of size^6 times the height over the size squared: 1e-30 and 1e30 lie between the
# ends of these sizes and their neighbours.
@pytest.mark.parametrize("size", [1e-7, 1e-5, 1e-2, 1.0, 1e3, 1e6])
@pytest.mark.parametrize("nv", [3, 4])
def test_integral_and_gradient(errors, size, nv):
    """A wrong turn is 2 pi in the gradient.  Low above an edge's line the angles are quotients of small terms and
    s - l is next to nothing beside s, where double precision loses up to half its digits by itself: the bound is
    four times the largest error of the formula written out in double precision over the same points."""
    d, plain, dg, plain_g = errors(size, nv)
    assert plain_g < 1e-3
    assert d <= 4 * plain and dg <= 4 * plain_g
