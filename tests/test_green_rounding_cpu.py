"""Rounding of the deep-water Green function and of Newman's panel integral
(hg_green.cuh, compiled for the host) against extended precision: no further
from it than the formulas written out in double precision, on average over
the pairs of a mesh's distances.  The averages are over some 10^5 pairs each
and fluctuate by about a per cent."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

PROGRAM = r'''
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <random>
#include <vector>
#include "hg_green.cuh"
using namespace hg;
typedef long double ld;

template <class T> T poly(std::vector<double> c, T t) {
  T g = c.back();
  for (int k = (int)c.size() - 2; k >= 0; --k) g = g * t + (T)c[k];
  return g;
}
// G and its gradient as the formulas stand, re and im of each.
template <class T> void green(const double* q, const double* p, double v_, int flag, T o[8]) {
  const T pi = acosl(-1.0L), v = v_, dx = (T)q[0] - p[0], dy = (T)q[1] - p[1], zz = (T)q[2] + p[2], dz = (T)q[2] - p[2];
  const T R = sqrt(dx * dx + dy * dy), r1 = sqrt(R * R + zz * zz), hh = v * R, vv = v * zz;
  const T dd = sqrt(hh * hh + vv * vv), al = -vv / dd, be = hh / dd, rho = dd / (1 + dd), om = 1 - rho, ev = exp(vv);
  const T d3 = 1 + dd * dd * dd;
  const T pa = poly<T>({1.21, -13.328, 215.896, -1763.96, 8418.94, -24314.21, 42002.57, -41592.9, 21859.0, -4838.6}, rho);
  const T pb = poly<T>({0.938, 5.373, -67.92, 796.534, -4780.77, 17137.74, -36618.81, 44894.06, -29030.24, 7671.22}, rho);
  const T pc = poly<T>({1.268, -9.747, 209.653, -1397.89, 5155.67, -9844.35, 9136.4, -3272.62}, rho);
  const T pd = poly<T>({0.632, -40.97, 667.16, -6072.07, 31127.39, -96293.05, 181856.75, -205690.43, 128170.2, -33744.6}, rho);
  const T da = poly<T>({2.948, -24.53, 249.69, -754.85, -1187.71, 16370.75, -48811.41, 68220.87, -46688.0, 12622.25}, rho);
  const T db = poly<T>({1.11, 2.894, -76.765, 1565.35, -11336.19, 44270.15, -97014.11, 118879.26, -76209.82, 19923.28}, rho);
  const T dc = poly<T>({14.19, -148.24, 847.8, -2318.58, 3168.35, -1590.27}, rho);
  const T pp = (log(dd / 2 - vv / 2) + (T)0.5772156649 - 2 * dd * dd) * ev + dd * dd - vv;
  T rr = (1 - be) * pa - be * pb - al * pc / (1 + 6 * al * rho * om) + be * (1 - be) * pd;
  const T l0 = 2 * pp / d3 + 2 * (rho * om * om * om * rr);
  T j0, j1, h0, h1;
  if (hh <= 3) {
    const T y = (hh / 3) * (hh / 3);
    j0 = poly<T>({0.999999999, -2.249999879, 1.265623060, -0.316394552, 0.044460948, -0.003954479, 0.000212950}, y);
    j1 = hh * poly<T>({0.5, -0.562499992, 0.210937377, -0.039550040, 0.004447331, -0.000330547, 0.000015525}, y);
    h0 = hh / 3 * poly<T>({1.909859164, -1.909855001, 0.687514637, -0.126164557, 0.013828813, -0.000876918}, y);
    h1 = y * poly<T>({1.909859286, -1.145914713, 0.294656958, -0.042070508, 0.003785727, -0.000207183}, y);
  } else {
    const T z = 3 / hh, y = z * z, s = 1 / sqrt(hh);
    const T f0 = poly<T>({0.79788454, -0.00553897, 0.00099336, -0.00044346, 0.00020445, -0.00004959}, y) * s;
    const T t0 = hh - pi / 4 + z * poly<T>({-0.04166592, 0.00239399, -0.00073984, 0.00031099, -0.00007605}, y);
    const T f1 = poly<T>({0.79788459, 0.01662008, -0.00187002, 0.00068519, -0.00029440, 0.00006952}, y) * s;
    const T t1 = hh - 3 * pi / 4 + z * poly<T>({0.12499895, -0.00605240, 0.00135825, -0.00049616, 0.00011531}, y);
    j0 = f0 * cos(t0); j1 = f1 * cos(t1);
    h0 = 2 * poly<T>({0.99999906, 4.77228920, 3.85542044, 0.32303607}, y) /
             (pi * hh * poly<T>({1.0, 4.88331068, 4.28957333, 0.52120508}, y)) + f0 * sin(t0);
    h1 = 2 * poly<T>({1.00000004, 3.92205313, 2.64893033, 0.27450895}, y) /
             (pi * poly<T>({1.0, 3.81095112, 2.26216956, 0.10885141}, y)) + f1 * sin(t1);
  }
  const T tp = 2 * pi * ev, ps = (be + hh) / (dd - vv) - 2 * be + 2 * ev * dd - hh, qs = exp(-dd) * (1 - be) * (1 + dd / d3);
  rr = be * da - (1 - al) * db + be * (1 - be) * rho * (1 - 2 * rho) * dc;
  const T ls = 2 * ps / d3 - 4 * qs + 2 * (rho * om * om * om * rr);
  const T g0 = l0 + tp * h0, i0 = -tp * j0, g1 = ls + tp * (2 / pi - h1), i1 = tp * j1, ir = 1 / r1, i3 = ir * ir * ir;
  const T cx = -v * v * dx / R, cy = -v * v * dy / R;
  o[0] = -v * g0 + ir; o[1] = -v * i0;
  o[2] = g1 * cx - dx * i3; o[3] = i1 * cx;
  o[4] = g1 * cy - dy * i3; o[5] = i1 * cy;
  o[6] = -v * v * g0 + 2 * v * ir - zz * i3; o[7] = -v * v * i0;
  if (!flag) {
    const T is = 1 / sqrt(R * R + dz * dz), s3 = is * is * is;
    o[0] += is; o[2] -= dx * s3; o[4] -= dy * s3; o[6] -= dz * s3;
  }
}
// Newman's integral as the formulas stand.
template <class T> void newman(const double* pr, const double* f, T o[4]) {
  T p[3], c[3];
  for (int k = 0; k < 3; ++k) p[k] = (T)f[k] - pr[PR_PO + k];
  for (int a = 0; a < 3; ++a) c[a] = pr[PR_UI + 3 * a] * p[0] + pr[PR_UI + 3 * a + 1] * p[1] + pr[PR_UI + 3 * a + 2] * p[2];
  const T x = c[0], y = c[1], z = c[2];
  const int nv = (int)pr[PR_NCN];
  T st = 0, sx = 0, sy = 0, sz = 0;
  for (int e = 0; e < nv; ++e) {
    const int n = (e + 1) % nv;
    const T k1 = pr[PR_KSI + e], e1 = pr[PR_ETA + e], k2 = pr[PR_KSI + n], e2 = pr[PR_ETA + n], l = pr[PR_L + e];
    const T dk = k2 - k1, de = e2 - e1;
    const T r1 = sqrt((k1 - x) * (k1 - x) + (e1 - y) * (e1 - y) + z * z), r2 = sqrt((k2 - x) * (k2 - x) + (e2 - y) * (e2 - y) + z * z);
    const T b1 = de * ((k1 - x) * (k1 - x) + z * z) - dk * (k1 - x) * (e1 - y), a1 = r1 * z * dk;
    const T b2 = de * ((k2 - x) * (k2 - x) + z * z) - dk * (k2 - x) * (e2 - y), a2 = r2 * z * dk;
    if (!(std::abs((double)z) < 1e-6)) sz += atan2(b1 * a2 - b2 * a1, a1 * a2 + b1 * b2);
    const T s = r1 + r2;
    if (std::abs((double)(s - l)) < 1e-6) continue;
    const T lg = log((s + l) / (s - l));
    sx -= de / l * lg; sy += dk / l * lg; st += (de * (x - k1) - dk * (y - e1)) / l * lg;
  }
  const T sg = nv == 3 ? 1 : -1;
  o[0] = sg * (st - z * sz);
  for (int k = 0; k < 3; ++k) o[1 + k] = sg * (pr[PR_UI + k] * sx + pr[PR_UJ + k] * sy + pr[PR_UK + k] * sz);
}

static std::mt19937_64 gen(5);
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(gen); }
static double nrm() { return std::normal_distribution<double>()(gen); }
static void direction(double d[3]) {
  double n = 0;
  for (int k = 0; k < 3; ++k) { d[k] = nrm(); n += d[k] * d[k]; }
  for (int k = 0; k < 3; ++k) d[k] /= std::sqrt(n);
}
// a planar panel of about `size` in a random frame
static void panel(double pr[PR_SIZE], bool tri, double size) {
  double a[3], b[3], dot = 0, n = 0;
  direction(a); direction(b);
  for (int k = 0; k < 3; ++k) dot += a[k] * b[k];
  for (int k = 0; k < 3; ++k) { b[k] -= dot * a[k]; n += b[k] * b[k]; }
  for (int k = 0; k < 3; ++k) b[k] /= std::sqrt(n);
  for (int k = 0; k < 3; ++k) {
    pr[PR_PO + k] = size * uni(-10, 10);
    pr[PR_UI + k] = a[k]; pr[PR_UJ + k] = b[k];
    pr[PR_UK + k] = a[(k + 1) % 3] * b[(k + 2) % 3] - a[(k + 2) % 3] * b[(k + 1) % 3];
  }
  const double w = uni(0.15, 0.65), h = uni(0.15, 0.65), sx[4] = {1, -1, -1, 1}, sy[4] = {1, 1, -1, -1};
  const int nv = tri ? 3 : 4;
  pr[PR_NCN] = nv;
  for (int e = 0; e < nv; ++e) {
    pr[PR_KSI + e] = size * (sx[e] * w + uni(-.05, .05));
    pr[PR_ETA + e] = size * (sy[e] * h + uni(-.05, .05));
  }
  for (int e = 0; e < nv; ++e) {
    const int x = (e + 1) % nv;
    pr[PR_L + e] = std::hypot(pr[PR_KSI + x] - pr[PR_KSI + e], pr[PR_ETA + x] - pr[PR_ETA + e]);
  }
}

int main() {
  // relative errors of G, of its horizontal and of its vertical derivative, ours and the double formula's
  for (int band = 0; band < 4; ++band) {  // near-vertical pairs, then R to 3, 20 and 80 m
    double e[3][2] = {};
    const double lo[] = {5e-5, 0.05, 3, 20}, hi[] = {0.05, 3, 20, 80};
    for (int k = 0; k < 100000; ++k) {
      const double w = uni(0.3, 2.0), v = w * w / 9.80665, r = lo[band] * std::pow(hi[band] / lo[band], uni(0, 1)), t = uni(0, 6.283185);
      const double q[3] = {uni(-30, 30), uni(-30, 30), -uni(.05, 10)}, p[3] = {q[0] + r * std::cos(t), q[1] + r * std::sin(t), -uni(.05, 10)};
      const int flag = r < 20;
      double2 g[4];
      double d[8];
      ld x[8];
      inf_green(q[0], q[1], q[2], p[0], p[1], p[2], v, 1.0 / v, flag, g);
      green<double>(q, p, v, flag, d);
      green<ld>(q, p, v, flag, x);
      const int first[] = {0, 2, 6}, count[] = {2, 4, 2};
      for (int m = 0; m < 3; ++m) {
        double s = 0, a = 0, b = 0;
        for (int c = first[m]; c < first[m] + count[m]; ++c) {
          s += (double)(x[c] * x[c]);
          const double ours = (c & 1) ? g[c / 2].y : g[c / 2].x;
          a += (double)((ours - x[c]) * (ours - x[c]));
          b += (double)((d[c] - x[c]) * (d[c] - x[c]));
        }
        e[m][0] += std::sqrt(a / s);
        e[m][1] += std::sqrt(b / s);
      }
    }
    for (int m = 0; m < 3; ++m) std::printf("green%d_%d %.6g %.6g\n", band, m, e[m][0], e[m][1]);
  }
  // the same of the integral and its gradient
  for (int band = 0; band < 5; ++band) {  // the panel's own point, then distances in panel sizes
    double e[2][2] = {};
    const double lo[] = {0, 0.3, 1.5, 5, 15}, hi[] = {0, 1.5, 5, 15, 50};
    for (int k = 0; k < 100000; ++k) {
      double pr[PR_SIZE] = {}, f[3], u[3], o[4], d[4];
      ld x[4];
      panel(pr, k % 4 == 3, 1.0);
      direction(u);
      const double r = band ? lo[band] * std::pow(hi[band] / lo[band], uni(0, 1)) : 0.0;
      for (int c = 0; c < 3; ++c) f[c] = pr[PR_PO + c] + r * u[c];
      newman_pair(pr, f[0], f[1], f[2], o[0], o[1], o[2], o[3]);
      newman<double>(pr, f, d);
      newman<ld>(pr, f, x);
      e[0][0] += std::abs((double)((o[0] - x[0]) / x[0]));
      e[0][1] += std::abs((double)((d[0] - x[0]) / x[0]));
      double s = 0, a = 0, b = 0;
      for (int c = 1; c < 4; ++c) {
        s += (double)(x[c] * x[c]);
        a += (double)((o[c] - x[c]) * (o[c] - x[c]));
        b += (double)((d[c] - x[c]) * (d[c] - x[c]));
      }
      e[1][0] += std::sqrt(a / s);
      e[1][1] += std::sqrt(b / s);
    }
    for (int m = 0; m < 2; ++m) std::printf("newman%d_%d %.6g %.6g\n", band, m, e[m][0], e[m][1]);
  }
  return 0;
}
'''


@pytest.fixture(scope="module")
def sums(tmp_path_factory):
    cxx = shutil.which("g++")
    if not cxx or not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no C++ compiler or CUDA headers")
    d = tmp_path_factory.mktemp("green")
    src, exe = d / "green.cpp", d / "green"
    src.write_text(PROGRAM)
    subprocess.run([cxx, "-std=c++17", "-O2", "-ffp-contract=off", "-w", "-I", os.path.join(ROOT, "hams-mrel_gb300", "csrc"),
                    "-I", os.path.join(CUDA, "include"), str(src), "-o", str(exe)], check=True)
    out = subprocess.run([str(exe)], check=True, capture_output=True, text=True).stdout
    return {k: (float(a), float(b)) for k, a, b in (line.split() for line in out.splitlines())}


# a mean further off than the plain formula's by more than three of its own fluctuations is a loss
@pytest.mark.parametrize("what", ["green%d_%d" % (b, m) for b in range(4) for m in range(3)] +
                         ["newman%d_%d" % (b, m) for b in range(5) for m in range(2)])
def test_no_further_off_than_the_formula_in_double(sums, what):
    ours, plain = sums[what]
    assert ours <= 1.03 * plain
