// Device-side free-surface Green functions and Newman panel integrals.
//
// Deep water: the Wu-Noblesse global approximation used by HAMS-MREL
// (src/InfGreen_Appr.f90:104-872).  exp(vv), exp(-dd) and log(dd-vv) are
// evaluated once per pair, and each J/Y Bessel pair shares one sincos: the
// reference's BesselY0/Y1 (:674-760) use the same modulus and phase
// polynomials as BesselJ0/J1 (:583-671), so Y = f*sin(theta)/sqrt(x) and
// J = f*cos(theta)/sqrt(x) come from one call.
//
// Finite depth: the region-decomposed Green function of src/FinGreen3D.f90
// (Linton / Pidcock / eigenfunction series with Wynn's epsilon algorithm),
// with every convergence loop bounded, the recursive Gauss-Kronrod 7-15
// quadrature turned into an explicit-stack loop, and the E_n(x) upward
// recursion of ENXA (src/FinGrnExtSubs.f90:82-107) advanced incrementally
// instead of restarted from E_1 on every series term.  Loops that hit their
// cap set HG_DEV_SERIES_CAP in the status word.
#pragma once
#include <string.h>
#include "hg_common.cuh"
#include "hg_rcp.cuh"

#ifdef __CUDACC__
#define HGD __host__ __device__
#define HGD_INL __host__ __device__ __forceinline__
#define HGD_CALL static __host__ __device__ __noinline__
#else
#define HGD
#define HGD_INL inline
#define HGD_CALL static inline
#endif

namespace hg {

#ifdef __CUDA_ARCH__
#define HGD_TABLE __device__ const
#else
#define HGD_TABLE static const
#endif

// ===================================================================
// Newman (1986) closed-form integral of 1/r and grad(1/r) over a flat
// panel, SingularIntgr.f90:44-244 (triangles) and :252-445 (quads).
// pr = 36-double source-panel record (hg_common.cuh).
//
// GB300's FP64 pipe (two operations a clock and SM) bounds every caller, so
// the work is arranged to spend few of them: vertex terms are formed once and
// shared by the two edges that meet there, distances are one rounded root each,
// 1 / l and 1 / (s - l) run on the integer pipes (hg_rcp.cuh) and each quotient
// takes one residual, and the edges' angles are added as the argument of one
// complex product: one atan2 instead of four, its multiple of 2 pi taken from
// the four single-precision angles.
//
// newman_pair is the form of the complex128 matrices; newman_pair_ref, in the
// reference's order of operations, that of entries rounded to single precision,
// where a last bit of the double now and then moves the stored value by one
// unit (outputs by up to 2e-8 near an irregular frequency).
// ===================================================================
HGD_INL void newman_pair_ref(const double* __restrict__ pr, double xf0, double xf1,
                                            double xf2, double& sij, double& d0, double& d1,
                                            double& d2) {
  const double p0 = xf0 - pr[PR_PO], p1 = xf1 - pr[PR_PO + 1], p2 = xf2 - pr[PR_PO + 2];
  const double x = pr[PR_UI] * p0 + pr[PR_UI + 1] * p1 + pr[PR_UI + 2] * p2;
  const double y = pr[PR_UJ] * p0 + pr[PR_UJ + 1] * p1 + pr[PR_UJ + 2] * p2;
  const double z = pr[PR_UK] * p0 + pr[PR_UK + 1] * p1 + pr[PR_UK + 2] * p2;
  const int nv = (int)pr[PR_NCN];
  const bool tri = (nv == 3);
  double st = 0.0, sxt = 0.0, syt = 0.0, szt = 0.0;
  const double z2 = z * z;
  double ksa = pr[PR_KSI], eta_a = pr[PR_ETA];
  const double r_first = sqrt((ksa - x) * (ksa - x) + (eta_a - y) * (eta_a - y) + z2);
  double r1 = r_first;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (e >= nv) break;
    const int nx = (e + 1 == nv) ? 0 : e + 1;
    const double ksb = pr[PR_KSI + nx], etb = pr[PR_ETA + nx];
    const double r2 = (nx == 0) ? r_first : sqrt((ksb - x) * (ksb - x) + (etb - y) * (etb - y) + z2);
    const double l = pr[PR_L + e];
    if (!tri && fabs(l) < 1.0e-8) {
      ksa = ksb; eta_a = etb; r1 = r2;
      continue;
    }
    const double dksi = ksb - ksa, deta = etb - eta_a;
    const double b1 = deta * ((ksa - x) * (ksa - x) + z2) - dksi * (ksa - x) * (eta_a - y);
    const double a1 = r1 * z * dksi;
    const double b2 = deta * ((ksb - x) * (ksb - x) + z2) - dksi * (ksb - x) * (etb - y);
    const double a2 = r2 * z * dksi;
    if (!(fabs(z) < 1.0e-6)) szt += atan2(b1 * a2 - b2 * a1, a1 * a2 + b1 * b2);
    const double s = r1 + r2;
    if (!(fabs(s - l) < 1.0e-6)) {
      const double lg = log((s + l) / (s - l));
      sxt -= deta / l * lg;
      syt += dksi / l * lg;
      const double t = (deta * (x - ksa) - dksi * (y - eta_a)) / l * lg;
      st = tri ? st + t : st - t;
    }
    ksa = ksb; eta_a = etb; r1 = r2;
  }
  sij = tri ? st - z * szt : st + z * szt;
  const double sg = tri ? 1.0 : -1.0;
  d0 = sg * (pr[PR_UI] * sxt + pr[PR_UJ] * syt + pr[PR_UK] * szt);
  d1 = sg * (pr[PR_UI + 1] * sxt + pr[PR_UJ + 1] * syt + pr[PR_UK + 1] * szt);
  d2 = sg * (pr[PR_UI + 2] * sxt + pr[PR_UJ + 2] * syt + pr[PR_UK + 2] * szt);
}

// The same out of line, for kernels that take it only for one option.
HGD_CALL void newman_pair_ref_call(const double* __restrict__ pr, double xf0, double xf1, double xf2,
                                                         double& sij, double& d0, double& d1, double& d2) {
  newman_pair_ref(pr, xf0, xf1, xf2, sij, d0, d1, d2);
}

// The angles' sum edge by edge (x, y, z in the panel's frame).
HGD_CALL double newman_angles(const double* __restrict__ pr, double x, double y, double z) {
  const int nv = (int)pr[PR_NCN];
  double szt = 0.0;
  for (int e = 0; e < nv; ++e) {
    const int nx = (e + 1 == nv) ? 0 : e + 1;
    if (nv == 4 && fabs(pr[PR_L + e]) < 1.0e-8) continue;
    const double dx = pr[PR_KSI + e] - x, dy = pr[PR_ETA + e] - y, ex = pr[PR_KSI + nx] - x, ey = pr[PR_ETA + nx] - y;
    const double dksi = pr[PR_KSI + nx] - pr[PR_KSI + e], deta = pr[PR_ETA + nx] - pr[PR_ETA + e], z2 = z * z;
    const double b1 = deta * (dx * dx + z2) - dksi * dx * dy, a1 = sqrt(dx * dx + dy * dy + z2) * z * dksi;
    const double b2 = deta * (ex * ex + z2) - dksi * ex * ey, a2 = sqrt(ex * ex + ey * ey + z2) * z * dksi;
    szt += atan2(b1 * a2 - b2 * a1, a1 * a2 + b1 * b2);
  }
  return szt;
}

HGD_INL void newman_pair(const double* __restrict__ pr, double xf0, double xf1, double xf2,
                                            double& sij, double& d0, double& d1, double& d2) {
  const double p0 = xf0 - pr[PR_PO], p1 = xf1 - pr[PR_PO + 1], p2 = xf2 - pr[PR_PO + 2];
  const double x = fma(pr[PR_UI + 2], p2, fma(pr[PR_UI + 1], p1, pr[PR_UI] * p0));
  const double y = fma(pr[PR_UJ + 2], p2, fma(pr[PR_UJ + 1], p1, pr[PR_UJ] * p0));
  const double z = fma(pr[PR_UK + 2], p2, fma(pr[PR_UK + 1], p1, pr[PR_UK] * p0));
  const int nv = (int)pr[PR_NCN];
  const bool tri = (nv == 3);
  const bool flat = fabs(z) < 1.0e-6;  // in the panel's plane: no angle terms
  const double z2 = z * z;
  // vertex terms: offset, p = dx^2 + z^2, q = dx dy, distance r
  double dx = pr[PR_KSI] - x, dy = pr[PR_ETA] - y;
  double va = fma(dx, dx, z2), vq = dx * dy, vr = fma(dy, dy, va);
  vr = sqrt_near(vr);
  const double fdx = dx, fdy = dy, fa = va, fq = vq, fr = vr;
  double st = 0.0, sxt = 0.0, syt = 0.0, szt = 0.0;
  double zr = 1.0, zi = 0.0;        // product of the edges' complex numbers
  float turns = 0.f;                // sum of their angles, single precision
  bool plain = false;               // a factor out of the product's safe range: add the angles one by one
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    if (e >= nv) break;
    const int nx = (e + 1 == nv) ? 0 : e + 1;
    double ex, ey, wa, wq, wr;
    if (nx == 0) {
      ex = fdx; ey = fdy; wa = fa; wq = fq; wr = fr;
    } else {
      ex = pr[PR_KSI + nx] - x;
      ey = pr[PR_ETA + nx] - y;
      wa = fma(ex, ex, z2);
      wq = ex * ey;
      wr = fma(ey, ey, wa);
      wr = sqrt_near(wr);
    }
    const double l = pr[PR_L + e];
    if (tri || !(fabs(l) < 1.0e-8)) {
      const double dksi = pr[PR_KSI + nx] - pr[PR_KSI + e], deta = pr[PR_ETA + nx] - pr[PR_ETA + e];
      if (!flat) {
        const double zd = z * dksi, a1 = vr * zd, a2 = wr * zd;
        const double b1 = fma(deta, va, -(dksi * vq)), b2 = fma(deta, wa, -(dksi * wq));
        const double im = fma(b1, a2, -(b2 * a1)), re = fma(a1, a2, b1 * b2);
        const float fi = (float)im, fre = (float)re, fm = fmaxf(fabsf(fi), fabsf(fre));
        plain = plain || !(fm > 1e-30f && fm < 1e30f);
        turns += atan2f(fi, fre);
        const double t = fma(zr, re, -(zi * im));
        zi = fma(zr, im, zi * re);
        zr = t;
      }
      const double s = vr + wr, gap = s - l;
      if (!(fabs(gap) < 1.0e-6)) {
        // both quotients rounded once: far from the panel the edges' logarithms cancel to the square of its
        // angle, and what their arguments are off by is left over
        const double ig = rcp_any(gap), top = s + l, q = top * ig, lq = log(fma(fma(-q, gap, top), ig, q));
        const double il = rcp_any(l), l0 = lq * il, lg = fma(fma(-l0, l, lq), il, l0);
        sxt = fma(-deta, lg, sxt);
        syt = fma(dksi, lg, syt);
        st = fma(fma(dksi, dy, -(deta * dx)), lg, st);  // deta (x - ksi) - dksi (y - eta)
      }
    }
    dx = ex; dy = ey; va = wa; vq = wq; vr = wr;
  }
  if (!flat) {
    if (!plain) {
      szt = atan2(zi, zr);
      szt = fma(rintf((turns - (float)szt) * 0.15915494f), 2.0 * HG_PI, szt);
    } else {
      szt = newman_angles(pr, x, y, z);
    }
  }
  const double sg = tri ? 1.0 : -1.0;
  sij = sg * fma(-z, szt, st);
  d0 = sg * fma(pr[PR_UK], szt, fma(pr[PR_UJ], syt, pr[PR_UI] * sxt));
  d1 = sg * fma(pr[PR_UK + 1], szt, fma(pr[PR_UJ + 1], syt, pr[PR_UI + 1] * sxt));
  d2 = sg * fma(pr[PR_UK + 2], szt, fma(pr[PR_UJ + 2], syt, pr[PR_UI + 2] * sxt));
}

// ===================================================================
// Deep water.  As above FP64 operations are what counts: Horner steps are
// fused, the nine divisions left of some thirty-five are reciprocals on the
// integer pipes, and the distances' square roots come from their reciprocals
// and are rounded by one residual (measured at 6048 panels: see k_green_fill).
// ===================================================================
template <int N>
HGD_INL double horner(const double (&c)[N], double t) {
  double g = c[N - 1];
#pragma unroll
  for (int k = N - 2; k >= 0; --k) g = fma(g, t, c[k]);
  return g;
}

// Havelock wave term GF and its horizontal derivative GFh at the
// non-dimensional horizontal distance hh = v*R and depth vv = v*(z+zeta);
// idd = 1 / |(hh, vv)| to a few units, ihh = 1 / hh (used beyond 3).  dd is the
// rounded root of the rounded hh^2 + vv^2, so that it equals -vv above the source:
// GFh is what is left there of terms of the size of exp(vv) and exp(-dd), and
// 1 - alpha is formed from dd + vv for the same reason.  (With dd taken from R
// and z + zeta the horizontal derivatives of near-vertical pairs were 1.6 times
// as far off, 2.0e-13 of their size against 1.2e-13.)
HGD_INL void havelock(double hh, double vv, double idd, double ihh, double2& gf, double2& gfh) {
  const double gama = 0.5772156649;
  const double dd = root_of(fma(hh, hh, vv * vv), idd), alpha = -vv * idd, oma = (dd + vv) * idd, beta = hh * idd;
  const double opd = 1.0 + dd, omr = rcp_any(opd);  // 1 - rho
  double rho = dd * omr;
  rho = fma(fma(-rho, opd, dd), omr, rho);  // dd / (1 + dd), rounded
  const double ev = exp(vv), emd = exp(-dd);
  const double id3 = rcp_any(fma(dd * dd, dd, 1.0));
  const double ro3 = rho * (omr * omr * omr), ob = 1.0 - beta, lam = dd - vv;
  const double pa = horner({1.21, -13.328, 215.896, -1763.96, 8418.94, -24314.21, 42002.57, -41592.9, 21859.0, -4838.6},
                           rho);
  const double pb = horner({0.938, 5.373, -67.92, 796.534, -4780.77, 17137.74, -36618.81, 44894.06, -29030.24, 7671.22},
                           rho);
  const double pc = horner({1.268, -9.747, 209.653, -1397.89, 5155.67, -9844.35, 9136.4, -3272.62}, rho);
  const double pd = horner({0.632, -40.97, 667.16, -6072.07, 31127.39, -96293.05, 181856.75, -205690.43, 128170.2,
                            -33744.6}, rho);
  const double da = horner({2.948, -24.53, 249.69, -754.85, -1187.71, 16370.75, -48811.41, 68220.87, -46688.0, 12622.25},
                           rho);
  const double db = horner({1.11, 2.894, -76.765, 1565.35, -11336.19, 44270.15, -97014.11, 118879.26, -76209.82,
                            19923.28}, rho);
  const double dc = horner({14.19, -148.24, 847.8, -2318.58, 3168.35, -1590.27}, rho);
  const double bob = beta * ob, dd2 = dd * dd;
  const double pp = fma(fma(-2.0, dd2, log(0.5 * lam) + gama), ev, dd2 - vv);
  double rr = fma(bob, pd, fma(-(alpha * pc), rcp_any(fma(6.0 * alpha, rho * omr, 1.0)), fma(-beta, pb, ob * pa)));
  const double l0 = 2.0 * fma(pp, id3, ro3 * rr);
  double j0, j1, h0, h1;
  if (hh <= 3.0) {
    const double th = hh * (1.0 / 3.0), yy = th * th;
    j0 = horner({0.999999999, -2.249999879, 1.265623060, -0.316394552, 0.044460948, -0.003954479, 0.000212950}, yy);
    j1 = horner({0.5, -0.562499992, 0.210937377, -0.039550040, 0.004447331, -0.000330547, 0.000015525}, yy) * hh;
    h0 = horner({1.909859164, -1.909855001, 0.687514637, -0.126164557, 0.013828813, -0.000876918}, yy) * th;
    h1 = horner({1.909859286, -1.145914713, 0.294656958, -0.042070508, 0.003785727, -0.000207183}, yy) * yy;
  } else {
    const double y = 3.0 * ihh, y2 = y * y, isq = rsqrt_near(hh);
    const double f0 = horner({0.79788454, -0.00553897, 0.00099336, -0.00044346, 0.00020445, -0.00004959}, y2) * isq;
    const double t0 = fma(horner({-0.04166592, 0.00239399, -0.00073984, 0.00031099, -0.00007605}, y2), y,
                          hh - 0.25 * HG_PI);
    const double f1 = horner({0.79788459, 0.01662008, -0.00187002, 0.00068519, -0.00029440, 0.00006952}, y2) * isq;
    const double t1 = fma(horner({0.12499895, -0.00605240, 0.00135825, -0.00049616, 0.00011531}, y2), y,
                          hh - 0.75 * HG_PI);
    double s0, c0, s1, c1;
    sincos(t0, &s0, &c0);
    sincos(t1, &s1, &c1);
    j0 = f0 * c0;
    j1 = f1 * c1;
    const double e0 = horner({1.0, 4.88331068, 4.28957333, 0.52120508}, y2);
    const double e1 = horner({1.0, 3.81095112, 2.26216956, 0.10885141}, y2);
    const double ie = rcp_any(e0 * e1) * (2.0 / HG_PI);  // both denominators in one reciprocal
    h0 = fma(horner({0.99999906, 4.77228920, 3.85542044, 0.32303607}, y2) * (ie * e1), ihh, f0 * s0);
    h1 = fma(horner({1.00000004, 3.92205313, 2.64893033, 0.27450895}, y2), ie * e0, f1 * s1);
  }
  const double tpe = 2.0 * HG_PI * ev;
  gf = make_double2(fma(tpe, h0, l0), -tpe * j0);
  const double ps = fma(beta + hh, rcp_any(lam), fma(2.0 * ev, dd, fma(-2.0, beta, -hh)));
  const double qs = emd * ob * fma(dd, id3, 1.0);
  rr = fma(bob * rho * fma(-2.0, rho, 1.0), dc, fma(beta, da, -(oma * db)));
  const double ls = fma(2.0, fma(ps, id3, ro3 * rr), -4.0 * qs);
  gfh = make_double2(fma(tpe, 2.0 / HG_PI - h1, ls), tpe * j1);
}

// INFGREEN3D (InfGreen_Appr.f90:104-186).  Source (xq,yq,zq), field (xp,yp,zp).
HGD_INL void inf_green(double xq, double yq, double zq, double xp, double yp, double zp, double v,
                                          double iv, int flag, double2 g[4]) {
  const double xpq = xq - xp, ypq = yq - yp, zpq = zp + zq, zd = zq - zp;
  const double h2 = fma(xpq, xpq, ypq * ypq);
  const double irr = h2 > 0.0 ? rsqrt_near(h2) : 0.0, rr = root_of(h2, irr);
  const double q1 = fma(zpq, zpq, h2), ir1 = rsqrt_near(q1), ir13 = ir1 * ir1 * ir1;
  double sgn1 = 1.0;  // sign of the image term: -1 at the infinite-frequency limit
  if (fabs(v) < SPD(1.e-8) || fabs(v + 1.0) < SPD(1.e-8)) {
    if (!(fabs(v) < SPD(1.e-8))) sgn1 = -1.0;
    g[0] = make_double2(0.0, 0.0); g[1] = g[0]; g[2] = g[0]; g[3] = g[0];
  } else {
    double2 gf, gfh;
    havelock(v * rr, v * zpq, fabs(iv) * ir1, irr * iv, gf, gfh);
    const double v2 = v * v;
    if (rr > SPD(1.e-6)) {
      const double c = -v2 * irr, cx = c * xpq, cy = c * ypq;
      g[1] = make_double2(gfh.x * cx, gfh.y * cx);
      g[2] = make_double2(gfh.x * cy, gfh.y * cy);
    } else {
      g[1] = make_double2(0.0, 0.0);
      g[2] = make_double2(0.0, 0.0);
    }
    g[0] = make_double2(-v * gf.x, -v * gf.y);
    g[3] = make_double2(fma(2.0 * v, ir1, -v2 * gf.x), -v2 * gf.y);
  }
  const double i3 = sgn1 * ir13;
  g[0].x = fma(sgn1, ir1, g[0].x);
  g[1].x = fma(-xpq, i3, g[1].x);
  g[2].x = fma(-ypq, i3, g[2].x);
  g[3].x = fma(-zpq, i3, g[3].x);
  if (flag == 0) {
    const double ir = rsqrt_near(fma(zd, zd, h2)), ir3 = ir * ir * ir;
    g[0].x += ir;
    g[1].x = fma(-xpq, ir3, g[1].x);
    g[2].x = fma(-ypq, ir3, g[2].x);
    g[3].x = fma(-zd, ir3, g[3].x);
  }
}

// ===================================================================
// Finite depth: special functions (FinGrnExtSubs.f90)
// ===================================================================
// p[k] = x**k, k = 1 .. 12, each by binary powering (the evaluation order a
// Fortran compiler uses for an integer exponent), the squares shared.
HGD inline void powers12(double x, double p[13]) {
  p[1] = x;
  p[2] = x * x;
  p[4] = p[2] * p[2];
  p[8] = p[4] * p[4];
  p[3] = p[1] * p[2];
  p[5] = p[1] * p[4];
  p[6] = p[2] * p[4];
  p[7] = p[3] * p[4];
  p[9] = p[1] * p[8];
  p[10] = p[2] * p[8];
  p[11] = p[3] * p[8];
  p[12] = p[4] * p[8];
}
HGD inline double d_error(double x) {  // ERROR :62-93
  const double x2 = x * x;
  if (fabs(x) < 3.5) {
    double er = 1.0, r = 1.0;
    for (int k = 1; k <= 50; ++k) {
      r = r * x2 / (k + 0.5);
      er += r;
      if (fabs(r) <= fabs(er) * 1.0e-15) break;
    }
    return 2.0 / sqrt(HG_PI) * x * exp(-x2) * er;
  }
  double er = 1.0, r = 1.0;
  for (int k = 1; k <= 12; ++k) {
    r = -r * (k - 0.5) / x2;
    er += r;
  }
  double e = 1.0 - exp(-x2) / (fabs(x) * sqrt(HG_PI)) * er;
  return x < 0.0 ? -e : e;
}
HGD inline double d_erfcc(double x) { return 1.0 - d_error(x); }
HGD inline double d_derfcc(double x) { return -2.0 / sqrt(HG_PI) * exp(-(x * x)); }

HGD inline double d_e1xa(double x) {  // E1XA :119-133
  if (x == 0.0) return 1.0e+300;
  if (x <= 1.0)
    return -log(x) + ((((1.07857e-3 * x - 9.76004e-3) * x + 5.519968e-2) * x - 0.24991055) * x +
                      0.99999193) * x - 0.57721566;
  const double es1 = (((x + 8.5733287401) * x + 18.059016973) * x + 8.6347608925) * x + 0.2677737343;
  const double es2 = (((x + 9.5733223454) * x + 25.6329561486) * x + 21.0996530827) * x + 3.9584969228;
  return exp(-x) / x * es1 / es2;
}

HGD inline double d_eix(double x) {  // EIX :146-172
  if (x == 0.0) return -1.0e+300;
  if (x <= 40.0) {
    double ei = 1.0, r = 1.0;
    for (int k = 1; k <= 100; ++k) {
      r = r * k * x / ((k + 1.0) * (k + 1.0));
      ei += r;
      if (fabs(r / ei) <= 1.0e-15) break;
    }
    return 0.5772156649015328 + log(x) + x * ei;
  }
  double ei = 1.0, r = 1.0;
  for (int k = 1; k <= 20; ++k) {
    r = r * k / x;
    ei += r;
  }
  return exp(x) / x * ei;
}

// Divisors of the K0/K1 power series, known in advance: k*k and k*(k+1) with
// their correctly rounded reciprocals, and the partial sums of 1/k in the order
// the series adds them.
#ifdef __CUDA_ARCH__
#define HGD_CONST __constant__ const
#else
#define HGD_CONST static const
#endif
HGD_CONST double c_kk[51] = {0.0,
1.0, 4.0, 9.0, 16.0, 25.0, 36.0, 49.0, 64.0, 81.0, 100.0,
    121.0, 144.0, 169.0, 196.0, 225.0, 256.0, 289.0, 324.0, 361.0, 400.0,
    441.0, 484.0, 529.0, 576.0, 625.0, 676.0, 729.0, 784.0, 841.0, 900.0,
    961.0, 1024.0, 1089.0, 1156.0, 1225.0, 1296.0, 1369.0, 1444.0, 1521.0, 1600.0,
    1681.0, 1764.0, 1849.0, 1936.0, 2025.0, 2116.0, 2209.0, 2304.0, 2401.0, 2500.0};
HGD_CONST double c_kk1[51] = {0.0,
2.0, 6.0, 12.0, 20.0, 30.0, 42.0, 56.0, 72.0, 90.0, 110.0,
    132.0, 156.0, 182.0, 210.0, 240.0, 272.0, 306.0, 342.0, 380.0, 420.0,
    462.0, 506.0, 552.0, 600.0, 650.0, 702.0, 756.0, 812.0, 870.0, 930.0,
    992.0, 1056.0, 1122.0, 1190.0, 1260.0, 1332.0, 1406.0, 1482.0, 1560.0, 1640.0,
    1722.0, 1806.0, 1892.0, 1980.0, 2070.0, 2162.0, 2256.0, 2352.0, 2450.0, 2550.0};
HGD_CONST double c_rcp_kk[51] = {0.0,
1.0, 0.25, 0.1111111111111111, 0.0625,
    0.04, 0.027777777777777776, 0.02040816326530612, 0.015625,
    0.012345679012345678, 0.01, 0.008264462809917356, 0.006944444444444444,
    0.005917159763313609, 0.00510204081632653, 0.0044444444444444444, 0.00390625,
    0.0034602076124567475, 0.0030864197530864196, 0.002770083102493075, 0.0025,
    0.0022675736961451248, 0.002066115702479339, 0.001890359168241966, 0.001736111111111111,
    0.0016, 0.0014792899408284023, 0.0013717421124828531, 0.0012755102040816326,
    0.0011890606420927466, 0.0011111111111111111, 0.001040582726326743, 0.0009765625,
    0.0009182736455463728, 0.0008650519031141869, 0.0008163265306122449, 0.0007716049382716049,
    0.0007304601899196494, 0.0006925207756232687, 0.0006574621959237344, 0.000625,
    0.000594883997620464, 0.0005668934240362812, 0.0005408328826392645, 0.0005165289256198347,
    0.0004938271604938272, 0.0004725897920604915, 0.0004526935264825713, 0.00043402777777777775,
    0.00041649312786339027, 0.0004};
HGD_CONST double c_rcp_kk1[51] = {0.0,
0.5, 0.16666666666666666, 0.08333333333333333, 0.05,
    0.03333333333333333, 0.023809523809523808, 0.017857142857142856, 0.013888888888888888,
    0.011111111111111112, 0.00909090909090909, 0.007575757575757576, 0.00641025641025641,
    0.005494505494505495, 0.004761904761904762, 0.004166666666666667, 0.003676470588235294,
    0.0032679738562091504, 0.0029239766081871343, 0.002631578947368421, 0.002380952380952381,
    0.0021645021645021645, 0.001976284584980237, 0.0018115942028985507, 0.0016666666666666668,
    0.0015384615384615385, 0.0014245014245014246, 0.0013227513227513227, 0.0012315270935960591,
    0.0011494252873563218, 0.001075268817204301, 0.0010080645161290322, 0.000946969696969697,
    0.00089126559714795, 0.0008403361344537816, 0.0007936507936507937, 0.0007507507507507507,
    0.0007112375533428165, 0.0006747638326585695, 0.000641025641025641, 0.0006097560975609756,
    0.0005807200929152149, 0.0005537098560354374, 0.0005285412262156448, 0.000505050505050505,
    0.0004830917874396135, 0.00046253469010175765, 0.0004432624113475177, 0.00042517006802721087,
    0.00040816326530612246, 0.000392156862745098};
HGD_CONST double c_harm[51] = {0.0,
1.0, 1.5, 1.8333333333333333, 2.083333333333333,
    2.283333333333333, 2.4499999999999997, 2.5928571428571425, 2.7178571428571425,
    2.8289682539682537, 2.9289682539682538, 3.0198773448773446, 3.103210678210678,
    3.180133755133755, 3.251562326562327, 3.3182289932289937, 3.3807289932289937,
    3.439552522640758, 3.4951080781963135, 3.547739657143682, 3.597739657143682,
    3.6453587047627294, 3.690813250217275, 3.73429151108684, 3.7759581777535067,
    3.8159581777535068, 3.854419716215045, 3.8914567532520823, 3.927171038966368,
    3.9616537975870574, 3.9949871309203906, 4.02724519543652, 4.05849519543652,
    4.08879822573955, 4.118209990445433, 4.146781419016861, 4.174559196794639,
    4.201586223821666, 4.22790201329535, 4.2535430389363755, 4.278543038936376,
    4.302933282838815, 4.326742806648339, 4.349998620601827, 4.3727258933290996,
    4.394948115551322, 4.416687245986104, 4.4379638417307845, 4.4587971750641175,
    4.4792053383294235, 4.499205338329423};

// a / d, correctly rounded, for a small integer d (here below 2^12) whose
// correctly rounded reciprocal rd is at hand (Markstein 1990; Brisebarre,
// Muller and Raina 2004): q = a rd is within 1.5 units in the last place, the
// residual a - d q is then exact (d is short), and q + residual rd is off the
// true quotient by far less than its distance from any midpoint (a multiple
// of 1 / (2 d) units).  Three FP64 operations where the general division
// takes about ten.
HGD inline double div_small(double a, double d, double rd) {
  const double q = a * rd;
  return fma(fma(-d, q, a), rd, q);
}

// fabs(num / den) < 1e-15 as the rounded division decides it.  The high words
// of two positive doubles differ by 2^20 times the logarithm (base 2) of their
// ratio, to 0.09 either way; 1e-15 is 2^-49.83, so outside a window around it
// they decide, and only inside is the division made.
HGD inline int hi_word(double x) {
#ifdef __CUDA_ARCH__
  return __double2hiint(x) & 0x7fffffff;
#else
  long long b;
  memcpy(&b, &x, sizeof b);
  return (int)(b >> 32) & 0x7fffffff;
#endif
}
// 1: below, 0: not below, -1: undecided; slack (in 2^-20) widens the window for
// a num known only to that relative accuracy.
HGD inline int ratio_guess(double num, double den, int slack) {
  const int hn = hi_word(num), hd = hi_word(den), g = hd - hn;
  if (hn >= 0x7ff00000 || hd >= 0x7ff00000 || hd < (60 << 20)) return -1;
  if (g > 52533657 + slack) return 1;   // 50.1 2^20
  if (g < 52009369 - slack) return 0;   // 49.6 2^20
  return -1;
}
HGD inline bool ratio_below(double num, double den) {
  const int t = ratio_guess(num, den, 0);
  return t < 0 ? fabs(num / den) < 1.0e-15 : t != 0;
}

// IK01A :538-640, returning K0 and K1.
HGD inline void d_ik01a(double x, double& bk0, double& bk1) {
  if (x == 0.0) { bk0 = 1.0e+300; bk1 = 1.0e+300; return; }
  const double x2 = x * x;
  double bi0, bi1;
  if (x <= 18.0) {
    const double xq = 0.25 * x2;  // the factor 0.25 is exact wherever it is applied
    bi0 = 1.0;
    double r = 1.0;
    for (int k = 1; k <= 50; ++k) {
      r = div_small(r * xq, c_kk[k], c_rcp_kk[k]);
      bi0 += r;
      if (ratio_below(r, bi0)) break;
    }
    bi1 = 1.0;
    r = 1.0;
    for (int k = 1; k <= 50; ++k) {
      r = div_small(r * xq, c_kk1[k], c_rcp_kk1[k]);
      bi1 += r;
      if (ratio_below(r, bi1)) break;
    }
    bi1 = 0.5 * x * bi1;
  } else {
    const double A[12] = {0.125, 7.03125e-2, 7.32421875e-2, 1.1215209960938e-1, 2.2710800170898e-1,
                          5.7250142097473e-1, 1.7277275025845, 6.0740420012735, 2.4380529699556e01,
                          1.1001714026925e02, 5.5133589612202e02, 3.0380905109224e03};
    const double B[12] = {-0.375, -1.171875e-1, -1.025390625e-1, -1.4419555664063e-1,
                          -2.7757644653320e-1, -6.7659258842468e-1, -1.9935317337513,
                          -6.8839142681099, -2.7248827311269e01, -1.2159789187654e02,
                          -6.0384407670507e02, -3.3022722944809e03};
    int k0 = 12;
    if (x >= 35.0) k0 = 9;
    if (x >= 50.0) k0 = 7;
    const double ca = exp(x) / sqrt(2.0 * HG_PI * x), xr = 1.0 / x;
    double p[13];
    powers12(xr, p);
    double s0 = 1.0, s1 = 1.0;
    for (int k = 1; k <= 12; ++k) {
      if (k > k0) break;
      s0 += A[k - 1] * p[k];
    }
    for (int k = 1; k <= 12; ++k) {
      if (k > k0) break;
      s1 += B[k - 1] * p[k];
    }
    bi0 = ca * s0;
    bi1 = ca * s1;
  }
  if (x <= 9.0) {
    const double ct = -(log(x / 2.0) + 0.5772156649015329);
    double k0v = 0.0, r = 1.0, ww = 0.0;
    const double xq = 0.25 * x2;
    for (int k = 1; k <= 50; ++k) {
      r = div_small(r, c_kk[k], c_rcp_kk[k]) * xq;
#ifdef HG_NO_CONTRACTION
      // the sum grew by the term to within half a unit, a ninth of the threshold: the term decides
      const double term = r * (c_harm[k] + ct);
      k0v += term;
      int t = ratio_guess(term, k0v, 524288);
      if (t < 0) t = ratio_below(k0v - ww, k0v);
      if (t) break;
#else  // the product of one use, so that it is fused into the sum
      k0v += r * (c_harm[k] + ct);
      if (ratio_below(k0v - ww, k0v)) break;
#endif
      ww = k0v;
    }
    bk0 = k0v + ct;
  } else {
    const double A1[8] = {0.125, 0.2109375, 1.0986328125, 1.1775970458984e01, 2.1461706161499e02,
                          5.9511522710323e03, 2.3347645606175e05, 1.2312234987631e07};
    const double xr2 = 1.0 / x2;
    double p[13];
    powers12(xr2, p);
    double s = 1.0;
    for (int k = 0; k < 8; ++k) s += A1[k] * p[k + 1];
    bk0 = 0.5 / x * s / bi0;
  }
  bk1 = (1.0 / x - bi1 * bk0) / bi0;
}

// JY01B :663-736
HGD inline void d_jy01b(double x, double& bj0, double& bj1, double& by0, double& by1) {
  if (x == 0.0) { bj0 = 1.0; bj1 = 0.0; by0 = -1.0e+300; by1 = -1.0e+300; return; }
  if (x <= 4.0) {
    const double t = x / 4.0, t2 = t * t;
    bj0 = ((((((-.5014415e-3 * t2 + .76771853e-2) * t2 - .0709253492) * t2 + .4443584263) * t2 -
             1.7777560599) * t2 + 3.9999973021) * t2 - 3.9999998721) * t2 + 1.0;
    bj1 = t * (((((((-.1289769e-3 * t2 + .22069155e-2) * t2 - .0236616773) * t2 + .1777582922) * t2 -
                  .8888839649) * t2 + 2.6666660544) * t2 - 3.9999999710) * t2 + 1.9999999998);
    const double lg = 2.0 / HG_PI * log(x / 2.0);
    by0 = lg * bj0 + ((((((((-.567433e-4 * t2 + .859977e-3) * t2 - .94855882e-2) * t2 + .0772975809) * t2 -
                         .4261737419) * t2 + 1.4216421221) * t2 - 2.3498519931) * t2 + SPD(1.0766115157)) * t2 +
                      .3674669052);
    by1 = lg * bj1 + (((((((((.6535773e-3 * t2 - .0108175626) * t2 + .107657606) * t2 - .7268945577) * t2 +
                           3.1261399273) * t2 - 7.3980241381) * t2 + 6.8529236342) * t2 + .3932562018) * t2 -
                        .6366197726) / x);
    return;
  }
  const double t = 4.0 / x, t2 = t * t, a0 = sqrt(2.0 / (HG_PI * x));
  const double p0 = ((((-.9285e-5 * t2 + .43506e-4) * t2 - .122226e-3) * t2 + .434725e-3) * t2 - .4394275e-2) * t2 + .999999997;
  const double q0 = t * (((((.8099e-5 * t2 - .35614e-4) * t2 + .85844e-4) * t2 - .218024e-3) * t2 + .1144106e-2) * t2 - .031249995);
  const double p1 = ((((.10632e-4 * t2 - .50363e-4) * t2 + .145575e-3) * t2 - .559487e-3) * t2 + .7323931e-2) * t2 + 1.000000004;
  const double q1 = t * (((((-.9173e-5 * t2 + .40658e-4) * t2 - .99941e-4) * t2 + .266891e-3) * t2 - .1601836e-2) * t2 + .093749994);
  double s0, c0;
  sincos(x - .25 * HG_PI, &s0, &c0);
  // cos(x - 3pi/4) = -sin... computed directly for fidelity with the reference
  double s1, c1;
  sincos(x - .75 * HG_PI, &s1, &c1);
  bj0 = a0 * (p0 * c0 - q0 * s0);
  by0 = a0 * (p0 * s0 + q0 * c0);
  bj1 = a0 * (p1 * c1 - q1 * s1);
  by1 = a0 * (p1 * s1 + q1 * c1);
}

// Wynn epsilon algorithm, Limes FinGrnExtSubs.f90:370-503.  s[0..n] is
// overwritten; a[] is caller scratch of n+1 entries.
HGD inline double d_limes(int n, double* s, double* a) {
  double a_max = 0.0, rl = s[n];
  for (int i = 0; i <= n; ++i) a[i] = 0.0;
  for (int k = 1;; ++k) {
    if (n - 2 * k + 1 < 0) break;
    for (int i = 0; i <= n - 2 * k + 1; ++i)
      a[i] = (s[i + 1] != s[i]) ? a[i + 1] + 1.0 / (s[i + 1] - s[i]) : a[i + 1];
    if (n - 2 * k < 0) break;
    for (int i = 0; i <= n - 2 * k; ++i) {
      s[i] = (a[i + 1] != a[i]) ? s[i + 1] + 1.0 / (a[i + 1] - a[i]) : s[i + 1];
      if (fabs(a[i]) > a_max) {
        a_max = fabs(a[i]);
        rl = s[i];
        if (s[i + 1] == s[i]) return rl;
      }
    }
  }
  return rl;
}

// Pidcock's image-source sums IMGS / DGSR / DGSZ (FinGreen3D.f90:908-1102).
HGD inline void d_imgs_all(double r, double zf, double zp, double h, double& gs, double& gr,
                                  double& gz) {
  // AMN(M,N), M = 0..4 (rows), N = 0..4
  const double AMN[5][5] = {{0.0, 0.05051418, 0.00230838, 0.00012934, 0.00000913},
                            {-0.02525711, -0.00692380, -0.00097875, -0.00010879, -0.00001270},
                            {0.00086546, 0.00073292, 0.00020597, 0.00003965, 0.00000466},
                            {-0.00004063, -0.00006636, -0.00003333, -0.00000891, 0.0},
                            {0.00000193, 0.00000398, 0.00000524, 0.0, 0.0}};
  const double t1 = r / h, t2 = (zf - zp) / h, t3 = (zf + zp + 2.0 * h) / h;
  double s1 = 0.0, s1r = 0.0, s1z = 0.0;
  for (int l = -1; l <= 1; ++l) {
    const double za = t2 + 2.0 * l, zb = t3 + 2.0 * l;
    const double ra = sqrt(t1 * t1 + za * za), rb = sqrt(t1 * t1 + zb * zb);
    const double ra3 = ra * ra * ra, rb3 = rb * rb * rb;
    s1 = s1 + 1.0 / ra + 1.0 / rb;
    s1r = s1r + t1 / ra3 + t1 / rb3;
    s1z = s1z + za / ra3 + zb / rb3;
  }
  // real powers t^(2m), t^(2m-1) as in the reference (pow with a real exponent)
  double p1[5], p2[5], p3[5], q2[5], q3[5], pr1[5];
  for (int k = 0; k < 5; ++k) {
    p1[k] = pow(t1, 2.0 * k); p2[k] = pow(t2, 2.0 * k); p3[k] = pow(t3, 2.0 * k);
    pr1[k] = k ? pow(t1, 2.0 * k - 1.0) : 0.0;
    q2[k] = k ? pow(t2, 2.0 * k - 1.0) : 0.0;
    q3[k] = k ? pow(t3, 2.0 * k - 1.0) : 0.0;
  }
  double s2 = 0.0, s2r = 0.0, s2z = 0.0;
  for (int m = 0; m <= 4; ++m)
    for (int n = 0; n <= 4; ++n) {
      const double a = AMN[m][n];
      s2 += a * p1[m] * (p2[n] + p3[n]);
      if (m >= 1) s2r += 2.0 * m * a * pr1[m] * (p2[n] + p3[n]);
      if (n >= 1) s2z += 2.0 * n * a * p1[m] * (q2[n] + q3[n]);
    }
  gs = (s1 - 2.0 + s2) / h;
  gr = (-s1r + s2r) / (h * h);
  gz = (-s1z + s2z) / (h * h);
}

// Subtraction of the Rankine pair shared by EIGEN / EIGENE / PIDCOCK.
HGD inline void d_sub_rankine(double r, double zf, double zp, double& g0, double& g1,
                                              double& g2) {
  const double sr = sqrt(r * r + (zf - zp) * (zf - zp)), sr1 = sqrt(r * r + (zf + zp) * (zf + zp));
  g0 -= (1.0 / sr + 1.0 / sr1);
  g1 += (r / sr / (sr * sr) + r / sr1 / (sr1 * sr1));
  g2 += ((zf - zp) / sr / (sr * sr) + (zf + zp) / sr1 / (sr1 * sr1));
}

struct FinState {
  double v, wk, h, nm0;  // nm0 = h/2 (1 + sinh(2 wk h)/(2 wk h))
  const double* wvn;     // roots, wvn[0] = wk
  int nk;
  int* status;
};

// Imaginary (propagating) part shared by the three series methods:
// P0 (i J0 - Y0) etc. of EIGEN/EIGENE/PIDCOCK, from the factors
// czf = cosh wk (zf + h), szf = sinh wk (zf + h), czp = cosh wk (zp + h) and
// the Bessel functions at wk r.
HGD inline void d_prop_factors(const FinState& s, double r, double czf, double szf, double czp, double j0, double j1,
                               double y0, double y1, double g[6], bool pid) {
  const double wk = s.wk, h = s.h;
  const double p0 = HG_PI / s.nm0 * czf * czp;
  // DP0 carries WK inside (PIDCOCK :601) or outside (EIGEN :317, EIGENE :442);
  // kept in the reference's order so the rounding matches.
  const double dp0 = pid ? wk * HG_PI / s.nm0 * szf * czp : wk * (HG_PI / s.nm0 * szf * czp);
  g[0] = -p0 * y0;  g[1] = p0 * j0;
  g[2] = wk * p0 * y1; g[3] = -(wk * p0) * j1;
  g[4] = -dp0 * y0; g[5] = dp0 * j0;
  if (pid) {
    g[0] += 2.0 / h * (0.5772156649015328 + log(r / 4.0 / h));
    g[2] += 2.0 / (r * h);
  }
}
HGD inline void d_prop_part(const FinState& s, double r, double zf, double zp, double g[6],
                                            bool pid) {
  const double wk = s.wk, h = s.h;
  double j0, j1, y0, y1;
  d_jy01b(wk * r, j0, j1, y0, y1);
  d_prop_factors(s, r, cosh(wk * (zf + h)), sinh(wk * (zf + h)), cosh(wk * (zp + h)), j0, j1, y0, y1, g, pid);
}

// EIGEN (R/h >= 0.5), FinGreen3D.f90:281-362.  g = [re0, im0, re1, im1, re2, im2]
HGD inline void d_eigen(const FinState& s, double r, double zf, double zp, double g[6]) {
  d_prop_part(s, r, zf, zp, g, false);
  const double h = s.h;
  for (int i = 2; i <= 10; ++i) {
    const double km = s.wvn[i - 1], tkh = 2.0 * km * h;
    const double pm = 4.0 / (1.0 + sin(tkh) / tkh) / h;
    double k0, k1, skzf, ckzf;
    d_ik01a(km * r, k0, k1);
    sincos(km * (zf + h), &skzf, &ckzf);
    const double ckzp = cos(km * (zp + h));
    const double rm1 = pm * k0 * ckzf * ckzp, rm2 = -(pm * km * k1 * ckzf * ckzp),
                 rm3 = -(pm * km * k0 * skzf * ckzp);
    g[0] += rm1; g[2] += rm2; g[4] += rm3;
    if (fabs(rm1) < SPD(1.e-6) && fabs(rm2) < SPD(1.e-6) && fabs(rm3) < SPD(1.e-6)) break;
  }
  d_sub_rankine(r, zf, zp, g[0], g[2], g[4]);
}

// EIGENE (0.05 <= R/h < 0.5), :413-506, and PIDCOCK (0.0005 <= R/h < 0.05), :558-660.
HGD inline void d_series_eps(const FinState& s, double r, double zf, double zp, double g[6],
                                    bool pid) {
  double gs[101], gr[101], gz[101], scratch[101];
  const double h = s.h, v = s.v, rhp = fabs(r / h);
  int nt = pid ? (int)(SPD(-1010.10) * rhp + SPD(100.50)) : (int)(SPD(-88.89) * rhp + SPD(54.45));
  if (nt > 101) nt = 101;
  if (nt > s.nk) nt = s.nk;
  d_prop_part(s, r, zf, zp, g, pid);
  gs[0] = 0.0; gr[0] = 0.0; gz[0] = 0.0;
  for (int i = 2; i <= nt; ++i) {
    const double um = s.wvn[i - 1];
    double k0, k1;
    d_ik01a(um * r, k0, k1);
    double su, cu;
    sincos(um * (zf + h), &su, &cu);
    const double cp = cos(um * (zp + h));
    if (!pid) {
      const double tkh = 2.0 * um * h, pm = 4.0 / (1.0 + sin(tkh) / tkh) / h;
      gs[i - 1] = gs[i - 2] + pm * k0 * cu * cp;
      gr[i - 1] = gr[i - 2] - pm * um * k1 * cu * cp;
      gz[i - 1] = gz[i - 2] - pm * um * k0 * su * cp;
    } else {
      const double umt = (i - 1) * HG_PI / h;
      double k0t, k1t, st, ct;
      d_ik01a(umt * r, k0t, k1t);
      sincos(umt * (zf + h), &st, &ct);
      const double cpt = cos(umt * (zp + h));
      const double ac = (um * um + v * v) / ((um * um + v * v) * h - v);
      const double am = ac * cu * cp, amt = ct * cpt / h;
      const double dam = -(um * ac * su * cp), damt = -(umt * st * cpt / h);
      gs[i - 1] = gs[i - 2] + (am * k0 - amt * k0t);
      gr[i - 1] = gr[i - 2] + (-(um * am * k1) + umt * amt * k1t);
      gz[i - 1] = gz[i - 2] + (dam * k0 - damt * k0t);
    }
  }
  const double l0 = d_limes(nt - 1, gs, scratch);
  const double l1 = d_limes(nt - 1, gr, scratch);
  const double l2 = d_limes(nt - 1, gz, scratch);
  if (pid) {
    double is, ir, iz;
    d_imgs_all(r, zf, zp, h, is, ir, iz);
    g[0] = g[0] + 4.0 * l0 + is;
    g[2] = g[2] + 4.0 * l1 + ir;
    g[4] = g[4] + 4.0 * l2 + iz;
  } else {
    g[0] += l0; g[2] += l1; g[4] += l2;
  }
  d_sub_rankine(r, zf, zp, g[0], g[2], g[4]);
}

// ---- Linton's method (R/h < 0.0005), FinGreen3D.f90:712-861 ----
struct LintonPar {
  double v, r, zf, zp, h;
};

// Integrands G1/G2/G3 (:1904-2057) of the deep-water-like correction.
HGD inline double d_gfun(const LintonPar& p, double t, int tag) {
  if (fabs(t) < 1.0e-8) return 0.0;
  const double val[4] = {-p.zp - p.zf, 2.0 * p.h - p.zp + p.zf, 2.0 * p.h + p.zp - p.zf,
                         4.0 * p.h + p.zp + p.zf};
  const double dval[4] = {-1.0, 1.0, -1.0, 1.0};
  double sum = 0.0;
  for (int i = 0; i < 4; ++i) {
    const double e = exp(-p.v * val[i]), arg = val[i] / 2.0 / t - p.v * t;
    if (tag == 3)
      sum = sum - p.v * dval[i] * e * d_erfcc(arg) + e * d_derfcc(arg) * dval[i] / 2.0 / t;
    else
      sum += e * d_erfcc(arg);
  }
  const double ex = exp(p.v * p.v * (t * t) - p.r * p.r / 4.0 / (t * t));
  if (tag == 2) return p.r / 2.0 / (t * t * t) * ex * sum;
  return ex * sum / t;
}
// Integrands F1/F2 (:1795-1880) of the expansion coefficients.
HGD inline double d_ffun(double r, double wvn, int no, double t, int tag) {
  if (fabs(t) < 1.0e-8) return 0.0;
  const double e = (no == 1) ? exp(-r * r / 4.0 / t + wvn * wvn * t) : exp(-r * r / 4.0 / t - wvn * wvn * t);
  return tag == 1 ? e / 4.0 / HG_PI / t : -r * e / 8.0 / HG_PI / (t * t);
}

HGD_TABLE double c_xgq[7] = {-0.949107912342759, -0.741531185599394, -0.405845151377397, 0.0,
                                0.405845151377397, 0.741531185599394, 0.949107912342759};
HGD_TABLE double c_wgq[7] = {0.129484966168870, 0.279705391489277, 0.381830050505119,
                                0.417959183673469, 0.381830050505119, 0.279705391489277,
                                0.129484966168870};
HGD_TABLE double c_xkq[15] = {-0.991455371120813, -0.949107912342759, -0.864864423359769,
                                 -0.741531185599394, -0.586087235467691, -0.405845151377397,
                                 -0.207784955007898, 0.0, 0.207784955007898, 0.405845151377397,
                                 0.586087235467691, 0.741531185599394, 0.864864423359769,
                                 0.949107912342759, 0.991455371120813};
HGD_TABLE double c_wkq[15] = {0.022935322010529, 0.063092092629979, 0.104790010322250,
                                 0.140653259715525, 0.169004726639267, 0.190350578064785,
                                 0.204432940075298, 0.209482141084728, 0.204432940075298,
                                 0.190350578064785, 0.169004726639267, 0.140653259715525,
                                 0.104790010322250, 0.063092092629979, 0.022935322010529};

// Adaptive Gauss-Kronrod 7-15 (AQUADF :2387-2532 / AQUAD :2599-2745) with an
// explicit stack: an interval is split while (200|K-G|)^1.5 > eps and it is
// wider than eps.  kind 0 integrates d_gfun(tag), kind 1 d_ffun(no, tag).
template <int KIND>
HGD inline double d_aquad(const LintonPar& lp, double r, double wvn, int no, double a, double b,
                                 double eps, int tag, int& flags) {
  const int kMaxStack = 64;
  double sa[kMaxStack], sb[kMaxStack];
  int top = 0;
  sa[0] = a; sb[0] = b; top = 1;
  double total = 0.0;
  int guard = 0;
  while (top > 0) {
    --top;
    const double aa = sa[top], bb = sb[top];
    double stf[7], gi = 0.0, gk = 0.0;
    for (int i = 0; i < 7; ++i) {
      const double t = 0.5 * (bb + aa + (bb - aa) * c_xgq[i]);
      stf[i] = KIND == 0 ? d_gfun(lp, t, tag) : d_ffun(r, wvn, no, t, tag);
      gi += c_wgq[i] * (bb - aa) / 2.0 * stf[i];
    }
    for (int i = 1; i <= 15; ++i) {
      double f;
      if (i % 2 == 0) f = stf[i / 2 - 1];
      else {
        const double t = 0.5 * (bb + aa + (bb - aa) * c_xkq[i - 1]);
        f = KIND == 0 ? d_gfun(lp, t, tag) : d_ffun(r, wvn, no, t, tag);
      }
      gk += c_wkq[i - 1] * (bb - aa) / 2.0 * f;
    }
    const double err = pow(200.0 * fabs(gk - gi), 1.5);
    if (err > eps && fabs(aa - bb) > eps && top + 2 <= kMaxStack && guard < 4096) {
      const double mid = (aa + bb) / 2.0;
      sa[top] = mid; sb[top] = bb; ++top;   // right half, popped second
      sa[top] = aa; sb[top] = mid; ++top;   // left half, popped first
    } else {
      if (err > eps && fabs(aa - bb) > eps) flags |= HG_DEV_QUAD_STACK;
      total += gk;
    }
    ++guard;
  }
  return total;
}

// SA0 / DSA0 (:1389-1524): series for the m=0 coefficient and its R-derivative.
HGD inline void d_sa0(double r, double pa, double wk, double& sa, double& dsa, int& flags) {
  const double ga = 0.5772156649015328, eps = SPD(1.e-6);
  const double x = (r / pa) * (r / pa), ex = exp(-x), lg = log(wk * r / 2.0);
  // SA0 uses E_{n+1}(x), DSA0 uses E_n(x), n = 1, 2, ...
  double e_n = d_e1xa(x);  // E_1
  double e_np1 = (ex - x * e_n) / 1.0;  // E_2
  double s = -ga - 2.0 * log(wk * pa / 2.0), ds = 0.0, sgn = -1.0, facn = 1.0, psi = 0.0;
  bool sdone = false, ddone = false;
  for (int n = 1; n <= 400; ++n) {
    psi += 1.0 / n;
    if (!sdone) {
      const double rm = sgn * pow(r / pa, 2.0 * n) / facn / n - pow(wk * pa / 2.0, 2.0 * n) / facn * e_np1 -
                        2.0 * sgn / (facn * facn) * pow(wk * r / 2.0, 2.0 * n) * (lg + ga - psi);
      s += rm;
      if (!(fabs(rm) > eps)) sdone = true;
    }
    if (!ddone) {
      const double rm = 2.0 * sgn * pow(r / pa, 2.0 * n - 1.0) / facn / pa +
                        pow(wk * pa / 2.0, 2.0 * n) / facn * e_n * 2.0 * r / (pa * pa) -
                        2.0 * sgn * n * wk / (facn * facn) * pow(wk * r / 2.0, 2.0 * n - 1.0) * (lg + ga - psi) -
                        2.0 * sgn / (facn * facn) * pow(wk * r / 2.0, 2.0 * n) / r;
      ds += rm;
      if (!(fabs(rm) > eps)) ddone = true;
    }
    if (sdone && ddone) break;
    if (n == 400) flags |= HG_DEV_SERIES_CAP;
    sgn = -sgn;
    facn *= (n + 1);
    e_n = e_np1;
    e_np1 = (ex - x * e_n) / (double)(n + 1);
  }
  sa = s / 4.0 / HG_PI;
  dsa = ds / 4.0 / HG_PI;
}

// SAM / DSAM (:1575-1693) for m >= 1.
HGD inline void d_sam(double r, double pa, double wvn, double& sa, double& dsa, int& flags) {
  const double eps = SPD(1.e-6);
  const double x = (wvn * pa / 2.0) * (wvn * pa / 2.0), ex = exp(-x);
  double e = d_e1xa(x);  // E_{n+1} for n = 0
  double s = 0.0, ds = 0.0, sgn = 1.0, facn = 1.0;
  bool sdone = false, ddone = false;
  // SAM runs n = 0,1,2,... with E_{n+1}; DSAM runs n = 1,2,... with E_{n+1}
  // and the sign/factorial of its own n.
  for (int n = 0; n <= 400; ++n) {
    if (!sdone) {
      const double rm = sgn * pow(r / pa, 2.0 * n) / facn * e;
      s += rm;
      if (!(fabs(rm) > eps)) sdone = true;
    }
    if (n >= 1 && !ddone) {
      const double rm = 2.0 * n * sgn * pow(r / pa, 2.0 * n - 1.0) / facn / pa * e;
      ds += rm;
      if (!(fabs(rm) > eps)) ddone = true;
    }
    if (sdone && ddone) break;
    if (n == 400) flags |= HG_DEV_SERIES_CAP;
    sgn = -sgn;
    facn *= (n + 1);
    e = (ex - x * e) / (double)(n + 1);
  }
  sa = s / 4.0 / HG_PI;
  dsa = ds / 4.0 / HG_PI;
}

// Splitting parameter of the method: pa = a h (a depends on v alone).
HGD inline double d_linton_a(const FinState& st) {
  const double v = st.v;
  double a;
  if (v < 0.02) a = 3324.2 * (v * v * v) - 258.89 * (v * v) + 8.3958 * v + 1.3208;
  else if (v < 0.1) a = -30.303 * (v * v * v) - 2.8138 * (v * v) + 2.7740 * v + 0.05052;
  else if (v < 1.0) a = 1.5699 * (v * v * v) - 2.5075 * (v * v) + 1.8316 * v + 0.1077;
  else a = -0.000069641 * (v * v * v) - 0.0017082 * (v * v) + 0.45566 * v + 0.80551;
  return fabs(a) / (st.wk * st.h);
}

// Term i = 1 .. 20 of the series with coefficients COEF/DCOEF (:1170-1340).
HGD inline void d_linton_term(const FinState& st, int i, double a, double r, double zf, double zp, double czf, double czp,
                              double szf, double rm[3], int& flags) {
  const double eps = SPD(1.e-6), wk = st.wk, h = st.h;
  const double pa = a * h, dnt = pa * pa / 4.0;
  double cof, dcof;
  const double km = (i == 1) ? wk : st.wvn[i - 1];
  if (i == 1) {
    if (fabs(r) < SPD(1.e-6)) {
      cof = -d_eix(wk * wk * dnt) / 4.0 / HG_PI;
      dcof = 0.0;
    } else if (r / a <= 0.5) {
      d_sa0(r, pa, wk, cof, dcof, flags);
    } else {
      double j0, j1, y0, y1;
      d_jy01b(wk * r, j0, j1, y0, y1);
      LintonPar dummy{};
      cof = -y0 / 4.0 - d_aquad<1>(dummy, r, wk, 1, 0.0, dnt, eps, 1, flags);
      dcof = wk * y1 / 4.0 - d_aquad<1>(dummy, r, wk, 1, 0.0, dnt, eps, 2, flags);
    }
  } else {
    if (fabs(r) < SPD(1.e-6)) {
      cof = d_e1xa(km * km * dnt) / 4.0 / HG_PI;
      dcof = 0.0;
    } else if (r / a <= 1.0) {
      d_sam(r, pa, km, cof, dcof, flags);
    } else {
      LintonPar dummy{};
      double p1 = dnt + 100.0;
      for (int it = 0; fabs(d_ffun(r, km, i, p1, 1)) > eps; ++it) {
        if (it > 100000) { flags |= HG_DEV_SERIES_CAP; break; }
        p1 += 100.0;
      }
      cof = d_aquad<1>(dummy, r, km, i, dnt, p1, eps, 1, flags);
      p1 = dnt + 100.0;
      for (int it = 0; fabs(d_ffun(r, km, i, p1, 2)) > eps; ++it) {
        if (it > 100000) { flags |= HG_DEV_SERIES_CAP; break; }
        p1 += 100.0;
      }
      dcof = d_aquad<1>(dummy, r, km, i, dnt, p1, eps, 2, flags);
    }
  }
  if (i == 1) {
    rm[0] = -(cof / st.nm0 * czf * czp);
    rm[1] = -(dcof / st.nm0 * czf * czp);
    rm[2] = -(cof * wk / st.nm0 * szf * czp);
  } else {
    const double nm = h / 2.0 * (1.0 + sin(2.0 * km * h) / (2.0 * km * h));
    double s1, c1;
    sincos(km * (zf + h), &s1, &c1);
    const double c2 = cos(km * (zp + h));
    rm[0] = -(cof / nm * c1 * c2);
    rm[1] = -(dcof / nm * c1 * c2);
    rm[2] = cof * km / nm * s1 * c2;
  }
}
// The series ends at the first term after the second whose parts are all small.
HGD inline bool d_linton_last(int i, const double rm[3]) {
  const double eps = SPD(1.e-6);
  return i > 2 && fabs(rm[0]) < eps && fabs(rm[1]) < eps && fabs(rm[2]) < eps;
}

// The rest of the method from the series' sums re[3] and the integrals
// q[3] over [0, pa / 2] of d_gfun's three integrands.
HGD inline void d_linton_rest(const FinState& st, double a, double r, double zf, double zp, double czf, double czp,
                              double szf, const double re[3], const double q[3], double g[6]) {
  const double v = st.v, wk = st.wk, h = st.h, pa = a * h, p4 = 4.0 * HG_PI;
  const double sr = sqrt(r * r + (zf - zp) * (zf - zp));
  const double sr1 = sqrt(r * r + (2.0 * h + zf + zp) * (2.0 * h + zf + zp));
  const double sr2 = sqrt(r * r + (zf + zp) * (zf + zp));

  // IV. error-function image sums
  double e0 = 0.0, e1 = 0.0, e2 = 0.0;
  const double val[4] = {-zp - zf, 2.0 * h - zp + zf, 2.0 * h + zp - zf, 4.0 * h + zp + zf};
  for (int i = 0; i < 4; ++i) {
    const double ro = sqrt(r * r + val[i] * val[i]);
    const double dror = r / ro, droz = val[i] * ((i % 2 == 0) ? -1.0 : 1.0) / ro;
    const double ef = d_erfcc(ro / pa), df = d_derfcc(ro / pa);
    e0 += ef / (p4 * ro);
    e1 += (df / pa * dror * ro - dror * ef) / (p4 * (ro * ro));
    e2 += (df / pa * droz * ro - droz * ef) / (p4 * (ro * ro));
  }
  const double dsr1r = r / sr1, dsr1z = (2.0 * h + zf + zp) / sr1, dsr2r = r / sr2, dsr2z = (zf + zp) / sr2;
  const double ef1 = d_erfcc(sr1 / pa), df1 = d_derfcc(sr1 / pa);
  if (fabs(sr) > SPD(1.e-6)) {
    const double dsrr = r / sr, dsrz = (zf - zp) / sr;
    const double ef = d_erfcc(sr / pa), df = d_derfcc(sr / pa);
    e0 = e0 + (ef - 1.0) / (p4 * sr) + ef1 / (p4 * sr1) - 1.0 / (p4 * sr2);
    e1 = e1 - (ef - 1.0) / (p4 * (sr * sr)) * dsrr + df / (p4 * sr * pa) * dsrr - ef1 / (p4 * (sr1 * sr1)) * dsr1r +
         df1 / (p4 * sr1 * pa) * dsr1r + dsr2r / (p4 * (sr2 * sr2));
    e2 = e2 - (ef - 1.0) / (p4 * (sr * sr)) * dsrz + df / (p4 * sr * pa) * dsrz - ef1 / (p4 * (sr1 * sr1)) * dsr1z +
         df1 / (p4 * sr1 * pa) * dsr1z + dsr2z / (p4 * (sr2 * sr2));
  } else {
    e0 = e0 + ef1 / (p4 * sr1) - 1.0 / (p4 * sr2);
    e1 = e1 - ef1 / (p4 * (sr1 * sr1)) * dsr1r + df1 / (p4 * sr1 * pa) * dsr1r + dsr2r / (p4 * (sr2 * sr2));
    e2 = e2 - ef1 / (p4 * (sr1 * sr1)) * dsr1z + df1 / (p4 * sr1 * pa) * dsr1z + dsr2z / (p4 * (sr2 * sr2));
  }

  const double re0 = re[0] - e0 - v / 2.0 / HG_PI * q[0];
  const double re1 = re[1] - e1 + v / 2.0 / HG_PI * q[1];
  const double re2 = re[2] - e2 - v / 2.0 / HG_PI * q[2];

  double bj0, bj1, by0, by1;
  d_jy01b(wk * r, bj0, bj1, by0, by1);
  const double im0 = -(bj0 * czf * czp / 4.0 / st.nm0);
  const double im1 = wk * bj1 * czf * czp / 4.0 / st.nm0;
  const double im2 = -(wk * bj0 * szf * czp / 4.0 / st.nm0);
  g[0] = -p4 * re0; g[1] = -p4 * im0;
  g[2] = -p4 * re1; g[3] = -p4 * im1;
  g[4] = -p4 * re2; g[5] = -p4 * im2;
}

HGD inline void d_linton(const FinState& st, double r, double zf, double zp, double g[6]) {
  const double eps = SPD(1.e-6), wk = st.wk, h = st.h, a = d_linton_a(st);
  const double czf = cosh(wk * (zf + h)), czp = cosh(wk * (zp + h)), szf = sinh(wk * (zf + h));
  int flags = 0;
  double re[3] = {0.0, 0.0, 0.0}, q[3];
  for (int i = 1; i <= 20; ++i) {
    double rm[3];
    d_linton_term(st, i, a, r, zf, zp, czf, czp, szf, rm, flags);
    for (int k = 0; k < 3; ++k) re[k] += rm[k];
    if (d_linton_last(i, rm)) break;
  }
  // V. integrals over [0, PA/2]
  LintonPar lp{st.v, r, zf, zp, h};
  const double pa = a * h;
  for (int k = 0; k < 3; ++k) q[k] = d_aquad<0>(lp, 0.0, 0.0, 0, 0.0, pa / 2.0, eps, k + 1, flags);
  d_linton_rest(st, a, r, zf, zp, czf, czp, szf, re, q, g);
  if (flags) hg_set_status(st.status, flags);
}

// FINGREEN3D_R dispatch (FinGreen3D.f90:160-226): the Green function minus
// its Rankine pair 1/r + 1/r1 and its derivatives, f = [G, dG/dR, dG/dzq]
// as (re, im) pairs, at horizontal distance rr, source depth zq, field depth zp.
// method: -1 by R/h as the reference; 0 LINTON, 1 PIDCOCK, 2 EIGENE, 3 EIGEN.
HGD inline void fin_regions(const FinState& st, double rr, double zq, double zp, double f[6], int method = -1) {
  if (method < 0) {
    const double rhp = fabs(rr / st.h);
    method = (rhp < 0.0005) ? 0 : (rhp < 0.05) ? 1 : (rhp < 0.5) ? 2 : 3;
  }
  if (method == 0) d_linton(st, rr, zq, zp, f);
  else if (method == 1) d_series_eps(st, rr, zq, zp, f, true);
  else if (method == 2) d_series_eps(st, rr, zq, zp, f, false);
  else d_eigen(st, rr, zq, zp, f);
  if (rr == 0.0) { f[2] = 0.0; f[3] = 0.0; }
}

// FINGREEN3D (FinGreen3D.f90:81-155) for source (xq,yq,zq) and field (xp,yp,zp).
// fpre: the region methods' result f at this pair when already known (the
// de-duplicated near pairs of the mixed form), else nullptr; the arithmetic
// around it is the same either way.
HGD inline void fin_green(const FinState& st, double xq, double yq, double zq, double xp,
                                 double yp, double zp, int flag, double2 g[4], const double* fpre = nullptr) {
  const double xpq = xq - xp, ypq = yq - yp, zpq = zq + zp;
  const double rr = sqrt(xpq * xpq + ypq * ypq);
  const double r = sqrt(rr * rr + (zp - zq) * (zp - zq));
  const double r1 = sqrt(rr * rr + zpq * zpq);
  const double ir1 = 1.0 / r1, ir13 = ir1 * ir1 * ir1, ir = 1.0 / r, ir3 = ir * ir * ir;
  g[0] = make_double2(0.0, 0.0); g[1] = g[0]; g[2] = g[0]; g[3] = g[0];
  const double v = st.v;
  if (!(fabs(v) < SPD(1.e-8)) && fabs(v + 1.0) < SPD(1.e-8)) {
    g[0].x = -ir1; g[1].x = xpq * ir13; g[2].x = ypq * ir13; g[3].x = zpq * ir13;
    if (flag == 0) { g[0].x += ir; g[1].x -= xpq * ir3; g[2].x -= ypq * ir3; g[3].x -= (zq - zp) * ir3; }
    return;
  }
  if (!(fabs(v) < SPD(1.e-8))) {
    double f[6];
    if (fpre) {
      for (int q = 0; q < 6; ++q) f[q] = fpre[q];
    } else {
      fin_regions(st, rr, zq, zp, f);
    }
    if (rr > SPD(1.e-6)) {
      const double cx = xpq / rr, cy = ypq / rr;
      g[1] = make_double2(f[2] * cx, f[3] * cx);
      g[2] = make_double2(f[2] * cy, f[3] * cy);
    }
    g[0] = make_double2(f[0], f[1]);
    g[3] = make_double2(f[4], f[5]);
  }
  g[0].x += ir1; g[1].x -= xpq * ir13; g[2].x -= ypq * ir13; g[3].x -= zpq * ir13;
  if (flag == 0) { g[0].x += ir; g[1].x -= xpq * ir3; g[2].x -= ypq * ir3; g[3].x -= (zq - zp) * ir3; }
}

}  // namespace hg
