// Build of the finite-depth Green-function tables (hg_fintab.cuh): FP64
// evaluations of the reference's region methods (fin_regions, the method of
// the node's R segment) at the grid nodes, minus the propagating term that
// the pairs add back themselves.  Threads of a warp share a distance R_i (the
// fastest index runs along W or U), so they take the same method and series
// length.
#include "hg_fintab.cuh"
#include "hg_green.cuh"
#include "hg_kernels.cuh"
#include "hg_fin_keys_impl.cuh"

namespace hg {
namespace {

__device__ __forceinline__ void node_r(const FinTab& T, int i, double* r, int* g) {
  int s = 0;
  while (s + 1 < kFinSegs && i >= T.so[s + 1]) ++s;
  const double a = T.sa[s], b = T.sb[s], c = T.sc[s];
  const double u = (T.sn[s] > 1) ? (double)(i - T.so[s]) / (T.sn[s] - 1) : 0.0;
  *r = (c > 0.0) ? a + (b - a) * expm1(c * u) / expm1(c) : a + (b - a) * u;
  *g = s;
}

// F minus the propagating term at (R, W, U), by method g.
__device__ __forceinline__ void f_minus_prop(const FinState& fs, const FinTab& T, double r, double w, double u, int g,
                                             double out[6]) {
  const double zq = 0.5 * (u + w), zp = 0.5 * (u - w);
  double f[6], p[6];
  fin_regions(fs, r, zq, zp, f, g);
  fintab_prop<double>(fs.wk, T.pk_d, fs.h, r, zq, zp, p);
  for (int q = 0; q < 6; ++q) out[q] = f[q] - p[q];
}

// Nodes of the R segments from T.gmin on (the first i0 = T.so[T.gmin] R
// nodes are not built).
__global__ void k_fintab_build(FinState fs, FinTab T, float* __restrict__ tp, float* __restrict__ tq) {
  const int i0 = T.so[T.gmin];
  const long ntp = (long)(T.nr - i0) * T.nw, ntq = (long)(T.nr - i0) * T.nu;
  const long e = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (e >= ntp + ntq) return;
  const double h = fs.h;
  double f[6];
  float* out;
  if (e < ntp) {
    const int i = i0 + (int)(e / T.nw), j = (int)(e % T.nw);
    double r;
    int g;
    node_r(T, i, &r, &g);
    const double w = -h + (j + 0.5) * 2.0 * h / T.nw;
    f_minus_prop(fs, T, r, w, -h, g, f);
    out = tp + ((size_t)i * T.nw + j) * 8;
  } else {
    const long e2 = e - ntp;
    const int i = i0 + (int)(e2 / T.nu), k = (int)(e2 % T.nu);
    double r;
    int g;
    node_r(T, i, &r, &g);
    const double u = fmax(-(double)T.u0 * expm1((double)T.dt * (k + 0.5)), -1.98 * h);  // off the bottom image
    const double wr = 0.5 * fmin(fmin(-u, 2.0 * h + u), h);
    double f2[6];
    f_minus_prop(fs, T, r, wr, u, g, f);
    f_minus_prop(fs, T, r, wr, -h, g, f2);
    for (int q = 0; q < 6; ++q) f[q] -= f2[q];
    out = tq + ((size_t)i * T.nu + k) * 8;
  }
  for (int q = 0; q < 6; ++q) out[q] = (float)f[q];
  out[6] = 0.f;
  out[7] = 0.f;
}

// ---------------------------------------------------------------------------
// The EIGENE and EIGEN segments (gmin = 2) through the key kernels
// (hg_fin_keys.cuh): a distance R_i is shared by all nodes of its rows and
// the depths by all R_i, so the Bessel functions are tabulated once per R_i
// and the trigonometric factors once per depth, and each node's sums are
// extrapolated in shared memory.  Per R_i kNodeKeys evaluations: W_j against
// U0, then for each U_k the two of its difference.  76 000 evaluations: 6.9 ms
// with one thread per node (k_fintab_build), bound by FP64 divisions and by
// the nodes' sums in local memory.
// ---------------------------------------------------------------------------
constexpr int kNodeR = kFinSegN[2] + kFinSegN[3];
constexpr int kNodeKeys = kFinTabW + 2 * kFinTabU;
constexpr int kNodeLev = 2 * kNodeKeys;  // depths: source and field of each evaluation
constexpr int kNodeRows = 54;            // terms of the longest EIGENE series

// Scratch of the build, in doubles from the start of its buffer.
struct NodeWork {
  static constexpr size_t F = 0;
  static constexpr size_t zt = F + (size_t)6 * kNodeR * kNodeKeys;
  static constexpr size_t kt = zt + (size_t)kZRows * (kNodeLev * 6 + kTermVals) + (size_t)2 * kNodeLev;
  static constexpr size_t keys = kt + (size_t)2 * kNodeR * kNodeRows;
  static constexpr size_t jy = keys + (size_t)2 * kNodeR * kNodeKeys;
  static constexpr size_t rval = jy + (size_t)4 * kNodeR;
  static constexpr size_t zlev = rval + kNodeR;
  static constexpr size_t rnt = zlev + kNodeLev;
  static constexpr size_t total = rnt + (kNodeR + 1) / 2 + 2;
};

__device__ __forceinline__ double node_u(const FinTab& T, double h, int k) {
  return fmax(-(double)T.u0 * expm1((double)T.dt * (k + 0.5)), -1.98 * h);  // off the bottom image
}
// W and U of evaluation e of a row.
__device__ __forceinline__ void node_wu(const FinTab& T, double h, int e, double* w, double* u) {
  if (e < T.nw) {
    *w = -h + (e + 0.5) * 2.0 * h / T.nw;
    *u = -h;
  } else {
    const double uk = node_u(T, h, (e - T.nw) >> 1);
    *w = 0.5 * fmin(fmin(-uk, 2.0 * h + uk), h);
    *u = ((e - T.nw) & 1) ? -h : uk;
  }
}

__global__ void k_node_keys(FinState fs, FinTab T, double* __restrict__ rval, int* __restrict__ rnt,
                            double* __restrict__ zlev, int4* __restrict__ keys) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (e >= kNodeKeys) return;
  double r;
  int g;
  node_r(T, T.so[2] + i, &r, &g);
  int nt = 10;
  if (g == 2) {
    const double rhp = fabs(r / fs.h);
    nt = min((int)(SPD(-88.89) * rhp + SPD(54.45)), kNodeRows);
  }
  if (e == 0) {
    rval[i] = r;
    rnt[i] = nt;
  }
  if (i == 0) {
    double w, u;
    node_wu(T, fs.h, e, &w, &u);
    zlev[2 * e] = 0.5 * (u + w);
    zlev[2 * e + 1] = 0.5 * (u - w);
  }
  keys[(size_t)i * kNodeKeys + e] = make_int4(i, 2 * e, 2 * e + 1, nt);
}

// F minus the propagating term at evaluation e of row i.
__device__ __forceinline__ void node_value(const FinState& fs, const FinTab& T, double r, int i, int e,
                                           const double* __restrict__ zlev, const double* __restrict__ F, double f[6]) {
  double p[6];
  fintab_prop<double>(fs.wk, T.pk_d, fs.h, r, zlev[2 * e], zlev[2 * e + 1], p);
  const double* v = F + 6 * ((size_t)i * kNodeKeys + e);
  for (int q = 0; q < 6; ++q) f[q] = v[q] - p[q];
}

__global__ void k_node_store(FinState fs, FinTab T, const double* __restrict__ rval, const double* __restrict__ zlev,
                             const double* __restrict__ F, float* __restrict__ tp, float* __restrict__ tq) {
  const int e = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
  if (e >= T.nw + T.nu) return;
  const double r = rval[i];
  double f[6];
  float* out;
  if (e < T.nw) {
    node_value(fs, T, r, i, e, zlev, F, f);
    out = tp + ((size_t)(T.so[2] + i) * T.nw + e) * 8;
  } else {
    const int k = e - T.nw;
    double f2[6];
    node_value(fs, T, r, i, T.nw + 2 * k, zlev, F, f);
    node_value(fs, T, r, i, T.nw + 2 * k + 1, zlev, F, f2);
    for (int q = 0; q < 6; ++q) f[q] -= f2[q];
    out = tq + ((size_t)(T.so[2] + i) * T.nu + k) * 8;
  }
  for (int q = 0; q < 6; ++q) out[q] = (float)f[q];
  out[6] = 0.f;
  out[7] = 0.f;
}

cudaError_t node_build(cudaStream_t st, const FinState& fs, const FinTab& T, double* ws, float* tp, float* tq) {
  double *F = ws + NodeWork::F, *rval = ws + NodeWork::rval, *zlev = ws + NodeWork::zlev;
  int4* keys = reinterpret_cast<int4*>(ws + NodeWork::keys);
  int* rnt = reinterpret_cast<int*>(ws + NodeWork::rnt);
  double2* kt = reinterpret_cast<double2*>(ws + NodeWork::kt);
  BesselJY* jy = reinterpret_cast<BesselJY*>(ws + NodeWork::jy);
  const ZTab zt = ztab_of(ws + NodeWork::zt, kNodeLev);
  KeySegs g = {};
  g.n = 2;
  g.s[0] = KeySeg{0, kFinSegN[2], kNodeRows, 0, 0};
  g.s[1] = KeySeg{kFinSegN[2], kFinSegN[3], 9, 0, (long)kNodeRows * kFinSegN[2]};
  k_node_keys<<<dim3((kNodeKeys + 127) / 128, kNodeR), 128, 0, st>>>(fs, T, rval, rnt, zlev, keys);
  k_key_terms<1><<<1, 128, 0, st>>>(fs, zt);
  k_key_depths<1><<<dim3((kNodeLev + 127) / 128, kNodeRows), 128, 0, st>>>(fs, zlev, zt, 0);
  k_key_bessel<1><<<dim3((kNodeR + 127) / 128, kNodeRows), 128, 0, st>>>(fs, g, 0, kNodeR, rval, rnt, kt, jy);
  const int ne = kFinSegN[2] * kNodeKeys, nk = kNodeR * kNodeKeys;
  const size_t smem = (size_t)2 * (kNodeRows + 1) * kSerThreads * sizeof(double);
  const cudaError_t e =
      cudaFuncSetAttribute(k_key_series<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSerSmemMax);
  if (e != cudaSuccess) return e;
  k_key_series<1, false><<<series_blocks(ne), kSerThreads, smem, st>>>(fs, g, 0, ne, keys, zt, kt, kNodeRows, F);
  k_key_finish<1><<<(nk + 127) / 128, 128, 0, st>>>(fs, g, 0, nk, 0, ne, keys, rval, zlev, jy, zt, kt, F);
  k_node_store<<<dim3((T.nw + T.nu + 127) / 128, kNodeR), 128, 0, st>>>(fs, T, rval, zlev, F, tp, tq);
  return cudaGetLastError();
}

}  // namespace

// The tables, then (8-byte aligned: an even number of floats before it) the build's scratch.
size_t fintab_floats() { return (size_t)8 * kFinTabR * (kFinTabW + kFinTabU) + 2 * NodeWork::total; }

cudaError_t fintab_build(cudaStream_t st, const FinState& fs, double rmax, float* buf, FinTab* out, int gmin) {
  if (gmin < 0 || gmin >= kFinSegs) return cudaErrorInvalidValue;
  FinTab T = {};
  T.gmin = gmin;
  const double h = fs.h;
  T.nr = kFinTabR;
  T.nw = kFinTabW;
  T.nu = kFinTabU;
  T.h = (float)h;
  const double ends[kFinSegs + 1] = {0.0, 0.0005 * h, 0.05 * h, 0.5 * h, fmax(rmax, 0.5 * h + 1.0)};
  const double conc[kFinSegs] = {0.0, 3.0, 1.5, 1.0};
  int off = 0;
  for (int g = 0; g < kFinSegs; ++g) {
    T.sa[g] = (float)ends[g];
    T.sb[g] = (float)ends[g + 1];
    T.sc[g] = (float)conc[g];
    T.sx[g] = (float)expm1(conc[g]);
    T.so[g] = off;
    T.sn[g] = kFinSegN[g];
    off += kFinSegN[g];
  }
  T.u0 = 0.05f;
  T.dt = (float)(log1p(2.0 * h / T.u0) / (T.nu - 0.5));
  const double k0 = fs.wk;
  T.k0 = (float)k0;
  const double nm0e = 0.5 * h * exp(-2.0 * k0 * h) + (1.0 - exp(-4.0 * k0 * h)) / (8.0 * k0);  // N0 e^(-2 k0 h)
  T.pk_d = HG_PI / nm0e;
  T.pk = (float)T.pk_d;
  float* tp = buf;
  float* tq = tp + (size_t)8 * T.nr * T.nw;
  T.tp = tp;
  T.tq = tq;
  *out = T;
  if (gmin == 2)
    return node_build(st, fs, T, reinterpret_cast<double*>(buf + (size_t)8 * kFinTabR * (kFinTabW + kFinTabU)), tp, tq);
  const long total = (long)(T.nr - T.so[gmin]) * (T.nw + T.nu);
  k_fintab_build<<<(unsigned)((total + 63) / 64), 64, 0, st>>>(fs, T, tp, tq);
  return cudaGetLastError();
}

}  // namespace hg
