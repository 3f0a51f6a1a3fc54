// Kernels of hg_fin_keys.cuh, compiled once without fused multiply-adds (plain
// form, and the mixed form's pairs below R/h = 0.05) and once with them (small
// problems of the mixed form), as the per-pair kernels are.
#pragma once
#include "hg_fill_kernel.cuh"
#include "hg_fin_keys.cuh"
#include "hg_linalg.cuh"
#include "hg_rcp.cuh"

namespace hg {
namespace {

constexpr unsigned long long kKeyEmpty = ~0ull;
constexpr int kZBits = 18;
constexpr size_t kTableBudget = (size_t)256 << 20;  // bytes of Bessel tables in flight, or as few as
constexpr size_t kTableLeast = (size_t)4 << 20;     // these where memory is short
constexpr int kMaxSegs = 16;

__device__ __forceinline__ unsigned key_hash(unsigned long long k, unsigned mask) {
  k ^= k >> 33; k *= 0xff51afd7ed558ccdull; k ^= k >> 33; k *= 0xc4ceb9fe1a85ec53ull; k ^= k >> 33;
  return (unsigned)k & mask;
}

// Slot of key in an open-addressing table of mask + 1 slots (inserted if
// absent); the table holds at most half its slots, so one is found.
__device__ __forceinline__ unsigned key_insert(unsigned long long* tab, unsigned mask, unsigned long long key) {
  unsigned s = key_hash(key, mask);
  for (unsigned probe = 0; probe <= mask; ++probe) {
    unsigned long long seen = *(volatile unsigned long long*)&tab[s];
    if (seen != key) {
      if (seen == kKeyEmpty) seen = atomicCAS(&tab[s], kKeyEmpty, key);
      if (seen != kKeyEmpty && seen != key) {
        s = (s + 1) & mask;
        continue;
      }
    }
    break;
  }
  return s;
}

// Series length of the region method at R (d_series_eps; 10 terms for EIGEN).
__device__ __forceinline__ int key_terms(double rhp) {
  if (rhp < 0.0005) return 0;
  if (rhp < 0.05) return min((int)(SPD(-1010.10) * rhp + SPD(100.50)), 101);
  if (rhp < 0.5) return (int)(SPD(-88.89) * rhp + SPD(54.45));
  return 10;
}
__device__ __forceinline__ int key_bin(double rhp) {
  if (rhp < 0.0005) return 0;
  if (rhp < 0.05) return kKeyPid0 + min(6, max(0, (100 - key_terms(rhp)) / 8));
  if (rhp < 0.5) return kKeyEps0 + min(5, max(0, (54 - key_terms(rhp)) / 8));
  return kKeyEig;
}
// Place of R inside its band, kKeySub steps: R sorted this finely, the lanes of
// a warp sum Bessel series of about one length and on one side of the branches
// at x = 9 and 18.
constexpr int kKeySub = 256;
__device__ __forceinline__ int key_sub(double rhp, int bin) {
  double t;  // 0 .. 1 over the band (bands of eight terms: see key_terms)
  if (bin == 0) t = rhp / 0.0005;
  else if (bin < kKeyEps0) t = (1010.10 * rhp - 0.5) / 8.0 - (bin - kKeyPid0);
  else if (bin < kKeyEig) t = (88.89 * rhp - 0.45) / 8.0 - (bin - kKeyEps0);
  else t = 1.0 - 0.5 / rhp;
  return bin * kKeySub + min(kKeySub - 1, max(0, (int)(t * kKeySub)));
}
// Rows (terms i = 2, 3, ...) a band's table holds: its longest series.
inline int bin_rows(int b) {
  if (b < kKeyPid0) return 0;
  if (b < kKeyEps0) return b == kKeyPid0 ? 100 : 100 - 8 * (b - kKeyPid0);
  if (b < kKeyEig) return 54 - 8 * (b - kKeyEps0);
  return 9;
}
inline int bin_width(int b) { return (b >= kKeyPid0 && b < kKeyEps0) ? 2 : 1; }  // K0, K1 pairs per term

// INSERT = false: count the near pairs; true: insert every pair's R and key
// (near_only: list the near pairs).  R as fin_green computes it.
template <int FAST, bool INSERT>
__global__ void __launch_bounds__(128)
k_key_pairs(const double* __restrict__ rec, const double* __restrict__ fx, int ldf, int n, int tn, double h, int near_only,
            const int* __restrict__ zsrc, const int* __restrict__ zfld, unsigned long long* __restrict__ tabr,
            unsigned long long* __restrict__ tabk, unsigned mask, int* __restrict__ counter, int* __restrict__ pidx,
            int* __restrict__ pslot) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y;
  bool take = false;
  double rr = 0.0;
  if (i < tn) {
    const double* pr = rec + (size_t)j * PR_SIZE;
    const double xpq = pr[PR_XQ] - fx[i], ypq = pr[PR_XQ + 1] - fx[i + ldf];
    rr = sqrt(xpq * xpq + ypq * ypq);
    take = !near_only || fabs(rr / h) < 0.05;
  }
  int at = i + j * tn;
  if (near_only) {
    const unsigned act = __ballot_sync(0xffffffffu, take);
    if (!act) return;
    const int lane = threadIdx.x & 31, leader = __ffs(act) - 1;
    int base = 0;
    if (lane == leader) base = atomicAdd(counter, __popc(act));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (!INSERT || !take) return;
    at = base + __popc(act & ((1u << lane) - 1u));
    pidx[at] = i + j * tn;
  }
  if (!INSERT || !take) return;
  const unsigned sr = key_insert(tabr, mask, (unsigned long long)__double_as_longlong(rr));
  const unsigned long long key = ((unsigned long long)sr << (2 * kZBits)) | ((unsigned long long)zsrc[j] << kZBits) |
                                 (unsigned long long)zfld[i];
  pslot[at] = (int)key_insert(tabk, mask, key);
}

// Counter of each lane's bin, one atomic per bin and warp; returns the place
// of the lane (SCATTER: the cursors advance).
__device__ __forceinline__ int bin_place(int* counters, int b) {
  const unsigned peers = __match_any_sync(__activemask(), b);
  const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
  int base = 0;
  if (lane == leader) base = atomicAdd(&counters[b], __popc(peers));
  return __shfl_sync(peers, base, leader) + __popc(peers & ((1u << lane) - 1u));
}

// Occupied R slots, counted by place in the order of R and then placed at its cursors.
template <int FAST, bool SCATTER>
__global__ void k_key_r(const unsigned long long* __restrict__ tabr, unsigned cap, double h, int* __restrict__ cursor,
                        int* __restrict__ slot2r, double* __restrict__ rval, int* __restrict__ rnt) {
  const unsigned s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= cap || tabr[s] == kKeyEmpty) return;
  const double rr = __longlong_as_double((long long)tabr[s]), rhp = fabs(rr / h);
  const int at = bin_place(cursor, key_sub(rhp, key_bin(rhp)));
  if (SCATTER) {
    slot2r[s] = at;
    rval[at] = rr;
    rnt[at] = key_terms(rhp);
  }
}

// Occupied key slots, counted by group (the piece of R their R lies in) and
// then placed at the groups' cursors.
template <int FAST, bool SCATTER>
__global__ void k_key_unique(const unsigned long long* __restrict__ tabk, unsigned cap, const int* __restrict__ slot2r,
                             const int* __restrict__ rnt, const int* __restrict__ gend, int ngroups,
                             int* __restrict__ cursor, int* __restrict__ slot2k, int4* __restrict__ keys) {
  const unsigned s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= cap || tabk[s] == kKeyEmpty) return;
  const unsigned long long key = tabk[s];
  const int r = slot2r[key >> (2 * kZBits)];
  int lo = 0, hi = ngroups - 1;  // first group whose end is beyond r
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (gend[mid] > r) hi = mid;
    else lo = mid + 1;
  }
  const int at = bin_place(cursor, lo);
  if (SCATTER) {
    slot2k[s] = at;
    const unsigned zm = (1u << kZBits) - 1u;
    keys[at] = make_int4(r, (int)((key >> kZBits) & zm), (int)(key & zm), rnt[r]);
  }
}

// Occupied key slots.
template <int FAST>
__global__ void k_key_count(const unsigned long long* __restrict__ tabk, unsigned cap, int* __restrict__ count) {
  const unsigned s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < cap && tabk[s] != kKeyEmpty) bin_place(count, 0);
}

template <int FAST>
__global__ void k_key_map(int np, int* __restrict__ pslot, const int* __restrict__ slot2k) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < np) pslot[k] = slot2k[pslot[k]];
}

// Per-depth tables, rows i - 2 of nlev entries: cos and sin of um (z + h) as a
// source and cos as a field depth, the same for umt = (i - 1) pi / h, then
// cosh and sinh of wk (z + h).
struct ZTab {
  double2* src;   // sin, cos of um (z + h)
  double2* srct;  // of umt (z + h)
  double* fld;    // cos of um (z + h)
  double* fldt;
  double2* hyp;   // cosh, sinh of wk (z + h)
  double* term;   // kTermVals per term i (row i - 2)
  int nlev;
};
constexpr int kZRows = 100;
constexpr int kTermVals = 6;  // per term: um, the EIGENE / EIGEN coefficient pm, pm um, PIDCOCK's ac, umt
size_t ztab_doubles(int nlev) { return (size_t)kZRows * nlev * 6 + (size_t)2 * nlev + (size_t)kZRows * kTermVals; }
ZTab ztab_of(double* p, int nlev) {
  const size_t row = (size_t)kZRows * nlev;
  ZTab t;
  t.src = reinterpret_cast<double2*>(p);
  t.srct = reinterpret_cast<double2*>(p + 2 * row);
  t.hyp = reinterpret_cast<double2*>(p + 4 * row);
  t.fld = p + 4 * row + 2 * (size_t)nlev;
  t.fldt = t.fld + row;
  t.term = t.fldt + row;
  t.nlev = nlev;
  return t;
}

// The two expressions of PIDCOCK's terms whose fused form matters.  The
// extrapolation turns their last bit into differences far above single
// precision, so the contracted build spells out the fused operations that the
// contracted per-pair kernel (d_series_eps) takes; the plain build rounds
// every product.
// A coefficient (um^2 + v^2) / ((um^2 + v^2) h - v):
template <int FAST>
__device__ __forceinline__ double pid_ac(double um, double v, double h) {
  if (!FAST) return (um * um + v * v) / ((um * um + v * v) * h - v);
  const double t = fma(v, v, __dmul_rn(um, um));
  return t / fma(t, h, -v);
}
// A difference a x - b y, the first product fused:
template <int FAST>
__device__ __forceinline__ double pid_diff(double a, double x, double b, double y) {
  return FAST ? fma(a, x, -__dmul_rn(b, y)) : a * x - b * y;
}

// The per-term coefficients of the series.
template <int FAST>
__global__ void k_key_terms(FinState s, ZTab t) {
  const int i = threadIdx.x + 2;
  if (i > kZRows + 1 || i > s.nk) return;
  const double um = s.wvn[i - 1], h = s.h, tkh = 2.0 * um * h, pm = 4.0 / (1.0 + sin(tkh) / tkh) / h;
  double* o = t.term + (size_t)(i - 2) * kTermVals;
  o[0] = um;
  o[1] = pm;
  o[2] = pm * um;
  o[3] = pid_ac<FAST>(um, s.v, h);
  o[4] = (i - 1) * HG_PI / h;
}

template <int FAST>
__global__ void __launch_bounds__(128)
k_key_depths(FinState s, const double* __restrict__ zlev, ZTab t, int pid) {
  const int z = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y + 2;
  if (z >= t.nlev) return;
  const double h = s.h, zf = zlev[z], wk = s.wk;
  if (i == 2) t.hyp[z] = make_double2(cosh(wk * (zf + h)), sinh(wk * (zf + h)));
  if (i > s.nk) return;
  const size_t e = (size_t)(i - 2) * t.nlev + z;
  const double um = s.wvn[i - 1];
  double su, cu;
  sincos(um * (zf + h), &su, &cu);
  t.src[e] = make_double2(su, cu);
  t.fld[e] = cos(um * (zf + h));
  if (!pid) return;
  const double umt = (i - 1) * HG_PI / h;
  sincos(umt * (zf + h), &su, &cu);
  t.srct[e] = make_double2(su, cu);
  t.fldt[e] = cos(umt * (zf + h));
}

// The pieces of R whose Bessel tables are in flight: entry (i - 2) len + r -
// r0 from base on (PIDCOCK: the second series' table follows the first's).
struct KeySeg {
  int r0, len, rows, pid;
  long base;
};
struct KeySegs {
  KeySeg s[kMaxSegs];
  int n;
};
__device__ __forceinline__ const KeySeg& seg_of(const KeySegs& g, int r) {
  int k = 0;
  while (k + 1 < g.n && r >= g.s[k].r0 + g.s[k].len) ++k;
  return g.s[k];
}

template <int FAST>
__global__ void __launch_bounds__(128)
k_key_bessel(FinState s, KeySegs g, int r0, int r1, const double* __restrict__ rval, const int* __restrict__ rnt,
             double2* __restrict__ kt, BesselJY* __restrict__ jy) {
  const int r = r0 + blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y + 2;
  if (r >= r1) return;
  const double rr = rval[r];
  if (i == 2) {
    double j0, j1, y0, y1;
    d_jy01b(s.wk * rr, j0, j1, y0, y1);
    jy[r] = BesselJY{make_double2(j0, j1), make_double2(y0, y1)};
  }
  if (i > rnt[r] || i > s.nk) return;
  const KeySeg& q = seg_of(g, r);
  const long e = q.base + (long)(i - 2) * q.len + (r - q.r0);
  const double um = s.wvn[i - 1];
  double k0, k1;
  d_ik01a(um * rr, k0, k1);
  kt[e] = make_double2(k0, k1);
  if (q.pid) {
    const double umt = (i - 1) * HG_PI / s.h;
    d_ik01a(umt * rr, k0, k1);
    kt[e + (long)q.rows * q.len] = make_double2(k0, k1);
  }
}

// U entries of the epsilon table: out(j) = old(j) + 1 / (x(j+1) - x(j)), or
// old(j) where the two agree.  The reciprocals run on the integer pipes
// (hg_rcp.cuh, the bits of the division); of the FP64 pipe's operations only
// the difference and the sum remain.  They are all formed first, without
// branches between them, and the entries out of the reciprocal's range are
// put right afterwards: a difference is zero only where the two agree (gradual
// underflow), except for equal infinities, which take the last line.
template <int U>
__device__ __forceinline__ void wynn_entries(const double* x, const double* old, double* out) {
  bool fine = true;
#pragma unroll
  for (int j = 0; j < U; ++j) {
    const double d = x[j + 1] - x[j];
    fine = fine && rcp_in_range(rcp_bits(d));
    out[j] = old[j] + rcp_rn(d);
  }
  if (fine) return;
#pragma unroll
  for (int j = 0; j < U; ++j) {
    const double d = x[j + 1] - x[j];
    const uint64_t b = rcp_bits(d);
    if (rcp_in_range(b)) continue;
    out[j] = old[j];
    if ((b << 1) != 0 && x[j + 1] != x[j]) out[j] = old[j] + 1.0 / d;
  }
}

// Limes (d_limes, hg_green.cuh) on s[0..n] and scratch a[] with stride STR,
// the a and s steps of a level in one pass: a(i) needs s(i), s(i+1) and the
// old a(i+1), s(i - 1) the new a(i - 1), a(i) and the old s(i).  U entries at a
// time: their reciprocals are independent, and with a few warps per scheduler
// (shared memory holds no more) their latency is hidden mostly by each other.
// Every level is walked in whole groups, from i = 0 (which has no s step) to
// beyond its last entry (whose surplus is formed from what lies there and
// dropped): single entries would cost a group's latency each, and short
// series are mostly ends.  |a| is compared as its bits (the order of
// non-negative doubles).
// EIGENE sums of the irregular 627-panel hull (368 k keys): 17.3 ms entry by
// entry with FP64 reciprocals, 9.1 ms four at a time with single entries at the
// ends, 5.8 ms as here with the terms' coefficients tabulated.
template <int STR>
__device__ __forceinline__ double limes_pass(int n, double* __restrict__ s, double* __restrict__ a) {
  constexpr int U = 4;
  const uint64_t kInf = 0x7ff0000000000000ull;
  uint64_t a_max = 0;
  double rl = s[n * STR];
  for (int k = 1; n - 2 * k >= 0; ++k) {
    const int last = n - 2 * k + 1;
    double sv[U + 1], an[U + 1], sn[U], ao[U];
    sv[0] = s[0];
    an[0] = 0.0;
    for (int i = 0; i <= last; i += U) {
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const int at = min(i + 1 + j, n) * STR;
        sv[j + 1] = s[at];
        ao[j] = (k == 1) ? 0.0 : a[at];
      }
      wynn_entries<U>(sv, ao, an + 1);
      wynn_entries<U>(an, sv, sn);
#pragma unroll
      for (int j = 0; j < U; ++j) {
        const int q = i + j;  // entry of a; q - 1 that of s
        if (q <= last) a[q * STR] = an[j + 1];
        if (q <= last && q > 0) {
          s[(q - 1) * STR] = sn[j];
          const uint64_t m = rcp_bits(an[j]) & ~(1ull << 63);
          if (m > a_max && m <= kInf) {
            a_max = m;
            rl = sn[j];
            if (sv[j] == sn[j]) return rl;  // the extrapolation has come to rest
          }
        }
      }
      sv[0] = sv[U];
      an[0] = an[U];
    }
  }
  return rl;
}

// x / h, correctly rounded, from rh = 1 / h correctly rounded: the first
// residual correction brings the quotient within a unit of the last place,
// the second rounds it (Markstein 1990).
__device__ __forceinline__ double div_known(double x, double h, double rh) {
  double q = x * rh;
  q = fma(fma(-q, h, x), rh, q);
  return fma(fma(-q, h, x), rh, q);
}

// One sum of one key per thread (warps of 32 keys of one sum: 0 G, 1 dG/dR,
// 2 dG/dz): partial sums into shared memory, extrapolated there into
// F[6 key + 2 sum].
constexpr int kSerThreads = 32;  // a warp per block: shared memory packs the most warps onto an SM
constexpr size_t kSerSmemSM = (size_t)227 << 10;  // an SM's shared memory
constexpr size_t kSerSmemMax = (size_t)2 * (kZRows + 1) * kSerThreads * sizeof(double);
template <int FAST, bool PID>
__global__ void __launch_bounds__(kSerThreads)
k_key_series(FinState s, KeySegs g, int k0, int k1, const int4* __restrict__ keys, ZTab t, const double2* __restrict__ kt,
             int rows, double* __restrict__ F) {
  extern __shared__ double sm[];
  const int lane = threadIdx.x & 31;
  const int task = blockIdx.x * (kSerThreads / 32) + (threadIdx.x >> 5);
  const int q = task % 3, u = k0 + (task / 3) * 32 + lane;
  if (u >= k1) return;
  double* sq = sm + threadIdx.x;
  double* sa = sm + (size_t)(rows + 1) * kSerThreads + threadIdx.x;
  const int4 key = keys[u];
  const int nt = min(key.w, s.nk);
  const KeySeg& sg = seg_of(g, key.x);
  const double2* kr = kt + sg.base + (key.x - sg.r0);
  const long kstep = sg.len, kpid = (long)sg.rows * sg.len;
  const double h = s.h, rh = 1.0 / h;
  double sum = 0.0;
  sq[0] = 0.0;
  for (int i = 2; i <= nt; ++i) {
    const double* tv = t.term + (size_t)(i - 2) * kTermVals;
    const size_t zr = (size_t)(i - 2) * t.nlev;
    const double2 kk = kr[(i - 2) * kstep];
    const double2 sc = t.src[zr + key.y];
    const double cp = t.fld[zr + key.z];
    const double k0 = kk.x, k1 = kk.y, su = sc.x, cu = sc.y;
    if (!PID) {
      if (q == 0) sum = sum + tv[1] * k0 * cu * cp;
      else if (q == 1) sum = sum - tv[2] * k1 * cu * cp;
      else sum = sum - tv[2] * k0 * su * cp;
    } else {
      const double um = tv[0], ac = tv[3], umt = tv[4];
      const double2 kkt = kr[(i - 2) * kstep + kpid];
      const double2 sct = t.srct[zr + key.y];
      const double cpt = t.fldt[zr + key.z];
      const double k0t = kkt.x, k1t = kkt.y, st = sct.x, ct = sct.y;
      if (q < 2) {
        const double am = ac * cu * cp, amt = div_known(ct * cpt, h, rh);
        if (q == 0) sum = sum + pid_diff<FAST>(am, k0, amt, k0t);
        else sum = sum + pid_diff<FAST>(umt * amt, k1t, um * am, k1);
      } else {
        const double dam = -(um * ac * su * cp), damt = -div_known(umt * st * cpt, h, rh);
        sum = sum - pid_diff<FAST>(damt, k0t, dam, k0);
      }
    }
    sq[(i - 1) * kSerThreads] = sum;
  }
  F[6 * (size_t)u + 2 * q] = limes_pass<kSerThreads>(nt - 1, sq, sa);
}

inline unsigned series_blocks(int keys) {
  return (unsigned)((((keys + 31) / 32) * 3 + kSerThreads / 32 - 1) / (kSerThreads / 32));
}

// The rest of EIGENE and PIDCOCK (d_series_eps) around the extrapolated sums,
// and EIGEN (d_eigen) whole: one key per thread.
template <int FAST>
__global__ void __launch_bounds__(128)
k_key_finish(FinState s, KeySegs g, int k0, int k1, int pid_end, int eig0, const int4* __restrict__ keys,
             const double* __restrict__ rval, const double* __restrict__ zlev, const BesselJY* __restrict__ jy, ZTab t,
             const double2* __restrict__ kt, double* __restrict__ F) {
  const int u = k0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= k1) return;
  const int4 key = keys[u];
  const double r = rval[key.x], zf = zlev[key.y], zp = zlev[key.z], h = s.h;
  const BesselJY b = jy[key.x];
  const double2 hf = t.hyp[key.y];
  const double hp = t.hyp[key.z].x;
  double gq[6];
  double* out = F + 6 * (size_t)u;
  if (u < pid_end) {
    d_prop_factors(s, r, hf.x, hf.y, hp, b.j.x, b.j.y, b.y.x, b.y.y, gq, true);
    const double l0 = out[0], l1 = out[2], l2 = out[4];
    double is, ir, iz;
    d_imgs_all(r, zf, zp, h, is, ir, iz);
    gq[0] = gq[0] + 4.0 * l0 + is;
    gq[2] = gq[2] + 4.0 * l1 + ir;
    gq[4] = gq[4] + 4.0 * l2 + iz;
  } else if (u < eig0) {
    d_prop_factors(s, r, hf.x, hf.y, hp, b.j.x, b.j.y, b.y.x, b.y.y, gq, false);
    gq[0] += out[0]; gq[2] += out[2]; gq[4] += out[4];
  } else {
    d_prop_factors(s, r, hf.x, hf.y, hp, b.j.x, b.j.y, b.y.x, b.y.y, gq, false);
    const KeySeg& sg = seg_of(g, key.x);
    const double2* kr = kt + sg.base + (key.x - sg.r0);
    for (int i = 2; i <= 10; ++i) {
      const double* tv = t.term + (size_t)(i - 2) * kTermVals;
      const size_t zr = (size_t)(i - 2) * t.nlev;
      const double2 kk = kr[(long)(i - 2) * sg.len];
      const double k0 = kk.x, k1 = kk.y;
      const double2 sc = t.src[zr + key.y];
      const double skzf = sc.x, ckzf = sc.y, ckzp = t.fld[zr + key.z];
      const double rm1 = tv[1] * k0 * ckzf * ckzp, rm2 = -(tv[2] * k1 * ckzf * ckzp),
                   rm3 = -(tv[2] * k0 * skzf * ckzp);
      gq[0] += rm1; gq[2] += rm2; gq[4] += rm3;
      if (fabs(rm1) < SPD(1.e-6) && fabs(rm2) < SPD(1.e-6) && fabs(rm3) < SPD(1.e-6)) break;
    }
  }
  d_sub_rankine(r, zf, zp, gq[0], gq[2], gq[4]);
  for (int q = 0; q < 6; ++q) out[q] = gq[q];
}

// d_aquad<0> (adaptive Gauss-Kronrod 7-15 of d_gfun) by the 16 lanes of a half
// warp: lanes 0..6 take the Gauss nodes, 7..14 the nodes the Kronrod rule
// adds, and every lane forms both sums and walks the same interval stack.
// hm: the half's lanes.
template <int FAST>
__device__ double aquad_half(const LintonPar& lp, double a, double b, double eps, int tag, unsigned hm, int& flags) {
  const int kMaxStack = 64;
  double sa[kMaxStack], sb[kMaxStack];
  const int j = threadIdx.x & 15;
  const double node = j < 7 ? c_xgq[j] : c_xkq[j < 15 ? 2 * (j - 7) : 14];
  int top = 1, guard = 0;
  sa[0] = a; sb[0] = b;
  double total = 0.0;
  while (top > 0) {
    --top;
    const double aa = sa[top], bb = sb[top];
    const double t = 0.5 * (bb + aa + (bb - aa) * node);
    const double mine = d_gfun(lp, t, tag);
    double gi = 0.0, gk = 0.0;
    for (int i = 0; i < 7; ++i) gi += c_wgq[i] * (bb - aa) / 2.0 * __shfl_sync(hm, mine, i, 16);
    for (int i = 1; i <= 15; ++i) {
      const double f = __shfl_sync(hm, mine, i % 2 == 0 ? i / 2 - 1 : 7 + (i - 1) / 2, 16);
      gk += c_wkq[i - 1] * (bb - aa) / 2.0 * f;
    }
    const double err = pow(200.0 * fabs(gk - gi), 1.5);
    if (err > eps && fabs(aa - bb) > eps && top + 2 <= kMaxStack && guard < 4096) {
      const double mid = (aa + bb) / 2.0;
      sa[top] = mid; sb[top] = bb; ++top;
      sa[top] = aa; sb[top] = mid; ++top;
    } else {
      if (err > eps && fabs(aa - bb) > eps) flags |= HG_DEV_QUAD_STACK;
      total += gk;
    }
    ++guard;
  }
  return total;
}

// LINTON keys, one per warp: few (R/h < 0.0005) and each a long serial chain
// for one thread (three adaptive quadratures of some hundred integrand values,
// each of them error functions summed as series: 8.8 ms for the 168 keys of
// the three cylinders, 19 ms for the irregular hull's 1547).  The lanes take
// the 20 terms of the series side by side and then the 15 nodes of a
// quadrature interval, the two half warps different integrals (1.8 ms for the hull); sums are formed
// in d_linton's order.
template <int FAST>
__global__ void __launch_bounds__(128)
k_key_linton(FinState s, int nk, const int4* __restrict__ keys, const double* __restrict__ rval,
             const double* __restrict__ zlev, double* __restrict__ F) {
  const int u = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (u >= nk) return;
  const int4 key = keys[u];
  const double r = rval[key.x], zf = zlev[key.y], zp = zlev[key.z], h = s.h, wk = s.wk;
  const double eps = SPD(1.e-6), a = d_linton_a(s);
  const double czf = cosh(wk * (zf + h)), czp = cosh(wk * (zp + h)), szf = sinh(wk * (zf + h));
  double rm[3] = {0.0, 0.0, 0.0};
  int mine = 0, flags = 0;
  if (lane < 20) d_linton_term(s, lane + 1, a, r, zf, zp, czf, czp, szf, rm, mine);
  __syncwarp();
  double re[3] = {0.0, 0.0, 0.0};
  for (int i = 1; i <= 20; ++i) {
    double t[3];
    for (int k = 0; k < 3; ++k) t[k] = __shfl_sync(0xffffffffu, rm[k], i - 1);
    flags |= __shfl_sync(0xffffffffu, mine, i - 1);
    for (int k = 0; k < 3; ++k) re[k] += t[k];
    if (d_linton_last(i, t)) break;
  }
  const LintonPar lp{s.v, r, zf, zp, h};
  const double pa = a * h;
  const bool low = lane < 16;
  const unsigned hm = low ? 0xffffu : 0xffff0000u;
  int qf = 0;
  const double first = aquad_half<FAST>(lp, 0.0, pa / 2.0, eps, low ? 1 : 2, hm, qf);
  const double third = low ? aquad_half<FAST>(lp, 0.0, pa / 2.0, eps, 3, hm, qf) : 0.0;
  __syncwarp();
  double q[3], g[6];
  q[0] = __shfl_sync(0xffffffffu, first, 0);
  q[1] = __shfl_sync(0xffffffffu, first, 16);
  q[2] = __shfl_sync(0xffffffffu, third, 0);
  flags |= __shfl_sync(0xffffffffu, qf, 0) | __shfl_sync(0xffffffffu, qf, 16);
  d_linton_rest(s, a, r, zf, zp, czf, czp, szf, re, q, g);
  if (r == 0.0) { g[2] = 0.0; g[3] = 0.0; }
  if (lane == 0) {
    for (int k = 0; k < 6; ++k) F[6 * (size_t)u + k] = g[k];
    if (flags) hg_set_status(s.status, flags);
  }
}

template <int FAST, typename OUT, int NM>
__global__ void __launch_bounds__(128)
k_key_fill(const double* __restrict__ rec, const double* __restrict__ fx, int ldf, int tn, long np,
           const int* __restrict__ pidx, const int* __restrict__ pkey, const double* __restrict__ F, FinState fs,
           int grn_kind, OUT* __restrict__ A, OUT* __restrict__ S, long lda, int ndiag) {
  for (long k = blockIdx.x * (long)blockDim.x + threadIdx.x; k < np; k += (long)gridDim.x * blockDim.x) {
    const int p = pidx ? pidx[k] : (int)k;
    const int i = p % tn, j = p / tn;
    fill_pair<false, OUT, NM>(rec + (size_t)j * PR_SIZE, fx[i], fx[i + ldf], fx[i + 2 * (size_t)ldf], i, j, fs, grn_kind, A, S,
                          lda, ndiag, F + 6 * (size_t)pkey[k]);
  }
}

template <typename T>
cudaError_t key_alloc(T** p, size_t count) {
  return cudaMalloc((void**)p, (count ? count : 1) * sizeof(T));
}

struct KeyScratch {  // build-time device memory, freed on every way out
  void* p[8] = {};
  int n = 0;
  ~KeyScratch() {
    for (int k = 0; k < n; ++k) cudaFree(p[k]);
  }
  template <typename T>
  cudaError_t get(T** q, size_t count) {
    const cudaError_t e = key_alloc(q, count);
    if (e == cudaSuccess) p[n++] = *q;
    return e;
  }
};

// Slots of a hash table for np keys, and the bytes of the build's scratch: two such tables and their maps, and the
// cursors of the order of R.
inline unsigned key_slots(int np) {
  unsigned cap = 4096;
  while (cap < 2u * (unsigned)np) cap <<= 1;
  return cap;
}
constexpr int kPlaces = kKeyBins * kKeySub;
inline size_t key_scratch_bytes(int np) { return (size_t)24 * key_slots(np) + 2 * sizeof(int) * (1 + kPlaces); }
// Bytes of np listed pairs, nr distances and nk keys.
inline size_t keyed_bytes(int np, int near_only, size_t nr, size_t nk) {
  return sizeof(int) * (size_t)np * (near_only ? 2 : 1) + (sizeof(double) + sizeof(int) + sizeof(BesselJY)) * nr +
         (sizeof(int4) + 6 * sizeof(double)) * nk;
}

#define KE(call)                          \
  do {                                    \
    const cudaError_t e_ = (call);        \
    if (e_ != cudaSuccess) return e_;     \
  } while (0)

template <int FAST>
cudaError_t keys_build_body(cudaStream_t st, FinKeys& K, const double* rec, const double* fx, int ldf, int n, int tn,
                            double h, int near_only, const int* zsrc, const int* zfld, int nlev) {
  KeyScratch sc;
  const dim3 g((tn + 127) / 128, n);
  double avail = K.limit;
  if (avail < 0.0) {
    size_t free_b = 0, total_b = 0;
    KE(cudaMemGetInfo(&free_b, &total_b));
    avail = (double)(free_b / 4);
  }
  int* cnt = nullptr;  // pair counter, then the cursors of the order of R
  if (avail < (double)(1 << 20)) return cudaErrorMemoryAllocation;
  KE(sc.get(&cnt, 1 + kPlaces));
  KE(cudaMemsetAsync(cnt, 0, (1 + kPlaces) * sizeof(int), st));
  K.np = (int)((long long)tn * n);
  if (near_only) {
    k_key_pairs<FAST, false><<<g, 128, 0, st>>>(rec, fx, ldf, n, tn, h, 1, zsrc, zfld, nullptr, nullptr, 0, cnt, nullptr,
                                                nullptr);
    KE(cudaMemcpyAsync(&K.np, cnt, sizeof(int), cudaMemcpyDeviceToHost, st));
    KE(cudaStreamSynchronize(st));
    KE(cudaMemsetAsync(cnt, 0, sizeof(int), st));
  }
  if (K.np == 0) return cudaSuccess;
  if (K.np > kKeyMaxPairs) return cudaErrorMemoryAllocation;
  const unsigned cap = key_slots(K.np);
  const size_t scratch = key_scratch_bytes(K.np);
  if ((double)(scratch + keyed_bytes(K.np, near_only, 0, 0)) > avail) return cudaErrorMemoryAllocation;
  unsigned long long *tabr = nullptr, *tabk = nullptr;
  int *slot2r = nullptr, *slot2k = nullptr;
  KE(sc.get(&tabr, cap));
  KE(sc.get(&tabk, cap));
  KE(sc.get(&slot2r, cap));
  KE(sc.get(&slot2k, cap));
  if (near_only) KE(key_alloc(&K.pidx, K.np));
  KE(key_alloc(&K.pkey, K.np));
  KE(cudaMemsetAsync(tabr, 0xff, (size_t)cap * sizeof(*tabr), st));
  KE(cudaMemsetAsync(tabk, 0xff, (size_t)cap * sizeof(*tabk), st));
  k_key_pairs<FAST, true><<<g, 128, 0, st>>>(rec, fx, ldf, n, tn, h, near_only, zsrc, zfld, tabr, tabk, cap - 1, cnt,
                                             K.pidx, K.pkey);
  // distinct R by band, and the number of keys
  const unsigned cb = (cap + 255) / 256;
  std::vector<int> hc(kPlaces);
  int nkeys = 0;
  KE(cudaMemsetAsync(cnt, 0, sizeof(int), st));
  k_key_count<FAST><<<cb, 256, 0, st>>>(tabk, cap, cnt);
  KE(cudaMemcpyAsync(&nkeys, cnt, sizeof(int), cudaMemcpyDeviceToHost, st));
  k_key_r<FAST, false><<<cb, 256, 0, st>>>(tabr, cap, h, cnt + 1, nullptr, nullptr, nullptr);
  KE(cudaMemcpyAsync(hc.data(), cnt + 1, kPlaces * sizeof(int), cudaMemcpyDeviceToHost, st));
  KE(cudaStreamSynchronize(st));
  int start[kKeyBins + 1] = {0};
  for (int q = 0; q < kPlaces; ++q) {
    const int c = hc[q];
    hc[q] = K.nr;
    K.nr += c;
    start[q / kKeySub + 1] = K.nr;
  }
  // What stays: pairs, R, keys and their values, the tables.  The build's scratch is gone before the tables come.
  const size_t keyed = keyed_bytes(K.np, near_only, K.nr, nkeys);
  const size_t fixed = keyed + ztab_doubles(nlev) * sizeof(double);
  size_t whole = 0;
  for (int b = 0; b < kKeyBins; ++b)
    whole += (size_t)bin_rows(b) * bin_width(b) * sizeof(double2) * (start[b + 1] - start[b]);
  const size_t least = whole < kTableLeast ? whole : kTableLeast;
  if ((double)(scratch + keyed) > avail || (double)(fixed + least) > avail) return cudaErrorMemoryAllocation;
  const size_t room = (size_t)(avail - (double)fixed), most = room < kTableBudget ? room : kTableBudget;
  K.table = whole < most ? whole : most;
  K.bytes = fixed + K.table;
  K.peak = K.bytes > scratch + keyed ? K.bytes : scratch + keyed;
  KE(key_alloc(&K.rval, K.nr));
  KE(key_alloc(&K.rnt, K.nr));
  KE(key_alloc(&K.jy, K.nr));
  KE(cudaMemcpyAsync(cnt + 1, hc.data(), kPlaces * sizeof(int), cudaMemcpyHostToDevice, st));
  k_key_r<FAST, true><<<cb, 256, 0, st>>>(tabr, cap, h, cnt + 1, slot2r, K.rval, K.rnt);
  // groups of R whose table fits the budget, and the keys in their order
  std::vector<int> gend;
  for (int b = 0; b < kKeyBins; ++b) {
    const size_t per = (size_t)bin_rows(b) * bin_width(b) * sizeof(double2);
    const int step = per ? (int)(most / per) : 1 << 30;
    for (int r = start[b]; r < start[b + 1];) {
      const int e = (step < start[b + 1] - r) ? r + step : start[b + 1];
      K.groups.push_back(KeyGroup{b, r, e, 0, 0});
      gend.push_back(e);
      r = e;
    }
  }
  const int ng = (int)gend.size();
  int *dend = nullptr, *cur = nullptr;
  KE(sc.get(&dend, ng));
  KE(sc.get(&cur, ng));
  KE(cudaMemcpyAsync(dend, gend.data(), ng * sizeof(int), cudaMemcpyHostToDevice, st));
  KE(cudaMemsetAsync(cur, 0, ng * sizeof(int), st));
  k_key_unique<FAST, false><<<cb, 256, 0, st>>>(tabk, cap, slot2r, K.rnt, dend, ng, cur, nullptr, nullptr);
  std::vector<int> kc(ng), ks(ng);
  KE(cudaMemcpyAsync(kc.data(), cur, ng * sizeof(int), cudaMemcpyDeviceToHost, st));
  KE(cudaStreamSynchronize(st));
  for (int q = 0; q < ng; ++q) {
    ks[q] = K.nk;
    K.groups[q].k0 = K.nk;
    K.nk += kc[q];
    K.groups[q].k1 = K.nk;
  }
  KE(key_alloc(&K.keys, K.nk));
  KE(key_alloc(&K.F, (size_t)6 * K.nk));
  KE(cudaMemcpyAsync(cur, ks.data(), ng * sizeof(int), cudaMemcpyHostToDevice, st));
  k_key_unique<FAST, true><<<cb, 256, 0, st>>>(tabk, cap, slot2r, K.rnt, dend, ng, cur, slot2k, K.keys);
  k_key_map<FAST><<<(K.np + 255) / 256, 256, 0, st>>>(K.np, K.pkey, slot2k);
  KE(cudaGetLastError());
  return cudaStreamSynchronize(st);
}

}  // namespace

template <int FAST>
cudaError_t fin_keys_build(cudaStream_t st, FinKeys& K, const double* rec, const double* fx, int ldf, int n, int tn,
                           double h, int near_only, const int* zsrc, const int* zfld, int nlev) {
  K.release();
  ++K.builds;
  KE(cudaGetDevice(&K.device));
  cudaError_t e = cudaErrorMemoryAllocation;
  if (keys_index(tn, n, near_only, nlev)) {
    e = keys_build_body<FAST>(st, K, rec, fx, ldf, n, tn, h, near_only, zsrc, zfld, nlev);
    if (e == cudaSuccess && K.np > 0) e = key_alloc(&K.zt, ztab_doubles(nlev));
    if (e == cudaSuccess && K.np > 0) e = key_alloc(&K.kt, K.table / sizeof(double));
  }
  if (e != cudaSuccess) {
    K.release();
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();  // the per-pair kernels run instead
  }
  K.fit = e == cudaSuccess;
  K.tn = tn;
  K.h = h;
  K.near_only = near_only;
  K.fast = FAST;
  K.nlev = nlev;
  return cudaSuccess;
}

template <int FAST, typename OUT>
cudaError_t fin_keys_fill(cudaStream_t st, FinKeys& K, const double* rec, const double* fx, int ldf, const double* zlev,
                          const FinState& fs, int grn_kind, OUT* A, OUT* S, long lda, int ndiag, const LuAux* aux) {
  K.passes = 0;
  if (K.np == 0) return cudaSuccess;
  if (aux && (!aux->side || !aux->ev_main || !aux->ev_side)) aux = nullptr;
  bool side = false;
  const ZTab zt = ztab_of(K.zt, K.nlev);
  bool any_pid = false;
  int most = 0;
  for (const KeyGroup& q : K.groups) {
    any_pid = any_pid || (q.bin >= kKeyPid0 && q.bin < kKeyEps0);
    most = bin_rows(q.bin) > most ? bin_rows(q.bin) : most;
  }
  if (most > 0) k_key_terms<FAST><<<1, 128, 0, st>>>(fs, zt);
  if (most > 0)
    k_key_depths<FAST><<<dim3((K.nlev + 127) / 128, most), 128, 0, st>>>(fs, zlev, zt, any_pid ? 1 : 0);
  size_t gi = 0;
  if (K.groups[0].bin == 0) {
    size_t ge = 0;
    while (ge < K.groups.size() && K.groups[ge].bin == 0) ++ge;
    const int nl = K.groups[ge - 1].k1;
    cudaStream_t ls = st;
    if (aux) {
      KE(cudaEventRecord(aux->ev_main, st));
      KE(cudaStreamWaitEvent(aux->side, aux->ev_main, 0));
      ls = aux->side;
      side = true;
    }
    k_key_linton<FAST><<<(nl + 3) / 4, 128, 0, ls>>>(fs, nl, K.keys, K.rval, zlev, K.F);
    if (side) KE(cudaEventRecord(aux->ev_side, ls));
    gi = ge;
  }
  while (gi < K.groups.size()) {  // as many groups at a time as the table holds
    KeySegs g = {};
    size_t used = 0;
    const size_t g0 = gi;
    int rows = 0;
    ++K.passes;
    while (gi < K.groups.size() && g.n < kMaxSegs) {
      const KeyGroup& q = K.groups[gi];
      const size_t cnt = (size_t)bin_rows(q.bin) * bin_width(q.bin) * (q.r1 - q.r0);
      if (g.n && (used + cnt) * sizeof(double2) > K.table) break;
      g.s[g.n++] = KeySeg{q.r0, q.r1 - q.r0, bin_rows(q.bin), bin_width(q.bin) == 2 ? 1 : 0, (long)used};
      used += cnt;
      rows = bin_rows(q.bin) > rows ? bin_rows(q.bin) : rows;
      ++gi;
    }
    double2* kt = reinterpret_cast<double2*>(K.kt);
    const int r0 = K.groups[g0].r0, r1 = K.groups[gi - 1].r1;
    k_key_bessel<FAST><<<dim3((r1 - r0 + 127) / 128, rows), 128, 0, st>>>(fs, g, r0, r1, K.rval, K.rnt, kt, K.jy);
    const int ka = K.groups[g0].k0, kb = K.groups[gi - 1].k1;
    int pid_end = ka, eig0 = ka;
    // Each band with the shared memory its longest series needs, so that short series run with more warps
    // on an SM; bands that fit the SMs together go in one launch, since each launch lasts at least as long
    // as its longest extrapolation (fractions of a millisecond).
    for (size_t q = g0; q < gi && K.groups[q].bin < kKeyEig;) {
      const bool pid = K.groups[q].bin < kKeyEps0;
      const int a = K.groups[q].k0, rw = bin_rows(K.groups[q].bin);
      const size_t smem = (size_t)2 * (rw + 1) * kSerThreads * sizeof(double);
      const long wave = 152L * (long)(kSerSmemSM / smem < 32 ? kSerSmemSM / smem : 32);
      int b = K.groups[q].k1;
      for (++q; q < gi && K.groups[q].bin < kKeyEig && (K.groups[q].bin < kKeyEps0) == pid; ++q) {
        if (series_blocks(K.groups[q].k1 - a) > wave) break;
        b = K.groups[q].k1;
      }
      auto kern = pid ? k_key_series<FAST, true> : k_key_series<FAST, false>;
      // the attribute is the function's, not the launch's: the same value from every thread
      KE(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSerSmemMax));
      kern<<<series_blocks(b - a), kSerThreads, smem, st>>>(fs, g, a, b, K.keys, zt, kt, rw, K.F);
      if (pid) pid_end = b;
      eig0 = b;
    }
    if (pid_end > eig0) eig0 = pid_end;
    k_key_finish<FAST><<<(kb - ka + 127) / 128, 128, 0, st>>>(fs, g, ka, kb, pid_end, eig0, K.keys, K.rval, zlev, K.jy, zt,
                                                             kt, K.F);
  }
  if (side) KE(cudaStreamWaitEvent(st, aux->ev_side, 0));
  long fb = ((long)K.np + 127) / 128;
  if (fb > 152L * 64) fb = 152L * 64;
  auto fill = k_key_fill<FAST, OUT, kNewmanRef>;
  if constexpr (sizeof(OUT) == sizeof(double2))
    if (grn_kind != 4) fill = k_key_fill<FAST, OUT, kNewmanFused>;
  fill<<<(unsigned)fb, 128, 0, st>>>(rec, fx, ldf, K.tn, K.np, K.pidx, K.pkey, K.F, fs, grn_kind, A, S, lda, ndiag);
  return cudaGetLastError();
}

}  // namespace hg
