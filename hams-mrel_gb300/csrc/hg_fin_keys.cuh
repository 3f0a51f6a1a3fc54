// Finite-depth fill with FINGREEN3D's region methods evaluated once per
// distinct (R, zq, zp).
//
// The Green function minus its Rankine pair depends on a pair only through
// the horizontal distance R and the two depths.  Meshes repeat these triples
// bit for bit (mirror images, stacked panels, equal bodies at offsets that
// round alike), and even an irregular mesh repeats every R (the pair and its
// transpose) and every depth (a panel's whole row).  So the pairs are keyed,
// once per mesh and depth, by the bits of R as the pair kernel computes it
// and the indices of their depths, and a frequency then evaluates
//   per depth and term     the cosines and sines of the two eigenvalue series,
//   per R and term         K0, K1 of the two series, and J, Y once per R,
//   per key                the partial sums and Wynn's extrapolation,
//   per pair               the Rankine pair, the Newman integral and A, S.
// Every value comes from the same operations in the same order as the per-pair
// form (hg_green.cuh), so the results agree bit for bit.  Keys are exact:
// rounding R to share more of them changes the epsilon-extrapolated values of
// whole matrices coherently (measured: F moves to 1.2e-4).
//
// What bounds it: in the extrapolation n^2 / 2 entries per sum of n terms, three
// sums per key, each entry a reciprocal on the integer pipes (hg_rcp.cuh) and a
// difference and a sum on the FP64 pipe, whose two operations a clock and SM are
// 45 to 70 % used (shared memory holds few warps of sums); before it the FP64 pipe
// in the Bessel functions of distances and terms.  The sums run from shared
// memory, one per thread, the level pairs of the epsilon table fused into one
// pass.
#pragma once
#include <cuda_runtime.h>
#include <mutex>
#include <vector>
#include "hg_common.cuh"

namespace hg {

struct FinState;
struct LuAux;

// Bands of keys, in the order of their R: 0 LINTON, 1..7 PIDCOCK, 8..13
// EIGENE (both by series length), 14 EIGEN.
constexpr int kKeyBins = 15;
constexpr int kKeyPid0 = 1, kKeyEps0 = 8, kKeyEig = 14;
// The most the keys take: 2^27 pairs (28 bits of R slot), with near_only of those
// listed, among up to 2^31 - 1 in all, and 2^18 depths.  Where the near pairs of
// a mesh of 12096 panels in 60 m of water went pair by pair because all its
// pairs are more than 2^27, the fill took 1350 ms; keyed 91 ms.
constexpr long long kKeyMaxPairs = 1LL << 27;
constexpr int kKeyMaxLevels = 1 << 18;
// Whether the pairs of tn x n can be indexed and their depths keyed (how many
// there are to key is known after they are counted).
inline bool keys_index(int tn, int n, int near_only, int nlev) {
  const long long pairs = (long long)tn * n;
  return pairs <= (near_only ? 2147483647LL : kKeyMaxPairs) && nlev <= kKeyMaxLevels;
}

// Consecutive R (and their keys) of one band whose Bessel table fits the
// table budget.
struct KeyGroup {
  int bin, r0, r1, k0, k1;
};

struct BesselJY {
  double2 j, y;  // orders 0 and 1
};

// The keys of one mesh and depth, and the scratch their evaluation uses.  tn, h,
// near_only and fast say what they were built for; fit = false: they did not fit
// in the memory they may hold, which is not tried again for the same.
struct FinKeyData {
  int tn = -1, near_only = 0, fast = 0, nlev = 0;
  bool fit = false;
  double h = 0.0;
  int np = 0, nr = 0, nk = 0;
  int* pidx = nullptr;     // near_only: pair index i + j tn of each listed pair
  int* pkey = nullptr;     // key of each (listed) pair
  int4* keys = nullptr;    // (R index, source depth, field depth, series length)
  double* rval = nullptr;  // distinct R, grouped by band
  int* rnt = nullptr;      // series length of each R
  double* F = nullptr;     // region values, 6 per key
  double* zt = nullptr;    // per-depth tables
  double* kt = nullptr;    // Bessel tables of the groups in flight
  BesselJY* jy = nullptr;  // at wk R
  size_t table = 0;            // bytes of kt
  size_t bytes = 0, peak = 0;  // device memory held, and the most held while building
};
// Keys only save time, so an allocation of this library that fails takes all of
// the device's back (device_alloc) and is tried again: what a solve needs is there
// whether or not another context's keys came first.  mu is held while keys are
// built, evaluated (their launches queued) or given back; the list of all keys has
// a lock of its own, taken before mu and never while holding one.
struct FinKeys : FinKeyData {
  std::mutex mu;
  int device = -1;      // of the memory held
  std::vector<KeyGroup> groups;
  double limit = -1.0;  // bytes they may hold, tables and the build's scratch included; < 0: see fin_keys_build
  long builds = 0;      // builds tried
  int passes = 0;       // passes of the last evaluation over its tables
  FinKeys();
  FinKeys(const FinKeys&) = delete;
  FinKeys& operator=(const FinKeys&) = delete;
  ~FinKeys();
  void release();  // frees the device memory: no keys afterwards
};

// The most that the keys of np pairs (at most kKeyMaxPairs are keyed) over nlev
// depths can hold, the build's scratch included: every R and every key distinct.
size_t fin_keys_bound(long long np, int near_only, int nlev);

// Build the keys of the pairs (field row i < tn, source j < n): all of them, or
// with near_only those below R/h = 0.05, and everything their evaluation needs.
// K.fit = false where they do not fit into K.limit bytes (by default a quarter
// of the free device memory) or an allocation fails: the caller takes the
// per-pair kernels.
template <int FAST>
cudaError_t fin_keys_build(cudaStream_t st, FinKeys& K, const double* rec, const double* fx, int ldf, int n, int tn,
                           double h, int near_only, const int* zsrc, const int* zfld, int nlev);

// Evaluate the keys at fs and write A and S of their pairs (the others are
// left alone).  aux: a side stream for the LINTON keys, which are few and long
// (about a millisecond on a handful of SMs): they run beside the others.
template <int FAST, typename OUT>
cudaError_t fin_keys_fill(cudaStream_t st, FinKeys& K, const double* rec, const double* fx, int ldf, const double* zlev,
                          const FinState& fs, int grn_kind, OUT* A, OUT* S, long lda, int ndiag, const LuAux* aux);

}  // namespace hg
