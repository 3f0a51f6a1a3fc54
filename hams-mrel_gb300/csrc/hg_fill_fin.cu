// Finite-depth instantiations of the pair kernel.  This translation unit
// is compiled with -fmad=false: the Wynn epsilon extrapolation of the
// finite-depth series (Limes, src/FinGrnExtSubs.f90:370-503) divides by
// differences of nearly converged partial sums, so a fused multiply-add
// anywhere upstream changes its result far beyond one rounding; with
// separately rounded products the series reproduce the reference's
// arithmetic.  The mixed form, whose matrices are single precision, uses the
// instantiation of hg_fill_fin_fma.cu instead (same code, contracted).
#define HG_NO_CONTRACTION 1
#include <algorithm>
#include "hg_fin_keys_impl.cuh"

namespace hg {

// bins: device scratch of fin_bins_ints(n, tn) ints (pairs binned by cost,
// hg_fill_kernel.cuh); without it the tiled kernel runs.
template <typename OUT>
cudaError_t launch_green_fill_fin(cudaStream_t st, const double* rec, const double* fx, int ldf, int n, int tn,
                                  const FinState& fs, int grn_kind, OUT* A, OUT* S, long lda, int* status, int* bins,
                                  int ndiag) {
  if (bins) return launch_fin_binned<OUT, 0>(st, rec, fx, ldf, n, tn, fs, grn_kind, A, S, lda, bins, ndiag);
  const int cols = fill_cols(n, tn);
  dim3 grid((tn + FILL_ROWS - 1) / FILL_ROWS, (n + cols - 1) / cols);
  k_green_fill<false, OUT><<<grid, FILL_ROWS, 0, st>>>(rec, fx, ldf, n, tn, fs, grn_kind, A, S, lda, status, ndiag, cols);
  return cudaGetLastError();
}
template cudaError_t launch_green_fill_fin<double2>(cudaStream_t, const double*, const double*, int, int, int,
                                                    const FinState&, int, double2*, double2*, long, int*, int*, int);
template cudaError_t launch_green_fill_fin<float2>(cudaStream_t, const double*, const double*, int, int, int,
                                                   const FinState&, int, float2*, float2*, long, int*, int*, int);

// The pairs below R/h = 0.05 (FINGREEN3D's LINTON and PIDCOCK methods,
// FinGreen3D.f90:182-191) evaluated per pair with the reference's
// arithmetic and written over what A and S hold; the other pairs are left
// alone.  The mixed form's tabulated fill calls this after the tables:
// LINTON's adaptive quadrature and PIDCOCK's epsilon-extrapolated series
// make the reference's values in those bands jump with R and depth by far
// more than a smooth interpolation can follow, so only a per-pair
// evaluation reproduces them.
cudaError_t launch_fin_near(cudaStream_t st, const double* rec, const double* fx, int ldf, int n, int tn,
                            const FinState& fs, int grn_kind, float2* A, float2* S, long lda, int* bins, int ndiag) {
  return launch_fin_binned<float2, 0>(st, rec, fx, ldf, n, tn, fs, grn_kind, A, S, lda, bins, ndiag, kFinNearBins);
}

namespace {
// All keys of the process; never destroyed, since contexts may be closed while the process ends.
struct KeyList {
  std::mutex mu;
  std::vector<FinKeys*> v;
};
KeyList& key_list() {
  static KeyList* l = new KeyList;
  return *l;
}
}  // namespace

FinKeys::FinKeys() {
  KeyList& l = key_list();
  std::lock_guard<std::mutex> lock(l.mu);
  l.v.push_back(this);
}
FinKeys::~FinKeys() {
  {
    KeyList& l = key_list();
    std::lock_guard<std::mutex> lock(l.mu);
    l.v.erase(std::find(l.v.begin(), l.v.end(), this));
  }
  release();
}

cudaError_t device_alloc(void** p, size_t bytes) {
  cudaError_t e = cudaMalloc(p, bytes);
  if (e != cudaErrorMemoryAllocation) return e;
  cudaGetLastError();
  int dev = -1;
  bool given = false;
  if (cudaGetDevice(&dev) != cudaSuccess) return e;
  {
    KeyList& l = key_list();
    std::lock_guard<std::mutex> list(l.mu);
    for (FinKeys* K : l.v) {
      std::lock_guard<std::mutex> lock(K->mu);
      if (K->device != dev || K->bytes == 0) continue;
      const cudaError_t s = cudaDeviceSynchronize();  // evaluations still queued read them
      if (s != cudaSuccess) return s;
      // what they were built for stays noted, as not fitting
      const int tn = K->tn, near_only = K->near_only, fast = K->fast;
      const double h = K->h;
      K->release();
      K->tn = tn;
      K->h = h;
      K->near_only = near_only;
      K->fast = fast;
      given = true;
    }
  }
  if (!given) return e;
  e = cudaMalloc(p, bytes);
  if (e == cudaErrorMemoryAllocation) cudaGetLastError();
  return e;
}

size_t fin_keys_bound(long long pairs, int near_only, int nlev) {
  if (pairs <= 0 || nlev > kKeyMaxLevels) return 0;
  const int np = (int)(pairs < kKeyMaxPairs ? pairs : kKeyMaxPairs);
  size_t row = 0;  // table bytes of one R in the band with the longest series
  for (int b = 0; b < kKeyBins; ++b) row = std::max(row, (size_t)bin_rows(b) * bin_width(b) * sizeof(double2));
  const size_t keyed = keyed_bytes(np, near_only, np, np), table = std::min(kTableBudget, row * (size_t)np);
  return std::max(keyed + key_scratch_bytes(np), keyed + ztab_doubles(nlev) * sizeof(double) + table);
}

void FinKeys::release() {
  void* bufs[] = {pidx, pkey, keys, rval, rnt, F, zt, kt, jy};
  for (void* b : bufs)
    if (b) cudaFree(b);
  static_cast<FinKeyData&>(*this) = FinKeyData();
  groups.clear();
}
template cudaError_t fin_keys_build<0>(cudaStream_t, FinKeys&, const double*, const double*, int, int, int, double, int,
                                       const int*, const int*, int);
template cudaError_t fin_keys_fill<0, double2>(cudaStream_t, FinKeys&, const double*, const double*, int, const double*,
                                               const FinState&, int, double2*, double2*, long, int, const LuAux*);
template cudaError_t fin_keys_fill<0, float2>(cudaStream_t, FinKeys&, const double*, const double*, int, const double*,
                                              const FinState&, int, float2*, float2*, long, int, const LuAux*);

cudaError_t launch_green_points_fin(cudaStream_t st, int npts, const double* pts, const int* flags, const FinState& fs,
                                    double* out) {
  k_green_points<false><<<(npts + 63) / 64, 64, 0, st>>>(npts, pts, flags, fs, out);
  return cudaGetLastError();
}

}  // namespace hg
