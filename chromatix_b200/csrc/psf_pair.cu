// Passes of the fused PSF on pairs of rows and columns (see psf_pair.cuh).
#include "psf_pair.cuh"

namespace cx {

template <int NX>
static cx_status launch_psf_rows_pair(const PsfArgs& a, cudaStream_t st) {
  using C = PsfPairRows<NX>;
  auto k = k_psf_rows_pair<NX>;
  long npair = 0;
  for (int w = 0; w < a.W; ++w) npair += (a.nrows[w] + 1) / 2;
  const long items = (long)a.zc * npair;
  const int grid = persistent_grid(k, C::THREADS, C::SMEM, (items + C::TEAMS - 1) / C::TEAMS);
  k<<<grid, C::THREADS, C::SMEM, st>>>(a);
  CX_LAUNCH_CHECK();
  return CX_OK;
}

template <int NY>
static cx_status launch_psf_cols_pair(const PsfArgs& a, cudaStream_t st) {
  using C = PsfPairCols<NY>;
  auto k = k_psf_cols_pair<NY>;
  const int V = 2 * C::VP;
  const long items = (long)((a.nx + V - 1) / V) * a.zc;
  const int grid = persistent_grid(k, C::THREADS, C::SMEM, items);
  // 8-byte stores of a column pair's intensities: the fftshift keeps pairs together and aligned
  const int vec = a.nx % 4 == 0 && (reinterpret_cast<size_t>(a.out) & 7) == 0;
  k<<<grid, C::THREADS, C::SMEM, st>>>(a, vec);
  CX_LAUNCH_CHECK();
  return CX_OK;
}

cx_status psf_dispatch_rows_pair(int n, const PsfArgs& a, cudaStream_t st) {
  switch (n) {
#define CX_CASE_(N, ...) \
  case N:                \
    return launch_psf_rows_pair<N>(a, st);
    CX_PAIR_PLANS_4096(CX_CASE_)
#undef CX_CASE_
  }
  set_error("FFT length %d has no pair plan", n);
  return CX_ERR_UNSUPPORTED;
}

cx_status psf_dispatch_cols_pair(int n, const PsfArgs& a, cudaStream_t st) {
  switch (n) {
#define CX_CASE_(N, ...) \
  case N:                \
    return launch_psf_cols_pair<N>(a, st);
    CX_PAIR_PLANS_4096(CX_CASE_)
#undef CX_CASE_
  }
  set_error("FFT length %d has no pair plan", n);
  return CX_ERR_UNSUPPORTED;
}

}  // namespace cx
