// Row pass of the fused PSF (see psf.cuh).
#include "pair_fft.cuh"
#include "psf.cuh"

namespace cx {

// accurate mode below the lengths with a pair plan
template <int NX>
static cx_status launch_psf_rows_tab(const PsfArgs& a, cudaStream_t st) {
  using C = PsfRowCfg<NX>;
  auto k = k_psf_rows_tab<NX>;
  const long rows = (long)a.zc * a.rowsum;
  const int grid = persistent_grid(k, C::THREADS, C::SMEM, (rows + C::TEAMS - 1) / C::TEAMS);
  k<<<grid, C::THREADS, C::SMEM, st>>>(a);
  CX_LAUNCH_CHECK();
  return CX_OK;
}

template <int NX>
static cx_status launch_psf_rows_ref32(const PsfArgs& a, cudaStream_t st) {
  using C = RowCfg<NX>;
  auto k = k_psf_rows<NX>;
  const long rows = (long)a.zc * a.rowsum;
  const int grid = persistent_grid(k, C::THREADS, C::SMEM, (rows + C::TEAMS - 1) / C::TEAMS);
  k<<<grid, C::THREADS, C::SMEM, st>>>(a);
  CX_LAUNCH_CHECK();
  return CX_OK;
}

cx_status psf_dispatch_rows(int n, const PsfArgs& a, cudaStream_t st) {
  if (a.precision == CX_PREC_REF32) {
    switch (n) {
#define CX_CASE_(N) \
  case N:           \
    return launch_psf_rows_ref32<N>(a, st);
      CX_FOR_EACH_SIZE(CX_CASE_)
#undef CX_CASE_
    }
  } else if (pair_length(n)) {
    return psf_dispatch_rows_pair(n, a, st);
  } else {
    switch (n) {
#define CX_CASE_(N) \
  case N:           \
    return launch_psf_rows_tab<N>(a, st);
      CX_FOR_EACH_SHORT_SIZE(CX_CASE_)
#undef CX_CASE_
    }
  }
  set_error("FFT length %d is not supported", n);
  return CX_ERR_UNSUPPORTED;
}

}  // namespace cx
