// Row passes of the multislice loop on row pairs (see multislice_pair.cuh).
#include "multislice_pair.cuh"

namespace cx {

template <int NX, int MODE>
static cx_status launch_ms_rows_pair_mode(const MsArgs& a, cudaStream_t st) {
  using C = MsPairCfg<NX, MODE>;
  auto k = k_ms_rows_pair<NX, MODE>;
  const KernelFacts& f = kernel_facts(k, C::THREADS, C::SMEM);
  CX_CUDA_TRY(f.err);
  const int rows = MODE == MS_FINAL ? a.ny : a.py;
  // MS_LOAD follows the kernel that fills the propagator, which the next pass reads before it waits, and MS_FLUOR
  // the one that draws the phases: those two wait for their predecessor as a whole.  So does the first MS_BWD after
  // a recomputation: it copies a record before pdl_wait, and the pass that wrote it may be its predecessor.
  const bool pdl = MODE != MS_LOAD && MODE != MS_FLUOR && !(MODE == MS_BWD && a.rec_new);
  CX_CUDA_TRY(launch_kernel(k, (rows + 1) / 2, C::THREADS, C::SMEM, st, pdl, a));
  return CX_OK;
}

template <int NX>
static cx_status launch_ms_rows_pair(const MsArgs& a, cudaStream_t st) {
  switch (a.mode) {
    case MS_LOAD:
      return launch_ms_rows_pair_mode<NX, MS_LOAD>(a, st);
    case MS_FWD:
      return launch_ms_rows_pair_mode<NX, MS_FWD>(a, st);
    case MS_BWD:
      return launch_ms_rows_pair_mode<NX, MS_BWD>(a, st);
    case MS_FLUOR:
      return launch_ms_rows_pair_mode<NX, MS_FLUOR>(a, st);
    default:
      return launch_ms_rows_pair_mode<NX, MS_FINAL>(a, st);
  }
}

cx_status ms_dispatch_rows_pair(int n, const MsArgs& a, cudaStream_t st) {
  switch (n) {
#define CX_CASE_(N, ...) \
  case N:                \
    return launch_ms_rows_pair<N>(a, st);
    CX_PAIR_PLANS_4096(CX_CASE_)
#undef CX_CASE_
  }
  set_error("FFT length %d has no pair plan", n);
  return CX_ERR_UNSUPPORTED;
}

}  // namespace cx
