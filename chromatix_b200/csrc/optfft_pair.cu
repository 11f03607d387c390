// Passes of the chirped optical FFT on pairs of rows and columns (see optfft_pair.cuh).
#include "optfft_pair.cuh"

namespace cx {

template <int NX>
static cx_status launch_opt_rows_pair(const float2* u, float2* T, const OptArgs& a, cudaStream_t st) {
  using C = OptPairRows<NX>;
  auto k = k_opt_rows_pair<NX>;
  const long items = (long)a.n_out_planes * ((a.py + 1) / 2);
  k<<<persistent_grid(k, C::THREADS, C::SMEM, (items + C::TEAMS - 1) / C::TEAMS), C::THREADS, C::SMEM, st>>>(u, T, a);
  CX_LAUNCH_CHECK();
  return CX_OK;
}

template <int NY, bool VEC>
static cx_status launch_opt_cols_pair(const float2* T, float2* out, const OptArgs& a, cudaStream_t st) {
  using C = OptPairCols<NY>;
  auto k = k_opt_cols_pair<NY, VEC>;
  const long items = (long)((a.px + C::V - 1) / C::V) * a.n_out_planes;
  k<<<persistent_grid(k, C::THREADS, C::SMEM, items), C::THREADS, C::SMEM, st>>>(T, out, a);
  CX_LAUNCH_CHECK();
  return CX_OK;
}

cx_status opt_dispatch_rows_pair(int n, const float2* u, float2* T, const OptArgs& a, cudaStream_t st) {
  switch (n) {
#define CX_CASE_(N, ...) \
  case N:                \
    return launch_opt_rows_pair<N>(u, T, a, st);
    CX_PAIR_PLANS_4096(CX_CASE_)
#undef CX_CASE_
  }
  set_error("FFT length %d has no pair plan", n);
  return CX_ERR_UNSUPPORTED;
}

cx_status opt_dispatch_cols_pair(int n, const float2* T, float2* out, const OptArgs& a, cudaStream_t st) {
  const bool vec = a.px % 2 == 0 && (reinterpret_cast<size_t>(T) & 15) == 0;
  switch (n) {
#define CX_CASE_(N, ...) \
  case N:                \
    return vec ? launch_opt_cols_pair<N, true>(T, out, a, st) : launch_opt_cols_pair<N, false>(T, out, a, st);
    CX_PAIR_PLANS_4096(CX_CASE_)
#undef CX_CASE_
  }
  set_error("FFT length %d has no pair plan", n);
  return CX_ERR_UNSUPPORTED;
}

}  // namespace cx
