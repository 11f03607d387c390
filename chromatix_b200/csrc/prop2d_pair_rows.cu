// Row passes of the Fourier-multiplier propagation on row pairs (see prop2d_pair.cuh).
#include "prop2d_pair.cuh"

namespace cx {

template <int NX>
static cx_status launch_rows_fwd_pair(const float2* u, float2* T, const Prop2DArgs& a, cudaStream_t st) {
  using C = PairRows<NX>;
  auto k = k_prop_rows_fwd_pair<NX>;
  const long items = (long)a.n_in_planes * ((a.ny + 1) / 2);
  const int grid = persistent_grid(k, C::THREADS, C::SMEM, (items + C::TEAMS - 1) / C::TEAMS);
  k<<<grid, C::THREADS, C::SMEM, st>>>(u, T, a);
  CX_LAUNCH_CHECK();
  return CX_OK;
}

template <int NX>
static cx_status launch_rows_inv_pair(const float2* T2, float2* out, const Prop2DArgs& a, cudaStream_t st) {
  using C = PairRows<NX>;
  auto k = k_prop_rows_inv_pair<NX>;
  const long items = (long)a.n_out_planes * ((a.out_ny + 1) / 2);
  const int grid = persistent_grid(k, C::THREADS, C::SMEM, (items + C::TEAMS - 1) / C::TEAMS);
  k<<<grid, C::THREADS, C::SMEM, st>>>(T2, out, a);
  CX_LAUNCH_CHECK();
  return CX_OK;
}

cx_status dispatch_rows_fwd_pair(int n, const float2* u, float2* T, const Prop2DArgs& a, cudaStream_t st) {
  switch (n) {
#define CX_CASE_(N, ...) \
  case N:                \
    return launch_rows_fwd_pair<N>(u, T, a, st);
    CX_PAIR_PLANS(CX_CASE_)
#undef CX_CASE_
  }
  set_error("FFT length %d has no pair plan", n);
  return CX_ERR_UNSUPPORTED;
}

cx_status dispatch_rows_inv_pair(int n, const float2* T2, float2* out, const Prop2DArgs& a, cudaStream_t st) {
  switch (n) {
#define CX_CASE_(N, ...) \
  case N:                \
    return launch_rows_inv_pair<N>(T2, out, a, st);
    CX_PAIR_PLANS(CX_CASE_)
#undef CX_CASE_
  }
  set_error("FFT length %d has no pair plan", n);
  return CX_ERR_UNSUPPORTED;
}

}  // namespace cx
