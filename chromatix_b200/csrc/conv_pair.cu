// Row and column passes of the plane-wise convolution on pairs (see conv_pair.cuh).
#include "conv_pair.cuh"

namespace cx {

template <int M>
static cx_status launch_conv_rows_pair(const ConvArgs& a, cudaStream_t st) {
  using C = ConvPairRows<M>;
  auto k = k_conv_rows_pair<M>;
  const long items = (long)a.zc * (a.ldY / C::ROWS);
  k<<<persistent_grid(k, C::THREADS, C::SMEM, items), C::THREADS, C::SMEM, st>>>(a);
  CX_LAUNCH_CHECK();
  return CX_OK;
}

template <int P>
static cx_status launch_conv_cols_pair(const ConvArgs& a, cudaStream_t st) {
  using C = ConvPairCols<P>;
  auto k = k_conv_cols_pair<P>;
  k<<<persistent_grid(k, C::THREADS, C::SMEM, (long)a.NC * a.zc), C::THREADS, C::SMEM, st>>>(a);
  CX_LAUNCH_CHECK();
  return CX_OK;
}

cx_status conv_dispatch_rows_pair(int m, const ConvArgs& a, cudaStream_t st) {
  switch (m) {
#define CX_CASE_(N, ...)                                                          \
  case N:                                                                         \
    if constexpr (N <= 2048) return launch_conv_rows_pair<N>(a, st); else break;
    CX_PAIR_PLANS_4096(CX_CASE_)
#undef CX_CASE_
  }
  set_error("convolution row length %d has no pair plan", 2 * m);
  return CX_ERR_UNSUPPORTED;
}

cx_status conv_dispatch_cols_pair(int p, const ConvArgs& a, cudaStream_t st) {
  switch (p) {
#define CX_CASE_(N, ...) \
  case N:                \
    return launch_conv_cols_pair<N>(a, st);
    CX_PAIR_PLANS_4096(CX_CASE_)
#undef CX_CASE_
  }
  set_error("convolution column length %d has no pair plan", p);
  return CX_ERR_UNSUPPORTED;
}

}  // namespace cx
