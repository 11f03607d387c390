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

template <int P, bool SLAB>
static cx_status launch_conv_cols_pair(const ConvArgs& a, cudaStream_t st) {
  using C = ConvPairCols<P>;
  auto k = k_conv_cols_pair<P, SLAB>;
  const long units = (long)a.NC * a.zc;
  const int grid = persistent_grid(k, C::THREADS, C::SMEM, units < C::CTAS ? units : C::CTAS);
  k<<<grid, C::THREADS, C::SMEM, st>>>(a);
  CX_LAUNCH_CHECK();
  if constexpr (SLAB) {
    const long blocks = ((long)a.NC * P + 255) / 256, most = (long)sm_count() * 8;
    k_conv_sum<<<(int)(blocks < most ? blocks : most), 256, 0, st>>>(a, grid);
    CX_LAUNCH_CHECK();
  }
  return CX_OK;
}

int conv_pair_col_ctas(int p) {
  switch (p) {
#define CX_CASE_(N, ...) \
  case N:                \
    return ConvPairCols<N>::CTAS;
    CX_PAIR_PLANS_4096(CX_CASE_)
#undef CX_CASE_
  }
  return 0;
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
    return a.slabs > 1 ? launch_conv_cols_pair<N, true>(a, st) : launch_conv_cols_pair<N, false>(a, st);
    CX_PAIR_PLANS_4096(CX_CASE_)
#undef CX_CASE_
  }
  set_error("convolution column length %d has no pair plan", p);
  return CX_ERR_UNSUPPORTED;
}

}  // namespace cx
