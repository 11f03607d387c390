// Strided passes of the modified Born series on column pairs (see mbs_pair.cuh).
#include "mbs_pair.cuh"

namespace cx {

// axis lengths of the MBS grids with a pair plan
#define CX_MBS_PAIR_SIZES(X) X(128) X(160) X(192) X(224) X(256) X(320) X(384) X(448) X(512)

template <int N, bool INV>
static cx_status launch_cols_pair(const MbsArgs& a, long n_outer, int inner, long ostride, long E, cudaStream_t st) {
  using C = MbsPairCfg<N, 1>;
  auto k = k_mbs_cols_pair<N, INV>;
  const int V = 2 * C::VP;
  const long items = (long)((inner + V - 1) / V) * n_outer;
  k<<<persistent_grid(k, C::THREADS, C::SMEM, items), C::THREADS, C::SMEM, st>>>(a, n_outer, inner, ostride, E);
  CX_LAUNCH_CHECK();
  return CX_OK;
}

template <int N>
static cx_status launch_x_pair(const MbsArgs& a, cudaStream_t st) {
  using C = MbsPairCfg<N, 3>;
  auto k = k_mbs_x_pair<N>;
  const int V = 2 * C::VP;
  const long items = ((long)a.Y * a.Z + V - 1) / V;
  k<<<persistent_grid(k, C::THREADS, C::SMEM, items), C::THREADS, C::SMEM, st>>>(a);
  CX_LAUNCH_CHECK();
  return CX_OK;
}

bool mbs_on_pairs(int n, const MbsArgs& a) {
  return n >= 128 && n <= 512 && a.Z % 2 == 0 && (reinterpret_cast<size_t>(a.buf) & 15) == 0;
}

cx_status mbs_dispatch_cols_pair(int n, bool inv, const MbsArgs& a, long n_outer, int inner, long ostride, long E,
                                 cudaStream_t st) {
  switch (n) {
#define CX_CASE_(N)                                                                            \
  case N:                                                                                      \
    return inv ? launch_cols_pair<N, true>(a, n_outer, inner, ostride, E, st)                  \
               : launch_cols_pair<N, false>(a, n_outer, inner, ostride, E, st);
    CX_MBS_PAIR_SIZES(CX_CASE_)
#undef CX_CASE_
  }
  set_error("MBS grid length %d is not supported", n);
  return CX_ERR_UNSUPPORTED;
}

cx_status mbs_dispatch_x_pair(int n, const MbsArgs& a, cudaStream_t st) {
  switch (n) {
#define CX_CASE_(N) \
  case N:           \
    return launch_x_pair<N>(a, st);
    CX_MBS_PAIR_SIZES(CX_CASE_)
#undef CX_CASE_
  }
  set_error("MBS grid length %d is not supported", n);
  return CX_ERR_UNSUPPORTED;
}

}  // namespace cx
