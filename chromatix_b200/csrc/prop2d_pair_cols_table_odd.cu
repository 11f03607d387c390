// Column pass of the Fourier-multiplier propagation on column pairs (see prop2d_pair.cuh):
// the propagator from the caller's table, rows of odd length.
#include "prop2d_pair.cuh"

namespace cx {

cx_status dispatch_cols_pair_table_odd(int n, const float2* T, float2* T2, const Prop2DArgs& a, cudaStream_t st) {
  switch (n) {
#define CX_CASE_(N, ...) \
  case N:                \
    return launch_cols_pair<N, true, false>(T, T2, a, st);
    CX_PAIR_PLANS(CX_CASE_)
#undef CX_CASE_
  }
  set_error("FFT length %d has no pair plan", n);
  return CX_ERR_UNSUPPORTED;
}

}  // namespace cx
