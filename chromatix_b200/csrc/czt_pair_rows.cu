// Bluestein passes on pairs of vectors (see czt_pair.cuh): one pair per team.
#include "czt_pair.cuh"

namespace cx {

cx_status czt_dispatch_rows_pair(int L, const CztArgs& a, cudaStream_t st) {

  switch (L) {
#define CX_CASE_(N, ...) \
  case N:                \
    return launch_czt_pair<N, false, false>(a, st);
    CX_PAIR_PLANS(CX_CASE_)
#undef CX_CASE_
  }
  set_error("FFT length %d has no pair plan", L);
  return CX_ERR_UNSUPPORTED;
}

}  // namespace cx
