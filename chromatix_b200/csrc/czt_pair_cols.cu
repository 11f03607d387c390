// Bluestein passes on pairs of vectors (see czt_pair.cuh): column tiles.
#include "czt_pair.cuh"

namespace cx {

cx_status czt_dispatch_cols_pair(int L, const CztArgs& a, cudaStream_t st) {
  // 16-byte accesses to two adjacent vectors: even strides and count, aligned buffers
  const bool vec = a.inner % 2 == 0 && a.in_ostride % 2 == 0 && a.in_estride % 2 == 0 && a.out_ostride % 2 == 0 &&
                   a.out_estride % 2 == 0 && ((reinterpret_cast<size_t>(a.x) | reinterpret_cast<size_t>(a.y)) & 15) == 0;
  switch (L) {
#define CX_CASE_(N, ...) \
  case N:                \
    return vec ? launch_czt_pair<N, true, true>(a, st) : launch_czt_pair<N, true, false>(a, st);
    CX_PAIR_PLANS(CX_CASE_)
#undef CX_CASE_
  }
  set_error("FFT length %d has no pair plan", L);
  return CX_ERR_UNSUPPORTED;
}

}  // namespace cx
