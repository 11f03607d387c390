// Bluestein passes (czt.cuh) on pairs of vectors, for FFT lengths with a pair
// plan (pair_fft.cuh).
//
// Every vector of a call has the same input and output chirps (FP64 phases):
// a CTA evaluates them once into shared memory and uses them for all of its
// pairs, where each vector evaluated its own.  Between the transforms the
// filter's spectrum is applied in one pass over shared memory.
#pragma once

#include "czt.cuh"
#include "pair_fft.cuh"

namespace cx {

// VP = 1: rows, one pair of vectors per team; else column tiles of V = 2 VP
// adjacent vectors.  Shared memory: twiddles | input chirp [L] (n <= L of it,
// then the output chirp: n + m <= L + 1) | transform buffers
template <int L, bool COLS>
struct CztPairCfg {
  static constexpr int LN = PairPlan<L>::L;
  static constexpr size_t bytes(int v) { return (size_t)v * sizeof(float4) * PairPlan<L>::R1 * (L / PairPlan<L>::R1 + 1); }
  static constexpr int vp() {
    if (!COLS) return 1;
    int v = 4;
    while (v > 1 && (v * LN > 512 || bytes(v) > (v == 2 ? 150 : 84) * 1024)) v /= 2;
    return v;
  }
  static constexpr int VP = vp();
  using F = PairFFT<L, VP>;
  static constexpr bool OWN = !COLS && LN % 32 == 0;
  static constexpr int teams() {
    if (COLS) return 1;
    int t = 128 / LN > 0 ? 128 / LN : 1;
    if (OWN && t > 15) t = 15;
    while (!OWN && (t * LN) % 32 != 0) ++t;
    return t;
  }
  static constexpr int TEAMS = teams();
  static constexpr int THREADS = TEAMS * VP * LN;
  static constexpr int TWB = (F::TW * (int)sizeof(float2) + 15) & ~15;
  static constexpr size_t BUF_OFF = TWB + ((sizeof(float2) * (size_t)(L + 1) + 15) & ~(size_t)15);
  static constexpr size_t SMEM = BUF_OFF + sizeof(float4) * (size_t)TEAMS * F::ELEMS;
  static_assert(SMEM <= 227 * 1024, "chirp-Z pair does not fit one CTA");
  static constexpr int WARPS = (THREADS + 31) / 32;
  static constexpr int MINB = SMEM > 113 * 1024 ? 1 : (16 / WARPS > 0 ? 16 / WARPS : 1);
};

// VEC: 16-byte accesses to a pair of adjacent vectors
template <int L, bool COLS, bool VEC>
__global__ void __launch_bounds__(CztPairCfg<L, COLS>::THREADS, CztPairCfg<L, COLS>::MINB) k_czt_pair(CztArgs a) {
  using C = CztPairCfg<L, COLS>;
  using F = typename C::F;
  constexpr int VP = C::VP, NB = L / F::RL;
  extern __shared__ __align__(16) char smem[];
  float2* tw = reinterpret_cast<float2*>(smem);
  float2* cin = reinterpret_cast<float2*>(smem + C::TWB);
  float2* cout = cin + a.n;
  F::load_tables(tw, a.twg, threadIdx.x, blockDim.x);
#pragma unroll 1
  for (int i = threadIdx.x; i < a.n + a.m; i += C::THREADS) cin[i] = i < a.n ? czt_in_chirp(a, i) : czt_out_chirp(a, i - a.n);
  const int team = COLS ? 0 : threadIdx.x / C::LN;
  const int c = COLS ? threadIdx.x % VP : 0;
  const int t = COLS ? threadIdx.x / VP : threadIdx.x % C::LN;
  float4* s = reinterpret_cast<float4*>(smem + C::BUF_OFF) + (size_t)team * F::ELEMS + c;
  auto sync = [&] {
    if constexpr (C::OWN) {
      asm volatile("bar.sync %0, %1;" ::"r"(1 + team), "n"(C::LN) : "memory");
    } else {
      __syncthreads();
    }
  };
  // rows: pairs of vectors v, v + 1; columns: V adjacent inner indices of one outer index
  constexpr int V = COLS ? 2 * VP : 2;
  const long n_outer = a.n_vec / a.inner;
  const int tiles_i = (a.inner + V - 1) / V;
  const long total = COLS ? (long)tiles_i * n_outer : (a.n_vec + 1) / 2;
  __syncthreads();
  for (long base = (long)blockIdx.x * C::TEAMS; base < total; base += (long)gridDim.x * C::TEAMS) {
    const bool valid = base + team < total;
    const long item = valid ? base + team : total - 1;
    const float2 *x0, *x1;
    float2 *y0, *y1;
    bool two;
    bool one = valid;
    if constexpr (COLS) {
      const long o = item / tiles_i;
      const int i = (int)(item - o * tiles_i) * V + 2 * c;
      one = i < a.inner;
      two = i + 1 < a.inner;
      x0 = a.x + o * a.in_ostride + (one ? i : 0);
      y0 = a.y + o * a.out_ostride + (one ? i : 0);
      x1 = x0 + (two ? 1 : 0);
      y1 = y0 + (two ? 1 : 0);
    } else {
      const long v0 = 2 * item, v1 = v0 + 1 < a.n_vec ? v0 + 1 : v0;
      two = valid && v1 != v0;
      const long o0 = v0 / a.inner, i0 = v0 - o0 * a.inner, o1 = v1 / a.inner, i1 = v1 - o1 * a.inner;
      x0 = a.x + o0 * a.in_ostride + i0 * a.in_istride;
      x1 = a.x + o1 * a.in_ostride + i1 * a.in_istride;
      y0 = a.y + o0 * a.out_ostride + i0 * a.out_istride;
      y1 = a.y + o1 * a.out_ostride + i1 * a.out_istride;
    }
    auto load = [&](int j) -> c2 {
      const bool ok = one && j < a.n;
      const long e = (long)j * a.in_estride;
      const c2 v = VEC ? ppack(ld4z(x0 + e, ok)) : ppack(ld2z(x0 + e, ok), ld2z(x1 + e, ok && two));
      return pmulw<false>(v, cin[j < a.n ? j : 0]);
    };
    sync();  // the previous transform has been read
    F::template first<false>(s, tw, t, load);
    F::template inner<false>(s, tw, t, sync);
    auto f = [&](int b, int r, c2 v) -> c2 { return pmulw<false>(v, a.chat[b + r * NB]); };
    F::template centre<false>(s, t, f);
    auto out = [&](int k, c2 v) {
      const int r = k - (a.n - 1);
      if (r < 0 || r >= a.m || !one) return;
      v = pmulw<false>(v, cout[r]);
      const long e = (long)r * a.out_estride;
      if constexpr (VEC) {
        *reinterpret_cast<float4*>(y0 + e) = punpack(v);
      } else {
        y0[e] = pfirst(v);
        if (two) y1[e] = psecond(v);
      }
    };
    F::template back<true>(s, tw, t, out, sync);
  }
}

template <int L, bool COLS, bool VEC>
static cx_status launch_czt_pair(const CztArgs& a, cudaStream_t st) {
  using C = CztPairCfg<L, COLS>;
  auto k = k_czt_pair<L, COLS, VEC>;
  const int V = 2 * C::VP;
  const long items = COLS ? (long)((a.inner + V - 1) / V) * (a.n_vec / a.inner) : ((a.n_vec + 1) / 2 + C::TEAMS - 1) / C::TEAMS;
  k<<<persistent_grid(k, C::THREADS, C::SMEM, items), C::THREADS, C::SMEM, st>>>(a);
  CX_LAUNCH_CHECK();
  return CX_OK;
}

}  // namespace cx
