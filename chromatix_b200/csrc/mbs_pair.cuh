// The strided passes of the modified Born series (mbs.cuh) on column pairs,
// for axis lengths with a pair plan (pair_fft.cuh) and 16-byte aligned state.
//
// Each pass moves 1.57 GB at 320^3, 241 us at the measured copy rate.  Tiles go
// from global memory into the first stage's registers and from the last
// stage's registers back, in 64-byte row segments (8 columns), CTAs of adjacent
// tiles side by side.  The y passes take 297 us, near that rate.  The x pass
// takes 590: each tile's loads, transforms and stores follow one another, at 15
// warps per SM.
#pragma once

#include "mbs.cuh"
#include "pair_fft.cuh"

namespace cx {

// column tile of the strided passes: 4 pairs (64-byte segments), 8 where a pair has fewer than 16 lanes
template <int N, int COMPS>
struct MbsPairCfg {
  static constexpr int L = PairPlan<N>::L;
  static constexpr int VP = L < 16 && COMPS == 1 ? 8 : 4;
  using F = PairFFT<N, VP>;
  static constexpr int THREADS = VP * L;
  static constexpr int TWB = (F::TW * (int)sizeof(float2) + 15) & ~15;
  static constexpr size_t SMEM = TWB + sizeof(float4) * (size_t)COMPS * F::ELEMS;
  static constexpr int WARPS = (THREADS + 31) / 32;
  // 20 warps per SM (96 registers) for one component without a radix-16 stage, else 16 (128 registers)
  static constexpr int TARGET = COMPS == 1 && F::R1 < 16 ? 20 : 16;
  static constexpr int MINB = TARGET / WARPS > 0 ? TARGET / WARPS : 1;
  static_assert(SMEM <= 227 * 1024, "column tile does not fit one CTA");
};

template <int N, bool INV>
__global__ void __launch_bounds__(MbsPairCfg<N, 1>::THREADS, MbsPairCfg<N, 1>::MINB)
    k_mbs_cols_pair(MbsArgs a, long n_outer, int inner, long ostride, long E) {
  using C = MbsPairCfg<N, 1>;
  using F = typename C::F;
  constexpr int VP = C::VP, V = 2 * VP;
  extern __shared__ __align__(16) char smem[];
  float2* tw = reinterpret_cast<float2*>(smem);
  F::load_tables(tw, a.twg, threadIdx.x, blockDim.x);
  const int c = threadIdx.x % VP, t = threadIdx.x / VP;
  float4* s = reinterpret_cast<float4*>(smem + C::TWB) + c;
  auto sync = [] { __syncthreads(); };
  const int tiles_i = (inner + V - 1) / V;
  const long total = (long)tiles_i * n_outer;
  for (long i = blockIdx.x; i < total; i += gridDim.x) {
    const long o = i / tiles_i;
    const int col = (int)(i - o * tiles_i) * V + 2 * c;
    const bool ok = col < inner;
    float2* base = a.buf + o * ostride + col;
    auto load = [&](int j) -> c2 { return ppack(ld4z(base + (long)j * E, ok)); };
    auto out = [&](int k, c2 v) {
      if (ok) *reinterpret_cast<float4*>(base + (long)k * E) = punpack(v);
    };
    __syncthreads();  // the previous tile has been read
    F::template transform<INV>(s, tw, t, load, out, sync);
  }
}

// along x, the three components of a column pair in one CTA: FFT_x, the
// k-space projection and Green's-function division, IFFT_x
template <int N>
__global__ void __launch_bounds__(MbsPairCfg<N, 3>::THREADS, MbsPairCfg<N, 3>::MINB) k_mbs_x_pair(MbsArgs a) {
  using C = MbsPairCfg<N, 3>;
  using F = typename C::F;
  constexpr int VP = C::VP, V = 2 * VP, RL = F::RL, NB = N / RL;
  extern __shared__ __align__(16) char smem[];
  float2* tw = reinterpret_cast<float2*>(smem);
  F::load_tables(tw, a.twg, threadIdx.x, blockDim.x);
  const int c = threadIdx.x % VP, t = threadIdx.x / VP;
  float4* s[3];
#pragma unroll
  for (int m = 0; m < 3; ++m) s[m] = reinterpret_cast<float4*>(smem + C::TWB) + (size_t)m * F::ELEMS + c;
  auto sync = [] { __syncthreads(); };
  const long inner = (long)a.Y * a.Z;
  const long tiles = (inner + V - 1) / V;
  // 1 / kb2 (longitudinal part), a per-call constant
  const float bn = a.kb2.x * a.kb2.x + a.kb2.y * a.kb2.y;
  const float2 il = make_float2(a.kb2.x / bn, -a.kb2.y / bn);
  __syncthreads();
  for (long i = blockIdx.x; i < tiles; i += gridDim.x) {
    const long col = i * V + 2 * c;
    const bool ok = col < inner;
    const long cc = ok ? col : 0;
    const int iy = (int)(cc / a.Z), iz = (int)(cc - (long)iy * a.Z);  // (Z is even: a pair stays in one row)
    const float ky = a.kfy * (float)freq_index(iy, a.Y);
    const float2 kz = make_float2(a.kfz * (float)freq_index(iz, a.Z), a.kfz * (float)freq_index(iz + 1, a.Z));
    const float2 kyz = make_float2(ky * ky + kz.x * kz.x, ky * ky + kz.y * kz.y);
    __syncthreads();  // the previous tile has been read
#pragma unroll
    for (int m = 0; m < 3; ++m) {
      const float2* base = a.buf + (size_t)m * a.vox + cc;
      auto load = [&](int j) -> c2 { return ppack(ld4z(base + (long)j * inner, ok)); };
      F::template first<false>(s[0] + (size_t)m * F::ELEMS, tw, t, load);
    }
    __syncthreads();
    // inner stages of the three components between common barriers
    if constexpr (F::S >= 3) {
#pragma unroll 1
      for (int m = 0; m < 3; ++m) F::template mid2<false, false>(s[0] + (size_t)m * F::ELEMS, tw, t);
      __syncthreads();
    }
    // k-space operator on one frequency of the three components
    auto op = [&](int k, c2& y0, c2& y1, c2& y2) {
      const float kx = a.kfx * (float)freq_index(k, a.X);
      const float2 ksq = make_float2(kx * kx + kyz.x, kx * kx + kyz.y);
      // longitudinal part k (k . y) / |k|^2 (zero at k = 0)
      const float2 r = make_float2(ksq.x != 0.f ? __frcp_rn(ksq.x) : 0.f, ksq.y != 0.f ? __frcp_rn(ksq.y) : 0.f);
      c2 p = {__ffma2_rn(y2.re, kz, __ffma2_rn(y1.re, f2dup(ky), __fmul2_rn(y0.re, f2dup(kx)))),
              __ffma2_rn(y2.im, kz, __ffma2_rn(y1.im, f2dup(ky), __fmul2_rn(y0.im, f2dup(kx))))};
      p = {__fmul2_rn(p.re, r), __fmul2_rn(p.im, r)};
      // 1 / (kb2 - s ksq) = conj(dt) / |dt|^2
      const float2 dr = make_float2(a.kb2.x - a.s.x * ksq.x, a.kb2.x - a.s.x * ksq.y);
      const float2 di = make_float2(a.kb2.y - a.s.y * ksq.x, a.kb2.y - a.s.y * ksq.y);
      const float2 n2 = __ffma2_rn(di, di, __fmul2_rn(dr, dr));
      const float2 rd = make_float2(__frcp_rn(n2.x), __frcp_rn(n2.y));
      const c2 it = {__fmul2_rn(dr, rd), __fmul2_rn(di, f2neg(rd))};
      auto one = [&](c2 y, float2 kk) -> c2 {
        const c2 l = {__fmul2_rn(p.re, kk), __fmul2_rn(p.im, kk)};
        return padd(pmul(psub(y, l), it), pmulw<false>(l, il));
      };
      y0 = one(y0, f2dup(kx));
      y1 = one(y1, f2dup(ky));
      y2 = one(y2, kz);
    };
    if constexpr (RL <= 6) {
      // the three components' butterflies together in registers
#pragma unroll 1
      for (int b = t; b < NB; b += F::L) {
        c2 v[3][RL];
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          const float4* p = F::last_ptr(s[m], b);
#pragma unroll
          for (int r = 0; r < RL; ++r) v[m][r] = sload(p + r * VP);
          PDFT<RL, false>::run(v[m]);
        }
#pragma unroll
        for (int r = 0; r < RL; ++r) op(b + r * NB, v[0][r], v[1][r], v[2][r]);
#pragma unroll
        for (int m = 0; m < 3; ++m) {
          float4* p = F::last_ptr(s[m], b);
          PDFT<RL, true>::run(v[m]);
#pragma unroll
          for (int r = 0; r < RL; ++r) sstore(p + r * VP, v[m][r]);
        }
      }
    } else {
      // one component's butterfly at a time, through the buffer (each lane its own positions)
#pragma unroll 1
      for (int m = 0; m < 3; ++m) F::template last_in_place<false>(s[0] + (size_t)m * F::ELEMS, t);
#pragma unroll 1
      for (int b = t; b < NB; b += F::L) {
        const size_t off = F::last_ptr(s[0], b) - s[0];
#pragma unroll 1
        for (int r = 0; r < RL; ++r) {
          c2 y0 = sload(s[0] + off + r * VP), y1 = sload(s[1] + off + r * VP), y2 = sload(s[2] + off + r * VP);
          op(b + r * NB, y0, y1, y2);
          sstore(s[0] + off + r * VP, y0);
          sstore(s[1] + off + r * VP, y1);
          sstore(s[2] + off + r * VP, y2);
        }
      }
#pragma unroll 1
      for (int m = 0; m < 3; ++m) F::template last_in_place<true>(s[0] + (size_t)m * F::ELEMS, t);
    }
    __syncthreads();
    if constexpr (F::S >= 3) {
#pragma unroll 1
      for (int m = 0; m < 3; ++m) F::template mid2<true, true>(s[0] + (size_t)m * F::ELEMS, tw, t);
      __syncthreads();
    }
#pragma unroll 1
    for (int m = 0; m < 3; ++m) {
      float2* base = a.buf + (size_t)m * a.vox + cc;
      auto out = [&](int j, c2 v) {
        if (ok) *reinterpret_cast<float4*>(base + (long)j * inner) = punpack(v);
      };
      F::template back_last<true>(s[0] + (size_t)m * F::ELEMS, tw, t, out);
    }
    static_assert(F::S <= 3, "axis lengths up to 512 have at most three stages");
  }
}

}  // namespace cx
