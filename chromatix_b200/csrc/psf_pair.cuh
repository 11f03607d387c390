// The two passes of the fused PSF (psf.cuh) on pairs of pupil rows / columns,
// for every length with a pair plan (pair_fft.cuh).
#pragma once

#include "pair_fft.cuh"
#include "psf.cuh"

namespace cx {

// --------------------------------------------------------------------------
// pass A (accurate mode): rows 2 i, 2 i + 1 of one wavelength's pupil box
// --------------------------------------------------------------------------
// 640 lanes per SM (96 registers): the pass waits on its table reads and
// barriers, and a quarter more warps took it from 636 to 532 us per 64 x 3 x
// 1280^2 stack.  Variants of the first stage without the inputs outside the
// pupil box (their loads are skipped either way) measured no faster and triple the code.
// The loader is M * CX * CY: three table reads and two complex products per
// pixel pair (CX is shared by the two rows).  A box row outside the exact
// pupil is a row of zeros in M; its spectrum is stored and never read.
template <int NX>
using PsfPairRows = PairRows<NX, 128, 640>;

template <int NX>
__global__ void __launch_bounds__(PsfPairRows<NX>::THREADS, PsfPairRows<NX>::MINB) k_psf_rows_pair(PsfArgs a) {
  using C = PsfPairRows<NX>;
  using F = typename C::F;
  extern __shared__ __align__(16) char smem[];
  float2* tw = reinterpret_cast<float2*>(smem);
  F::load_tables(tw, a.twg, threadIdx.x, blockDim.x);
  const int team = threadIdx.x / C::L, t = threadIdx.x % C::L;
  float4* s = reinterpret_cast<float4*>(smem + C::TWB) + (size_t)team * F::ELEMS;
  auto sync = [&] { C::sync(team); };
  int npair = 0;  // row pairs of one plane
  for (int w = 0; w < a.W; ++w) npair += (a.nrows[w] + 1) / 2;
  const long total = (long)a.zc * npair;
  __syncthreads();
  for (long base = (long)blockIdx.x * C::TEAMS; base < total; base += (long)gridDim.x * C::TEAMS) {
    const bool valid = base + team < total;
    const long item = valid ? base + team : total - 1;
    const int zl = (int)(item / npair);
    int pr = (int)(item % npair), w = 0;
    while (w + 1 < a.W && pr >= (a.nrows[w] + 1) / 2) pr -= (a.nrows[w++] + 1) / 2;
    const int r = 2 * pr;  // box row
    const bool two = r + 1 < a.nrows[w];
    const float2* m = a.M + a.mprefix[w] + (size_t)r * a.ncols[w];
    const size_t up = two ? (size_t)a.ncols[w] : 0;
    const float2* cxz = a.CX + (size_t)(a.z0 + zl) * a.csum + a.cprefix[w];
    const float2* cyz = a.CY + (size_t)(a.z0 + zl) * a.rowsum + a.prefix[w] + r;
    const c2 cy = ppack(cyz[0], cyz[two ? 1 : 0]);
    const int xlo = a.xlo[w], nc = a.ncols[w];
    float2* dst = a.T + ((size_t)zl * a.rowsum + a.prefix[w]) * a.ldT + (size_t)r * a.rT;
    const int sh = a.shT, tile = a.nrows[w] << (sh & 15), low = (1 << sh) - 1, rT = a.rT;
    auto load = [&](int n) -> c2 {
      const int c = add_mod(n, NX / 2, NX) - xlo;  // ifftshift along x, then the box column
      const bool ok = (unsigned)c < (unsigned)nc;
      return pmul(pmulw<false>(ppack(ld2z(m + c, ok), ld2z(m + up + c, ok)), ld2z(cxz + c, ok)), cy);
    };
    auto out = [&](int k, c2 v) {
      if (valid) {
        float2* p = dst + (k >> sh) * tile + (k & low);
        p[0] = pfirst(v);
        if (two) p[rT] = psecond(v);
      }
    };
    sync();  // the pair's previous transform has been read
    F::template transform<false>(s, tw, t, load, out, sync);
  }
}

// --------------------------------------------------------------------------
// pass B: the wavelengths of one plane's column tile in turn, density |X|^2
// summed in shared memory by the lane that owns the frequency, the last
// wavelength's sum stored fftshifted
// --------------------------------------------------------------------------
// V = 2 VP columns: the widest tile of at most 256 lanes that leaves room for
// three CTAs per SM, at least 4 columns (32-byte row segments, whole sectors):
// 4 columns at 1280, 8 at 768, 16 at 256.
template <int NY>
struct PsfPairCols {
  static constexpr int L = PairPlan<NY>::L;
  static constexpr size_t bytes(int vp) {
    return (size_t)vp * (sizeof(float4) * PairPlan<NY>::R1 * (NY / PairPlan<NY>::R1 + 1) + sizeof(float2) * NY);
  }
  static constexpr int vp() {
    int v = 8;
    while (v > 2 && (v * L > 256 || bytes(v) > 75 * 1024)) v /= 2;
    return v;
  }
  static constexpr int VP = vp();
  using F = PairFFT<NY, VP>;
  static constexpr int THREADS = VP * L;
  static constexpr int TWB = (F::TW * (int)sizeof(float2) + 15) & ~15;
  static constexpr size_t ACC_OFF = TWB + sizeof(float4) * (size_t)F::ELEMS;
  static constexpr size_t SMEM = ACC_OFF + sizeof(float2) * (size_t)NY * VP;
  static constexpr int WARPS = (THREADS + 31) / 32;
  static constexpr int MINB = SMEM > 113 * 1024 ? 1 : (16 / WARPS > 0 ? 16 / WARPS : 1);
  static_assert(SMEM <= 227 * 1024, "column tile does not fit one CTA");
};

template <int NY>
__global__ void __launch_bounds__(PsfPairCols<NY>::THREADS, PsfPairCols<NY>::MINB) k_psf_cols_pair(PsfArgs a, int vec) {
  using C = PsfPairCols<NY>;
  using F = typename C::F;
  constexpr int VP = C::VP, V = 2 * VP;
  extern __shared__ __align__(16) char smem[];
  float2* tw = reinterpret_cast<float2*>(smem);
  F::load_tables(tw, a.twg, threadIdx.x, blockDim.x);
  const int c = threadIdx.x % VP, t = threadIdx.x / VP;
  float4* s = reinterpret_cast<float4*>(smem + C::TWB) + c;
  float2* acc = reinterpret_cast<float2*>(smem + C::ACC_OFF) + c;
  auto sync = [] { __syncthreads(); };
  const int tiles_x = (a.nx + V - 1) / V;
  const long total = (long)tiles_x * a.zc;
  const int rT = a.rT;
  for (long i = blockIdx.x; i < total; i += gridDim.x) {
    const int zl = (int)(i / tiles_x);
    const int x = (int)(i % tiles_x) * V + 2 * c;
    const bool ok = x < a.nx;  // (the row pitch is even: the pair's second column is readable)
    float* outz = a.out + (size_t)(a.z0 + zl) * a.ny * a.nx;
    const int xo0 = add_mod(x < a.nx ? x : 0, a.nx / 2, a.nx), xo1 = add_mod(x + 1 < a.nx ? x + 1 : 0, a.nx / 2, a.nx);
    for (int w = 0; w < a.W; ++w) {
      const float dens = (float)a.wv[w].dens;
      const int slo = support_lo(a, w), shi = support_hi(a, w);
      const float2* src = a.T + ((size_t)zl * a.rowsum + a.prefix[w]) * a.ldT - (ptrdiff_t)a.ylo[w] * a.rT +
                          (size_t)(x >> a.shT) * ((size_t)a.nrows[w] << (a.shT & 15)) + (x & ((1 << a.shT) - 1));
      auto load = [&](int n) -> c2 {
        const int y = add_mod(n, NY / 2, NY);  // ifftshift along y
        return ppack(ld4z(src + (size_t)y * rT, ok && y >= slo && y < shi));
      };
      const bool first = w == 0, last = w + 1 == a.W;
      auto out = [&](int k, c2 v) {
        float2 e = __fmul2_rn(f2dup(dens), __ffma2_rn(v.re, v.re, __fmul2_rn(v.im, v.im)));
        if (!first) e = __fadd2_rn(acc[k * VP], e);
        if (!last) {
          acc[k * VP] = e;
        } else if (ok) {
          float* p = outz + (size_t)add_mod(k, NY / 2, NY) * a.nx;  // fftshift along y
          if (vec) {
            *reinterpret_cast<float2*>(p + xo0) = e;
          } else {
            p[xo0] = e.x;
            if (x + 1 < a.nx) p[xo1] = e.y;
          }
        }
      };
      __syncthreads();  // the previous transform has been read
      F::template transform<false>(s, tw, t, load, out, sync);
    }
  }
}

}  // namespace cx
