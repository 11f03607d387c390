// The two passes of the chirped optical FFT (optfft.cuh) on pairs of rows /
// columns, for every length with a pair plan (pair_fft.cuh).
//
// A plane without chirp and pupil (ff_lens, optical_fft and their adjoints)
// goes straight from global memory into the first stage's registers and from
// the last stage's registers to the shifted output.  Chirps and pupils (FP64
// per element) run in a loop over the buffer instead, before the first or
// after the last stage, so that their code is emitted once.
#pragma once

#include "optfft.cuh"
#include "pair_fft.cuh"

namespace cx {

template <int NX>
using OptPairRows = PairRows<NX>;

template <int NX>
__global__ void __launch_bounds__(OptPairRows<NX>::THREADS, OptPairRows<NX>::MINB)
    k_opt_rows_pair(const float2* __restrict__ u, float2* __restrict__ T, OptArgs a) {
  using C = OptPairRows<NX>;
  using F = typename C::F;
  extern __shared__ __align__(16) char smem[];
  float2* tw = reinterpret_cast<float2*>(smem);
  F::load_tables(tw, a.twg, threadIdx.x, blockDim.x);
  const int team = threadIdx.x / C::L, t = threadIdx.x % C::L;
  float4* s = reinterpret_cast<float4*>(smem + C::TWB) + (size_t)team * F::ELEMS;
  auto sync = [&] { C::sync(team); };
  // FFT rows 2 i, 2 i + 1 of one plane; the planes of one field (its wavelengths) run fastest
  const int npair = (a.py + 1) / 2;
  const long total = (long)a.n_out_planes * npair;
  __syncthreads();
  for (long base = (long)blockIdx.x * C::TEAMS; base < total; base += (long)gridDim.x * C::TEAMS) {
    const bool valid = base + team < total;
    const long item = valid ? base + team : total - 1;
    const int w0 = a.W == 1 ? 0 : (int)(item % a.W);
    const long rest = a.W == 1 ? item : item / a.W;
    const int q = (int)(rest / npair) * a.W + w0, yy = 2 * (int)(rest % npair);
    const cx_fft_plane& pl = a.planes[q];
    const bool two = yy + 1 < a.py;
    const int yp0 = add_mod(yy, a.py / 2, a.py);  // ifftshift: padded-grid rows feeding FFT rows yy, yy + 1
    const int yp1 = add_mod(two ? yy + 1 : yy, a.py / 2, a.py);
    const int y0 = yp0 - a.pad_y, y1 = yp1 - a.pad_y;
    const bool d0 = valid && y0 >= 0 && y0 < a.ny, d1 = valid && two && y1 >= 0 && y1 < a.ny;
    const int in = pl.in_plane, b = in / a.W, w = in % a.W;
    const float2* plane = u + (size_t)b * a.ny * a.nx * a.W + w;
    const float2* r0 = plane + (size_t)(d0 ? y0 : 0) * a.nx * a.W;
    const float2* r1 = plane + (size_t)(d1 ? y1 : 0) * a.nx * a.W;
    const float cj = pl.conj ? -1.f : 1.f;
    const float2 pre = make_float2((float)pl.pre_re, (float)pl.pre_im);
    auto raw = [&](int x) -> c2 {
      const bool ok = (unsigned)x < (unsigned)a.nx;
      return ppack(ld2z(r0 + (ptrdiff_t)(x * a.W), ok && d0), ld2z(r1 + (ptrdiff_t)(x * a.W), ok && d1));
    };
    auto scale = [&](c2 v) -> c2 {
      v.im = __fmul2_rn(v.im, f2dup(cj));
      return pmulw<false>(v, pre);
    };
    sync();  // the pair's previous transform has been read
    if (pl.chirp_in == 0.0 && pl.pupil_r2 < 0.0) {
      auto load = [&](int n) -> c2 {
        return scale(raw(add_mod(n, NX / 2, NX) - a.pad_x));
      };
      F::template first<false>(s, tw, t, load);
    } else {
      const double ry0 = pl.dy_in * ((double)yp0 - 0.5 * a.py) + pl.oy;
      const double ry1 = pl.dy_in * ((double)yp1 - 0.5 * a.py) + pl.oy;
#pragma unroll 1
      for (int j = t; j < F::M; j += F::L) {
#pragma unroll 1
        for (int r = 0; r < F::R1; ++r) {
          const int xp = add_mod(j + r * F::M, NX / 2, NX), x = xp - a.pad_x;
          c2 v = pzero();
          if ((unsigned)x < (unsigned)a.nx) {
            v = raw(x);
            const double rx = pl.dx_in * ((double)xp - 0.5 * a.px) + pl.ox;
            if (pl.chirp_in != 0.0) v = pmul(v, ppack(chirp(pl.chirp_in, ry0, rx), chirp(pl.chirp_in, ry1, rx)));
            v = scale(v);
            // circular_pupil tests |field.grid|^2, the grid including the origin (pupils.py:17-23)
            if (pl.pupil_r2 >= 0.0) {
              if (ry0 * ry0 + rx * rx > pl.pupil_r2) v.re.x = v.im.x = 0.f;
              if (ry1 * ry1 + rx * rx > pl.pupil_r2) v.re.y = v.im.y = 0.f;
            }
          }
          sstore(s + r * F::PITCH + j, v);
        }
      }
      // each lane transforms the elements that it stored
      auto load = [&](int n) -> c2 { return sload(s + (n / F::M) * F::PITCH + n % F::M); };
      F::template first<false>(s, tw, t, load);
    }
    F::template inner<false>(s, tw, t, sync);
    float2* dst = T + ((size_t)q * a.py + yy) * a.px;
    auto out = [&](int k, c2 v) {
      if (valid) dst[k] = pfirst(v);
      if (valid && two) dst[a.px + k] = psecond(v);
    };
    F::template last<false>(s, t, out);
  }
}

// V = 2 VP columns; VEC: 16-byte reads of a column pair (even row length)
template <int NY>
using OptPairCols = PairCols<NY>;

template <int NY, bool VEC>
__global__ void __launch_bounds__(OptPairCols<NY>::THREADS, OptPairCols<NY>::MINB)
    k_opt_cols_pair(const float2* __restrict__ T, float2* __restrict__ outp, OptArgs a) {
  using C = OptPairCols<NY>;
  using F = typename C::F;
  constexpr int VP = C::VP, V = 2 * VP, NB = NY / F::RL;
  extern __shared__ __align__(16) char smem[];
  float2* tw = reinterpret_cast<float2*>(smem);
  F::load_tables(tw, a.twg, threadIdx.x, blockDim.x);
  const int c = threadIdx.x % VP, t = threadIdx.x / VP;
  float4* s = reinterpret_cast<float4*>(smem + C::TWB) + c;
  auto sync = [] { __syncthreads(); };
  const int tiles_x = (a.px + V - 1) / V;
  const long total = (long)tiles_x * a.n_out_planes;
  for (long i = blockIdx.x; i < total; i += gridDim.x) {
    const int q = (int)(i / tiles_x);
    const int x = (int)(i % tiles_x) * V + 2 * c;
    const cx_fft_plane& pl = a.planes[q];
    const bool ok0 = x < a.px, ok1 = x + 1 < a.px;
    const float2* src = T + (size_t)q * a.py * a.px + x;
    auto load = [&](int n) -> c2 {
      const float2* p = src + (size_t)n * a.px;
      if constexpr (VEC) return ppack(ld4z(p, ok0));
      return ppack(ld2z(p, ok0), ld2z(p + 1, ok1));
    };
    // fftshift along x, crop
    const int g0 = add_mod(ok0 ? x : 0, a.px / 2, a.px), g1 = add_mod(ok1 ? x + 1 : 0, a.px / 2, a.px);
    const int c0 = g0 - a.crop_x, c1 = g1 - a.crop_x;
    const bool w0 = ok0 && (unsigned)c0 < (unsigned)a.ox_n, w1 = ok1 && (unsigned)c1 < (unsigned)a.ox_n;
    const float cj = pl.conj ? -1.f : 1.f;
    const float2 post = make_float2((float)pl.post_re, (float)pl.post_im);
    const int b = q / a.W, w = q % a.W;
    float2* dst = outp + (size_t)b * a.oy_n * a.ox_n * a.W + w;
    const float2* h = a.H ? a.H + (size_t)q * a.py * a.px + x : nullptr;
    auto value = [&](int k, c2 v) -> c2 {
      if (h) v = pmul(v, ppack(ok0 ? h[(size_t)k * a.px] : make_float2(0.f, 0.f),
                               ok1 ? h[(size_t)k * a.px + 1] : make_float2(0.f, 0.f)));
      v.im = __fmul2_rn(v.im, f2dup(cj));
      return pmulw<false>(v, post);
    };
    auto store = [&](int row, c2 v) {
      const int r = row - a.crop_y;
      if ((unsigned)r >= (unsigned)a.oy_n) return;
      float2* o = dst + (size_t)r * a.ox_n * a.W;
      if (w0) o[(size_t)(c0 * a.W)] = pfirst(v);
      if (w1) o[(size_t)(c1 * a.W)] = psecond(v);
    };
    __syncthreads();  // the previous tile has been read
    F::template first<false>(s, tw, t, load);
    F::template inner<false>(s, tw, t, sync);
    if (pl.chirp_out == 0.0 && !(pl.pupil_out_r2 > 0.0)) {
      auto out = [&](int k, c2 v) { store(add_mod(k, NY / 2, NY), value(k, v)); };  // fftshift along y
      F::template last<false>(s, t, out);
    } else {
      const double rx0 = pl.dx_out * ((double)g0 - 0.5 * a.px) + pl.ox, rx1 = pl.dx_out * ((double)g1 - 0.5 * a.px) + pl.ox;
      F::template last_in_place<false>(s, t);
      // each lane finishes the butterflies that it stored
#pragma unroll 1
      for (int bf = t; bf < NB; bf += F::L) {
#pragma unroll 1
        for (int r = 0; r < F::RL; ++r) {
          const int k = bf + r * NB, row = add_mod(k, NY / 2, NY);
          c2 v = value(k, sload(F::last_ptr(s, bf) + r * VP));
          const double ry = pl.dy_out * ((double)row - 0.5 * a.py) + pl.oy;
          if (pl.chirp_out != 0.0) v = pmul(v, ppack(chirp(pl.chirp_out, ry, rx0), chirp(pl.chirp_out, ry, rx1)));
          // output-grid pupil (the adjoint of the input pupil of ff_lens)
          if (pl.pupil_out_r2 > 0.0) {
            if (ry * ry + rx0 * rx0 > pl.pupil_out_r2) v.re.x = v.im.x = 0.f;
            if (ry * ry + rx1 * rx1 > pl.pupil_out_r2) v.re.y = v.im.y = 0.f;
          }
          store(row, v);
        }
      }
    }
  }
}

}  // namespace cx
