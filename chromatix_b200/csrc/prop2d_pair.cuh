// The three passes of the Fourier-multiplier propagation (prop2d.cuh) on pairs
// of rows / columns, for every length with a pair plan (pair_fft.cuh).
//
// Work per point (1024): the scalar column pass ran 265 thread instructions
// (two transforms, the propagator in FP64, four copies through shared memory);
// here a column pair's tile goes from global memory into the first stage's
// registers and from the last stage's registers back, the forward and inverse
// transform share one pass over shared memory where the propagator is applied,
// and the propagator of a tile is evaluated once for as many planes as use it.
#pragma once

#include "pair_fft.cuh"
#include "prop2d.cuh"

namespace cx {

// first-stage inputs that a field in the central half of the padded axis leaves zero
template <int N, bool LONE = false>
constexpr unsigned pair_band_mask() {
  unsigned m = 0u;
  constexpr int R = PairPlan<N, LONE>::R1;
  for (int r = 0; r < R; ++r)
    if (r < R / 4 || r >= 3 * R / 4) m |= 1u << r;
  return m;
}

// row pitch of the stored spectra
__device__ __forceinline__ int prop_pitch(const Prop2DArgs& a) { return a.tsh == 30 ? a.px : 1 << a.tsh; }

// --------------------------------------------------------------------------
// pass A: forward row transform of row pairs, zero padding in the loader
// --------------------------------------------------------------------------
// Pairs are rows 2 i, 2 i + 1 of one plane; the wavelengths of a chromatic
// field run fastest, so that the CTA's teams read the interleaved row once.
template <int NX>
__global__ void __launch_bounds__(PairRows<NX>::THREADS, PairRows<NX>::MINB)
    k_prop_rows_fwd_pair(const float2* __restrict__ u, float2* __restrict__ T, Prop2DArgs a) {
  using C = PairRows<NX>;
  using F = typename C::F;
  extern __shared__ __align__(16) char smem[];
  float2* tw = reinterpret_cast<float2*>(smem);
  F::load_tables(tw, a.twg, threadIdx.x, blockDim.x);
  const int team = threadIdx.x / C::L, t = threadIdx.x % C::L;
  float4* s = reinterpret_cast<float4*>(smem + C::TWB) + (size_t)team * F::ELEMS;
  auto sync = [&] { C::sync(team); };
  const int npair = (a.ny + 1) / 2;
  const long total = (long)(a.n_in_planes / a.W) * npair * a.W;
  const bool band = 4 * a.pad_x >= NX && 4 * (a.pad_x + a.nx) <= 3 * NX;
  const int low = (1 << a.tsh) - 1, rT = prop_pitch(a), tstep = a.ny * rT;
  __syncthreads();
  for (long base = (long)blockIdx.x * C::TEAMS; base < total; base += (long)gridDim.x * C::TEAMS) {
    const long item = base + team;
    const bool valid = item < total;
    const int w = valid ? (int)(item % a.W) : 0;
    const long bi = valid ? item / a.W : 0;
    const int b = (int)(bi / npair), y = 2 * (int)(bi % npair);
    const bool two = valid && y + 1 < a.ny;
    const float2* ub = a.in_ptrs ? a.in_ptrs[b] : u + (size_t)b * a.ny * a.nx * a.W;
    const float2* src = ub + (size_t)y * a.nx * a.W + w;
    const size_t up = two ? (size_t)a.nx * a.W : 0;
    float2* dst = T + (size_t)(b * a.W + w) * a.ny * a.px + (size_t)y * rT;
    auto load = [&](int n) -> c2 {
      const int x = n - a.pad_x;
      if (!valid || (unsigned)x >= (unsigned)a.nx) return pzero();
      const float2* p = src + (size_t)(x * a.W);
      return ppack(p[0], p[up]);
    };
    auto out = [&](int k, c2 v) {
      float2* p = dst + (k >> a.tsh) * tstep + (k & low);
      if (valid) p[0] = pfirst(v);
      if (two) p[rT] = psecond(v);
    };
    sync();  // the pair's previous transform has been read
    if (band)
      F::template transform<false, pair_band_mask<NX>()>(s, tw, t, load, out, sync);
    else
      F::template transform<false>(s, tw, t, load, out, sync);
  }
}

// --------------------------------------------------------------------------
// pass C: inverse row transform of the output rows, crop in the store
// --------------------------------------------------------------------------
template <int NX>
__global__ void __launch_bounds__(PairRows<NX>::THREADS, PairRows<NX>::MINB)
    k_prop_rows_inv_pair(const float2* __restrict__ T2, float2* __restrict__ outp, Prop2DArgs a) {
  using C = PairRows<NX>;
  using F = typename C::F;
  extern __shared__ __align__(16) char smem[];
  float2* tw = reinterpret_cast<float2*>(smem);
  F::load_tables(tw, a.twg, threadIdx.x, blockDim.x);
  const int team = threadIdx.x / C::L, t = threadIdx.x % C::L;
  float4* s = reinterpret_cast<float4*>(smem + C::TWB) + (size_t)team * F::ELEMS;
  auto sync = [&] { C::sync(team); };
  const int npair = (a.out_ny + 1) / 2;
  const long total = (long)(a.n_out_planes / a.W) * npair * a.W;
  const int low = (1 << a.tsh) - 1, rT = prop_pitch(a), tstep = a.out_ny * rT;
  __syncthreads();
  for (long base = (long)blockIdx.x * C::TEAMS; base < total; base += (long)gridDim.x * C::TEAMS) {
    const long item = base + team;
    const bool valid = item < total;
    const int w = valid ? (int)(item % a.W) : 0;
    const long bi = valid ? item / a.W : 0;
    const int b = (int)(bi / npair), r = 2 * (int)(bi % npair);
    const bool two = valid && r + 1 < a.out_ny;
    const float2* src = T2 + (size_t)(b * a.W + w) * a.out_ny * a.px + (size_t)r * rT;
    const int up = two ? rT : 0;
    float2* ob = a.out_ptrs ? a.out_ptrs[b] : outp + (size_t)b * a.out_ny * a.out_nx * a.W;
    float2* dst = ob + (size_t)r * a.out_nx * a.W + w;
    auto load = [&](int n) -> c2 {
      if (!valid) return pzero();
      const float2* p = src + (n >> a.tsh) * tstep + (n & low);
      return ppack(p[0], p[up]);
    };
    auto out = [&](int k, c2 v) {
      const int x = k - a.out_x0;
      if ((unsigned)x < (unsigned)a.out_nx) {
        if (valid) dst[(size_t)(x * a.W)] = pfirst(v);
        if (two) dst[(size_t)((a.out_nx + x) * a.W)] = psecond(v);
      }
    };
    sync();
    F::template transform<true>(s, tw, t, load, out, sync);
  }
}

// --------------------------------------------------------------------------
// pass B: column transform -> x H -> inverse, on tiles of V = 2 VP columns
// --------------------------------------------------------------------------
// TABLE = false: H is evaluated per tile into a shared-memory table of about
// NY/2 rows.  Where it is even in k_y (no tilt, no output shift and no band
// centre along y) rows 0 .. NY/2 serve both halves and stay for the CTA's next plane
// if that has the same parameters; otherwise the product runs in two
// halves, each with its own rows of the table.
// TABLE = true: H is the caller's table; the tile's columns are copied into
// shared memory beside the tile's loads.
template <int NY, bool TABLE>
struct PropPairCols {
  using P = PairPlan<NY, TABLE>;
  static constexpr int L = P::L;
  static constexpr int HROWS = TABLE ? NY : NY / 2 + 1;
  static constexpr size_t bytes(int vp) {
    return sizeof(float4) * (size_t)vp * (P::R1 * (NY / P::R1 + 1) + HROWS);
  }
  // the widest tile of at most 512 lanes with two CTAs per SM; two column
  // pairs (whole 32-byte sectors) where one CTA per SM has room for them.  With a table (the multislice loop, whose
  // adjoint runs two chains of one-plane passes side by side) three CTAs per SM.
  static constexpr int vp() {
    int v = 4;
    while (v > 1 && (v * L > 512 || bytes(v) > (v == 2 ? 200 : (TABLE ? 74 : 104)) * 1024)) v /= 2;
    return v;
  }
  static constexpr int VP = vp();
  using F = PairFFT<NY, VP, TABLE>;
  static constexpr int THREADS = VP * L;
  static constexpr int TWB = (F::TW * (int)sizeof(float2) + 15) & ~15;
  static constexpr size_t H_OFF = TWB + sizeof(float4) * (size_t)F::ELEMS;
  // an 8192-row table does not fit beside its tile: it is read from global memory
  static constexpr bool STAGED = H_OFF + sizeof(float4) * (size_t)HROWS * VP <= 227 * 1024;
  static constexpr size_t SMEM = H_OFF + (STAGED ? sizeof(float4) * (size_t)HROWS * VP : 0);
  static constexpr int WARPS = (THREADS + 31) / 32;
  static constexpr int MINB = SMEM > 113 * 1024 ? 1 : (16 / WARPS > 0 ? 16 / WARPS : 1);
};

// parameters that H depends on, besides the columns
__device__ __forceinline__ bool prop_same_h(const cx_plane& p, const cx_plane& q) {
  return p.z == q.z && p.wavelength == q.wavelength && p.dy == q.dy && p.dx == q.dx && p.shift_y == q.shift_y &&
         p.shift_x == q.shift_x && p.bl_y0 == q.bl_y0 && p.bl_x0 == q.bl_x0 && p.bl_hy == q.bl_hy && p.bl_hx == q.bl_hx;
}

// VEC: 16-byte accesses to a column pair (even row length, aligned buffers);
// otherwise (rows of 3, 5 or 7) element by element.
template <int NY, bool TABLE, bool VEC>
__global__ void __launch_bounds__(PropPairCols<NY, TABLE>::THREADS, PropPairCols<NY, TABLE>::MINB)
    k_prop_cols_pair(const float2* T, float2* T2, Prop2DArgs a, int per_cta) {
  using C = PropPairCols<NY, TABLE>;
  using F = typename C::F;
  constexpr int VP = C::VP, V = 2 * VP;
  extern __shared__ __align__(16) char smem[];
  if constexpr (TABLE) pdl_trigger();
  float2* tw = reinterpret_cast<float2*>(smem);
  float4* s0 = reinterpret_cast<float4*>(smem + C::TWB);
  float4* hs = reinterpret_cast<float4*>(smem + C::H_OFF);
  F::load_tables(tw, a.twg, threadIdx.x, blockDim.x);
  const int c = threadIdx.x % VP, t = threadIdx.x / VP;
  float4* s = s0 + c;
  auto sync = [] { __syncthreads(); };
  const int tiles_x = (a.px + V - 1) / V, rT = prop_pitch(a);
  const float scale = 1.0f / ((float)a.py * (float)a.px);
  const bool band = 4 * a.pad_y >= NY && 4 * (a.pad_y + a.ny) <= 3 * NY;
  // CTAs of adjacent column tiles run at the same time (their 32- or 64-byte row segments share DRAM pages); a
  // CTA works through per_cta planes of its tile, the planes of one wavelength following one another
  const int tile = (int)(blockIdx.x % tiles_x);
  const int o0 = (int)(blockIdx.x / tiles_x) * per_cta;
  const int o1 = o0 + per_cta < a.n_out_planes ? o0 + per_cta : a.n_out_planes;
  // plane (of the batch, or of the caller's table) that the propagator in shared memory belongs to
  int h_plane = -1;
  for (int o = o0; o < o1; ++o) {
    const int nb = a.n_out_planes / a.W, q = (o % nb) * a.W + o / nb;
    const int x0 = tile * V;
    const cx_plane& pl = a.planes[q];
    const int x = x0 + 2 * c;
    const bool ok0 = x < a.px, ok1 = x + 1 < a.px;
    const int xt = x >> a.tsh, xl = x & ((1 << a.tsh) - 1);
    const float2* src = T + (size_t)pl.in_plane * a.ny * a.px + (size_t)(xt * rT) * a.ny + xl;
    auto load = [&](int n) -> c2 {
      const int r = n - a.pad_y;
      const bool ok = ok0 && (unsigned)r < (unsigned)a.ny;
      const float2* p = src + (ptrdiff_t)r * rT;
      if constexpr (VEC) return ppack(ld4z(p, ok));
      return ppack(ld2z(p, ok), ld2z(p + 1, ok && ok1));
    };
    __syncthreads();  // the previous tile (and its propagator) has been read
    const float2* Hp = TABLE ? a.H + (size_t)pl.h_plane * NY * a.px : nullptr;
    if constexpr (TABLE && C::STAGED) {
      if (h_plane != pl.h_plane) {
        h_plane = pl.h_plane;
        const bool al = VEC && (reinterpret_cast<size_t>(a.H) & 15) == 0;
        for (int e = threadIdx.x; e < NY * VP; e += C::THREADS) {
          const int k = e / VP, cc = e % VP, xx = x0 + 2 * cc;
          const float2* g = Hp + (size_t)k * a.px + xx;
          if (al) {
            if (xx < a.px) cp_async16(hs + e, g);
          } else {
            float2* d = reinterpret_cast<float2*>(hs + e);
            if (xx < a.px) cp_async8(d, g);
            if (xx + 1 < a.px) cp_async8(d + 1, g + 1);
          }
        }
      }
    }
    if constexpr (TABLE) {
      if (o == o0) pdl_wait();  // the table and the twiddles are on their way
    }
    if (band)
      F::template first<false, pair_band_mask<NY, TABLE>()>(s, tw, t, load);
    else
      F::template first<false>(s, tw, t, load);
    if constexpr (TABLE) {
      const float cj = a.conj_h ? -1.f : 1.f;
      cp_async_wait_all();
      F::template inner<false>(s, tw, t, sync);
      auto f = [&](int b, int r, c2 v) -> c2 {
        const int k = b + r * (NY / F::RL);
        if (!ok0) return v;
        c2 h;
        if constexpr (C::STAGED) {
          h = ppack(hs[k * VP + c]);
        } else {
          const float2* g = Hp + (size_t)k * a.px + x;
          h = ppack(g[0], ok1 ? g[1] : make_float2(0.f, 0.f));
        }
        h.im = __fmul2_rn(h.im, f2dup(cj));
        if (a.na_f2 >= 0.0) {
          if (outside_na(k, x, a, pl)) h.re.x = h.im.x = 0.f;
          if (outside_na(k, x + 1, a, pl)) h.re.y = h.im.y = 0.f;
        }
        return pmul(v, h);
      };
      F::template centre<false>(s, t, f);
    } else {
      const PropK kc = prop_consts(a, pl);
      const bool even = a.ky0 == 0.0 && pl.shift_y == 0.0 && (!a.bandlimit || pl.bl_y0 == 0.0);
      const bool have = even && h_plane >= 0 && prop_same_h(a.planes[h_plane], pl);
      constexpr int NB = NY / F::RL, HB = NB / 2;  // butterflies of the centre, and of a half
      static_assert(NB % 2 == 0, "the halves have as many butterflies");
      h_plane = even ? q : -1;
      F::template inner<false>(s, tw, t, sync);
#pragma unroll 1
      for (int half = 0; half < (even ? 1 : 2); ++half) {
        if (!have) {
          if (half) __syncthreads();  // the first half's rows have been read
          const int rows = even ? NY / 2 + 1 : NY / 2;
          const int cc = threadIdx.x % V, xx = x0 + cc < a.px ? x0 + cc : a.px - 1;
          const PropCol pc = prop_col(a, pl, kc, xx);
          float* hf = reinterpret_cast<float*>(hs + cc / 2) + (cc & 1);
          constexpr int STEP = C::THREADS / V;
          const int e0 = threadIdx.x / V;
          // the evaluation by mode, outside the loop; on an even axis the frequency number of row e is e itself
          auto fill = [&](auto at) {
            double kf = (double)e0;
#pragma unroll 2
            for (int e = e0; e < rows; e += STEP, kf += (double)STEP) {
              // row e of a half: butterfly e % HB, output e / HB of the centre
              const int k = even ? e : (e % HB) + half * HB + (e / HB) * NB;
              const float2 h = at(even ? kf : (double)freq_index(k, NY), k);
              hf[4 * VP * e] = h.x;
              hf[4 * VP * e + 2] = h.y;
            }
          };
          switch (pc.mode) {
            case 1:
              fill([&](double kf, int k) { return prop_col_at<1>(kf, k, xx, pc, a, pl, kc); });
              break;
            case 2:
              fill([&](double kf, int k) { return prop_col_at<2>(kf, k, xx, pc, a, pl, kc); });
              break;
            case 3:
              fill([&](double kf, int k) { return prop_col_at<3>(kf, k, xx, pc, a, pl, kc); });
              break;
            default:
              fill([&](double kf, int k) { return prop_col_at<0>(kf, k, xx, pc, a, pl, kc); });
          }
          __syncthreads();
        }
        auto f = [&](int b, int r, c2 v) -> c2 {
          const int k = b + r * NB;
          const int row = even ? (k <= NY / 2 ? k : NY - k) : b - half * HB + r * HB;
          return pmul(v, sload(hs + row * VP + c));
        };
        F::template centre<false>(s, t, f, even ? 0 : half * HB, even || half ? NB : HB);
      }
    }
    float2* dst = T2 + (size_t)q * a.out_ny * a.px + (size_t)(xt * rT) * a.out_ny + xl;
    auto out = [&](int n, c2 v) {
      const int r = n - a.out_y0;
      if (!ok0 || (unsigned)r >= (unsigned)a.out_ny) return;
      v = pscale(v, scale);
      float2* p = dst + (size_t)r * rT;
      if constexpr (VEC) {
        *reinterpret_cast<float4*>(p) = punpack(v);
      } else {
        p[0] = pfirst(v);
        if (ok1) p[1] = psecond(v);
      }
    };
    F::template back<true>(s, tw, t, out, sync);
  }
}

// Planes per CTA: as many as leave four CTAs for every resident one (a last
// wave then costs at most a fifth), eight at most: the propagator's evaluation is then an eighth.
template <int NY, bool TABLE, bool VEC>
static cx_status launch_cols_pair(const float2* T, float2* T2, const Prop2DArgs& a, cudaStream_t st) {
  using C = PropPairCols<NY, TABLE>;
  auto k = k_prop_cols_pair<NY, TABLE, VEC>;
  const long tiles = (a.px + 2 * C::VP - 1) / (2 * C::VP);
  const long items = tiles * a.n_out_planes;
  const long resident = persistent_grid(k, C::THREADS, C::SMEM, items);
  long per = items / (4 * resident);
  per = per < 1 ? 1 : (per > 8 ? 8 : per);
  const long grid = tiles * ((a.n_out_planes + per - 1) / per);
  CX_CUDA_TRY(launch_kernel(k, (int)grid, C::THREADS, C::SMEM, st, TABLE && a.pdl, T, T2, a, (int)per));
  return CX_OK;
}

}  // namespace cx
